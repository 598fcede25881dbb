"""Workloads of the GDN path for timing: what a program does with the package through its public entry points.

A case is one call pattern (``call``) at one size:

* ``decode``      one generated token per sequence, ``ops.gdn_decode_step``, the state updated in place;
* ``prefill``     ``ops.gdn_chunk`` without gradients: the prompt of a generation, or evaluation;
* ``train``       ``ops.gdn_chunk`` forward and backward through autograd (``ops.gdn_chunk_full`` where the erase and
                  write gates are per channel);
* ``six_input``   forward and backward through ``ops.gdn2_op``, the surface of models written for six inputs;
* ``step_graph``  a training step at fixed shapes, captured once by ``ops.GdnStepGraph`` and replayed.

``variant`` names the member of the family: ``scalar`` (gated delta rule, one decay per token-head), ``kda``
(channel-wise decay), ``full`` (channel-wise decay, independent per-channel erase and write gates), and without the
delta term ``gla`` (channel-wise decay), ``ssd`` (one decay) and ``la`` (none).  Sizes are those of the benchmark
configurations and of the tests, and the ragged ones that real prompts and batches have.
"""

from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from lethe_b200 import ops

CHUNK = 64
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
DELTA = ("scalar", "kda", "full")
CHANNEL = ("kda", "gla", "full")
# token-heads of the largest listed case (B=2, H=32, L=8192); no drawn case has more
MOST_TOKEN_HEADS = 2 * 32 * 8192


def _case(call, variant, B, H, L, K, V, *, dtype="bf16", l2norm=False, h0=False, mild=True, name=None):
    c = {} if name is None else {"name": name}
    c.update(call=call, variant=variant, B=B, H=H, L=L, K=K, V=V, dtype=dtype, l2norm=l2norm, h0=h0, mild=mild)
    return c


def listed():
    return [
        # interactive generation, one sequence: a call is launch and host latency
        _case("decode", "scalar", 1, 8, 1, 128, 64, name="decode_b1_scalar"),
        # batched serving: the state (134 MB) is read and written once per token
        _case("decode", "kda", 64, 32, 1, 128, 128, name="decode_b64_kda"),
        # a short prompt of no particular length, raw q and k normalised by the op
        _case("prefill", "scalar", 1, 8, 1000, 128, 64, l2norm=True, name="prefill_short_ragged_scalar"),
        # a long prompt continued from an earlier state
        _case("prefill", "kda", 1, 32, 16000, 128, 128, l2norm=True, h0=True, name="prefill_long_kda"),
        # the small language model of the training-loop test: fp32 activations into the six-input op
        _case("six_input", "scalar", 4, 2, 256, 128, 64, dtype="fp32", l2norm=True, name="six_input_tiny_lm_fp32"),
        # the headline configuration as a training loop calls it, and as a captured step
        _case("train", "scalar", 2, 8, 2048, 128, 64, h0=True, mild=False, name="train_scalar_B2_H8_L2048"),
        _case("step_graph", "scalar", 2, 8, 2048, 128, 64, h0=True, mild=False, name="graph_scalar_B2_H8_L2048"),
        # the second configuration: channel-wise decay, raw q and k
        _case("train", "kda", 2, 8, 2048, 128, 128, l2norm=True, name="train_kda_B2_H8_L2048"),
        # the same shape with independent per-channel gates through the six-input op
        _case("six_input", "full", 2, 8, 2048, 128, 128, l2norm=True, name="six_input_full_B2_H8_L2048"),
        # the third configuration, with channel-wise decay
        _case("train", "gla", 4, 16, 4096, 128, 128, mild=False, name="train_gla_B4_H16_L4096"),
        # a state-space layer with 64 key channels on batches that end where their documents end
        _case("train", "ssd", 3, 12, 3001, 64, 64, name="train_ssd_dk64_ragged"),
        # one GPU's share of the largest configuration
        _case("train", "kda", 2, 32, 8192, 128, 128, mild=False, name="train_kda_B2_H32_L8192"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    call = rng.choice(["decode", "prefill", "prefill", "train", "train", "train", "six_input", "step_graph"])
    V = rng.choice([64, 128])
    mild = rng.random() < 0.5
    if call == "decode":
        variant = rng.choice(["scalar", "kda", "gla", "ssd"])
        return _case("decode", variant, _log_int(rng, 1, 64), _log_int(rng, 1, 32), 1, 128, V,
                     dtype=rng.choice(["bf16", "bf16", "fp32"]), mild=mild)
    H, L = _log_int(rng, 1, 32), _log_int(rng, 64, 16384)
    B = _log_int(rng, 1, max(1, min(8, MOST_TOKEN_HEADS // (H * L))))
    variant, K, dtype, l2norm = rng.choice(["scalar", "kda", "gla", "ssd", "la"]), 128, "bf16", rng.random() < 0.5
    if call in ("prefill", "train"):
        K = rng.choice([64, 128, 128, 128])
        dtype = rng.choice(["bf16", "bf16", "bf16", "fp16"])
        if call == "train" and K == 128 and rng.random() < 0.2:
            variant = "full"
    elif call == "six_input":
        variant, dtype = rng.choice(["scalar", "kda", "full", "gla", "ssd"]), rng.choice(["bf16", "fp32"])
    else:
        l2norm = False
    if call in ("six_input", "step_graph") or variant == "full":
        L = -(-L // CHUNK) * CHUNK          # these take whole chunks
        if variant == "full" or call == "six_input":    # gates and their gradients come per channel, in fp32
            B = max(1, min(B, MOST_TOKEN_HEADS // 2 // (H * L)))
    return _case(call, variant, B, H, L, K, V, dtype=dtype, l2norm=l2norm,
                 h0=call != "six_input" and rng.random() < 0.5, mild=mild)


def prepare(case, seed):
    """Seeded inputs of the benchmark's distributions: q, k ~ N(0,1), unit rows unless the op normalises them;
    v, dO ~ N(0,1); beta = sigmoid(N(0,1)); g = -softplus(N(0,1) + 3), or the gentle -0.1 U(0,1) of trained models;
    h0 ~ 0.1 N(0,1)."""
    c = dict(case)
    dev, gen = "cuda", torch.Generator(device="cuda").manual_seed(int(seed))
    B, H, L, K, V = c["B"], c["H"], c["L"], c["K"], c["V"]
    call, variant, dt = c["call"], c["variant"], DTYPES[c["dtype"]]
    vdt = torch.float32 if c["dtype"] == "fp32" else torch.bfloat16      # fp16 is a choice for q and k

    def normal(*shape):
        return torch.randn(*shape, generator=gen, device=dev)

    lead = (B, H) if call == "decode" else (B, L, H)
    q, k = normal(*lead, K), normal(*lead, K)
    if not c["l2norm"]:
        q, k = F.normalize(q, dim=-1), F.normalize(k, dim=-1)
    s = {"case": c, "q": q.to(dt), "k": k.to(dt), "v": normal(*lead, V).to(vdt), "g": None, "beta": None, "h0": None}
    del q, k
    if variant != "la":
        gshape = (*lead, K) if variant in CHANNEL else lead
        if c["mild"]:
            s["g"] = torch.rand(*gshape, generator=gen, device=dev).mul_(-0.1)
        else:
            s["g"] = -F.softplus(normal(*gshape) + 3.0)
    if variant in ("scalar", "kda"):
        s["beta"] = normal(*lead).sigmoid()
    if variant == "full":
        s["b"], s["w"] = normal(*lead, K).sigmoid(), normal(*lead, V).sigmoid()
    if call == "decode":
        s["state"] = 0.1 * normal(B, H, K, V)
        return s
    if c["h0"]:
        s["h0"] = 0.1 * normal(B, H, K, V)
    if call == "prefill":
        return s
    s["do"] = normal(B, L, H, V).to(vdt)
    if call == "step_graph":
        gate = {"la": ops.GATE_NONE}.get(variant, ops.GATE_CHANNEL if variant in CHANNEL else ops.GATE_SCALAR)
        s["buf"] = ops.GdnBuffers(B, L, H, K, V, gate, variant in DELTA, torch.device(dev), qk_dtype=dt)
        s["step"] = ops.GdnStepGraph(s["buf"], s["q"], s["k"], s["v"], s["g"], s["beta"], s["h0"], s["do"], None,
                                     float(K) ** -0.5)
        return s
    if call == "six_input":
        # the op takes every gate per channel; a model with one decay or one beta per head hands over expanded gates
        if variant in ("scalar", "ssd"):
            s["g"] = s["g"].unsqueeze(-1).expand(B, L, H, K).contiguous()
        if variant in ("scalar", "kda"):
            beta = s.pop("beta").unsqueeze(-1)
            s["b"], s["w"] = beta.expand(B, L, H, K).contiguous(), beta.expand(B, L, H, V).contiguous()
        elif variant != "full":
            s["b"], s["w"] = torch.zeros(B, L, H, K, device=dev), torch.ones(B, L, H, V, device=dev)
        names = ("q", "k", "v", "g", "b", "w")
    elif variant == "full":
        names = ("q", "k", "v", "g", "b", "w", "h0")
    else:
        names = ("q", "k", "v", "g", "beta", "h0")
    s["wrt"] = [n for n in names if s.get(n) is not None]
    for n in s["wrt"]:
        s[n].requires_grad_(True)
    return s


def run(s):
    c = s["case"]
    call = c["call"]
    if call == "decode":
        o = ops.gdn_decode_step(s["q"], s["k"], s["v"], s["g"], s["beta"], s["state"])
        return {"o": o, "state": s["state"]}
    if call == "step_graph":
        s["step"].replay()
        b = s["buf"]
        out = {"o": b.o, "hT": b.hT, "dq": b.dq, "dk": b.dk, "dv": b.dv, "dg": b.dg, "dbeta": b.dbeta, "dh0": b.dh0}
        return {n: t for n, t in out.items() if t is not None}
    if call == "prefill":
        with torch.no_grad():
            o, hT = ops.gdn_chunk(s["q"], s["k"], s["v"], s["g"], s["beta"], s["h0"], use_qk_l2norm=c["l2norm"])
        return {"o": o, "hT": hT}
    hT = None
    if call == "six_input":
        o = ops.gdn2_op(s["q"], s["k"], s["v"], s["g"], s["b"], s["w"], use_qk_l2norm=c["l2norm"])
    elif c["variant"] == "full":
        o, hT = ops.gdn_chunk_full(s["q"], s["k"], s["v"], s["g"], s["b"], s["w"], s["h0"], use_qk_l2norm=c["l2norm"])
    else:
        o, hT = ops.gdn_chunk(s["q"], s["k"], s["v"], s["g"], s["beta"], s["h0"], use_qk_l2norm=c["l2norm"])
    grads = torch.autograd.grad(o, [s[n] for n in s["wrt"]], s["do"])
    out = {"d" + n: t for n, t in zip(s["wrt"], grads)}
    out["o"] = o.detach()
    if hT is not None:
        out["hT"] = hT.detach()
    return out


def work(case):
    """Bytes: every input read once, every output written once.  Operations: the dense products of the chunk form
    (64 tokens), forward and backward; for a decoded token those on the state."""
    c = dict(case)
    B, H, L, K, V = c["B"], c["H"], c["L"], c["K"], c["V"]
    TH, C = B * H * L, CHUNK
    e = 4 if c["dtype"] == "fp32" else 2
    variant, call = c["variant"], c["call"]
    state = 4 * B * H * K * V
    gates = {"la": 0, "scalar": 4, "ssd": 4}.get(variant, 4 * K)
    gates += {"scalar": 4, "kda": 4, "full": 4 * (K + V)}.get(variant, 0)
    if call == "six_input":
        gates = 4 * (2 * K + V)              # per-channel tensors at this surface, whatever they hold
    qkv = e * (2 * K + V)
    delta = variant in DELTA
    if call == "decode":
        return {"bytes": TH * (qkv + gates + 2 * V) + 2 * state, "flops": TH * K * V * (7 if delta else 5)}
    fwd_bytes = TH * (qkv + gates + e * V) + state * (0 if call == "six_input" else 2 if c["h0"] else 1)
    if delta:
        chunk_fwd = 6 * C * C * K + 4 * C * C * V + 6 * C * K * V + C ** 3 / 3
        chunk_bwd = 12 * C * C * K + 8 * C * C * V + 12 * C * K * V + 4 * C ** 3
    else:
        chunk_fwd = 2 * C * C * K + 2 * C * C * V + 4 * C * K * V
        chunk_bwd = 4 * C * C * K + 4 * C * C * V + 8 * C * K * V
    if call == "prefill":
        return {"bytes": fwd_bytes, "flops": TH / C * chunk_fwd}
    # the backward adds dO in and a gradient for each input out
    dh0 = state if (c["h0"] or call == "step_graph") else 0
    return {"bytes": fwd_bytes + TH * (e * V + qkv + gates) + dh0, "flops": TH / C * (chunk_fwd + chunk_bwd)}


def tolerance(case):
    # decode computes in fp32: the state to rounding, o rounded once to bf16.  Elsewhere operands are 16-bit with fp32
    # sums and the results bf16, or fp32 sums of such products.
    if case["call"] == "decode":
        return {"rel": 4e-3, "max": 2e-2}
    return {"rel": 1e-2, "max": 1e-1}
