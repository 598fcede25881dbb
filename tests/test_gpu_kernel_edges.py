"""Sizes at the edges of the kernels' dispatch rules and work splits, against the token-serial fp64 oracle (reference
``gdn_backward.py:16-57``)."""
import pytest
import torch

from lethe_b200 import ops
from lethe_b200.synth import make_inputs
from oracle.gdn_oracle import scale_rel, serial_backward, serial_backward_full, serial_forward

from .wsview import report

pytestmark = pytest.mark.gpu
TOL = 5e-3


@pytest.mark.parametrize("gate,delta,dtype,extra,shift", [
    ("channel", True, torch.bfloat16, 0, 0), ("channel", True, torch.bfloat16, 1, 0), ("scalar", False, torch.float32, 150, 0),
    ("none", True, torch.bfloat16, 3, 1)])
def test_decode_of_many_pairs(gate, delta, dtype, extra, shift):
    """The fewest pairs that the persistent kernel takes, a last round with few CTAs at work, and a state
    that starts off a 16-byte boundary."""
    dev = torch.device("cuda")
    H, V = 4 * torch.cuda.get_device_properties(dev).multi_processor_count + extra, 128
    inp = make_inputs(1, 1, H, 128, V, gate=gate, delta=delta, seed=4)
    f64 = {n: (None if t is None else t.double()) for n, t in inp.items()}
    o_ref, hT_ref = serial_forward(f64["q"], f64["k"], f64["v"], f64["g"], f64["beta"], f64["h0"])
    tok = lambda n, dt: None if inp[n] is None else inp[n][:, 0].to(dev, dt)      # noqa: E731
    flat = torch.empty(H * 128 * V + shift, device=dev)
    state = flat[shift:].view(1, H, 128, V)
    state.copy_(inp["h0"])
    o = ops.gdn_decode_step(tok("q", dtype), tok("k", dtype), tok("v", dtype), tok("g", torch.float32), tok("beta", torch.float32), state)
    errs = {"o": scale_rel(o.double().cpu(), o_ref[:, 0]), "state": scale_rel(state.double().cpu(), hT_ref)}
    report(f"decode gate={gate} delta={delta} pairs={H}", errs)
    assert max(errs.values()) <= TOL, errs


@pytest.mark.parametrize("gate,delta,V,K,H,L,dtype", [
    # more chunks than any persistent grid has CTAs (up to four per SM), the last of every sequence ragged
    ("scalar", True, 64, 128, 450, 100, torch.bfloat16), ("scalar", True, 128, 128, 310, 128, torch.bfloat16),
    ("scalar", False, 64, 64, 450, 100, torch.bfloat16), ("none", False, 128, 128, 310, 128, torch.float16),
    ("channel", True, 128, 128, 155, 100, torch.bfloat16), ("channel", True, 64, 64, 155, 128, torch.float16),
    ("channel", False, 64, 128, 155, 100, torch.bfloat16),
    # channel-wise prepare: one chunk per SM for the last time, two CTAs per SM for the first
    ("channel", True, 128, 128, 148, 64, torch.bfloat16), ("channel", True, 64, 64, 149, 60, torch.float16),
    ("channel", False, 128, 128, 149, 64, torch.bfloat16),
    # state scans: 8 and 16 columns per CTA for the last time, 16 and 64 for the first, on fewer chunks than stages and more; without
    # the delta term 16 and 8 records ahead
    ("scalar", True, 64, 128, 18, 70, torch.bfloat16), ("scalar", True, 64, 64, 19, 448, torch.float16),
    ("none", True, 128, 128, 9, 320, torch.bfloat16), ("channel", True, 128, 128, 10, 192, torch.bfloat16),
    ("scalar", True, 128, 128, 18, 100, torch.bfloat16), ("scalar", True, 128, 64, 19, 320, torch.bfloat16),
    ("scalar", True, 64, 128, 37, 320, torch.bfloat16), ("scalar", True, 64, 128, 38, 320, torch.bfloat16),
    ("none", False, 64, 128, 74, 1088, torch.bfloat16), ("none", False, 64, 128, 75, 1088, torch.bfloat16)])
def test_persistent_grids_and_scan_rules(gate, delta, V, K, H, L, dtype):
    dev = torch.device("cuda")
    inp = make_inputs(1, L, H, K, V, gate=gate, delta=delta, seed=9, mild=True)
    heads = [0, H // 2, H - 1]               # the pairs are independent: the oracle takes three of them
    pick = lambda n, t: None if t is None else t[:, heads] if n == "h0" else t[:, :, heads]      # noqa: E731
    f64 = {n: (None if t is None else pick(n, t).double()) for n, t in inp.items()}
    o_ref, hT_ref, gr = serial_backward(*(f64[n] for n in ("q", "k", "v", "g", "beta", "h0", "do")))
    names = [n for n in ("q", "k", "v", "g", "beta", "h0") if inp[n] is not None]
    cast = lambda n, t: t.to(dev, dtype) if n in ("q", "k") else t.to(dev)      # noqa: E731
    d = {n: cast(n, inp[n]).requires_grad_(True) for n in names}
    o, hT = ops.gdn_chunk(*(d.get(n) for n in ("q", "k", "v", "g", "beta", "h0")))
    got = dict(zip(names, torch.autograd.grad(o, [d[n] for n in names], inp["do"].to(dev))))
    back = lambda n, t: pick(n, t.detach().double().cpu())      # noqa: E731
    ref = {"q": gr.dq, "k": gr.dk, "v": gr.dv, "g": gr.dg, "beta": gr.dbeta, "h0": gr.dh0}
    errs = {"o": scale_rel(back("o", o), o_ref), "hT": scale_rel(back("h0", hT), hT_ref)}
    errs.update({"d" + n: scale_rel(back(n, got[n]), ref[n]) for n in names})
    report(f"edges gate={gate} delta={delta} V={V} K={K} H={H} L={L}", errs)
    assert max(errs.values()) <= TOL, errs


@pytest.mark.parametrize("V,H,dtype", [(64, 150, torch.float32), (128, 150, torch.bfloat16)])
def test_per_channel_gates_with_more_chunks_than_ctas(V, H, dtype):
    dev = torch.device("cuda")
    inp = make_inputs(1, 128, H, 128, V, gate="channel", seed=6, mild=True, full=True)
    heads = [0, H - 1]
    names = ("q", "k", "v", "g", "b", "w")
    f64 = {n: inp[n][:, :, heads].double() for n in names}
    o_ref, _, ref = serial_backward_full(*(f64[n] for n in names), None, inp["do"][:, :, heads].double())
    d = {n: inp[n].to(dev, dtype if n in "qkv" else torch.float32).requires_grad_(True) for n in names}
    o = ops.gdn2_op(*(d[n] for n in names), use_qk_l2norm=False)
    got = dict(zip(names, torch.autograd.grad(o, [d[n] for n in names], inp["do"].to(dev, o.dtype))))
    errs = {"o": scale_rel(o.detach().double().cpu()[:, :, heads], o_ref)}
    errs.update({"d" + n: scale_rel(got[n].double().cpu()[:, :, heads], ref[n]) for n in names})
    report(f"per-channel gates V={V} {dtype}", errs)
    assert max(errs.values()) <= TOL, errs


@pytest.mark.parametrize("rows,K,V", [(1, 64, 64), (97, 128, 64), (5000, 128, 128)])
def test_gate_regime_sees_one_differing_channel(rows, K, V):
    dev = torch.device("cuda")
    g = -torch.rand(1, rows, 1, 1, device=dev).expand(1, rows, 1, K).contiguous()
    b = torch.rand(1, rows, 1, 1, device=dev).expand(1, rows, 1, K).contiguous()
    w = b[..., :1].expand(1, rows, 1, V).contiguous()
    assert ops.gate_regime(g, b, w) == (True, True, False)
    assert ops.gate_regime(g, torch.zeros_like(b), torch.ones_like(w)) == (True, False, True)
    for t, want in ((g, (False, True, False)), (b, (True, False, False)), (w, (True, False, False))):
        last = t[0, -1, 0, -1].clone()
        t[0, -1, 0, -1] = torch.nextafter(last, torch.zeros_like(last))
        assert ops.gate_regime(g, b, w) == want
        t[0, -1, 0, -1] = last


@pytest.mark.parametrize("K,V,L,H,dtype,delta", [(128, 128, 200, 150, torch.bfloat16, True), (64, 64, 130, 3, torch.float16, True),
                                                 (128, 64, 64, 5, torch.bfloat16, False)])
def test_rows_normalised_on_the_way_in(K, V, L, H, dtype, delta):
    """Channel-wise gate: the prepare kernel normalises q and k itself; same op on rows normalised beforehand."""
    dev = torch.device("cuda")
    inp = make_inputs(1, L, H, K, V, gate="channel", delta=delta, seed=12, mild=True)
    d = {n: (None if inp[n] is None else inp[n].to(dev)) for n in ("v", "g", "beta", "h0", "do")}
    q, k = ((3 * inp[n]).to(dev, dtype).requires_grad_(True) for n in ("q", "k"))
    rest = (d["v"], d["g"], d["beta"], d["h0"])
    o, hT = ops.gdn_chunk(q, k, *rest, use_qk_l2norm=True)
    o_ref, hT_ref = ops.gdn_chunk(*ops.l2norm_qk(q, k), *rest)
    with torch.no_grad():
        o_eval, hT_eval = ops.gdn_chunk(q, k, *rest, use_qk_l2norm=True)
    assert torch.equal(o, o_eval) and torch.equal(hT, hT_eval)
    got, ref = (torch.autograd.grad(x, (q, k), d["do"]) for x in (o, o_ref))
    errs = {"o": scale_rel(o.detach().double(), o_ref.detach().double()), "hT": scale_rel(hT.detach().double(), hT_ref.detach().double()),
            "dq": scale_rel(got[0].double(), ref[0].double()), "dk": scale_rel(got[1].double(), ref[1].double())}
    report(f"normalised on the way in K={K} V={V} {dtype}", errs)
    assert max(errs.values()) <= TOL, errs
