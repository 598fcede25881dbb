"""The scans that are joint with the kernel beside them: that they are what ran, and the bits of the kernels apart (``lean`` 0) for
batches, ranges of pairs, ragged lengths, 64 key channels and calls without initial states; and the captured step that consists of them."""
import ctypes

import pytest
import torch

from lethe_b200 import native, ops
from lethe_b200.synth import make_inputs

from .wsview import layout

PATTERN = 0x7f           # (fp16 0x7f7f is a NaN)


def run(d, buf, lean, dhT, L, K, delta, ranges, backward=True):
    """One forward and backward by the C ABI: user tensors of L tokens and K channels, in ranges of the pairs."""
    o = d["out"]
    st = torch.cuda.current_stream().cuda_stream
    for b0, n in ranges:
        a = ops._Args(dims=buf.dims, scale=K ** -0.5, saved=buf.saved.data_ptr(), saved_bytes=buf.saved.numel(), status=buf.status.data_ptr(),
                      l_tokens=L, k_channels=K, lean=lean, bh_begin=b0, bh_count=n,
                      **{n: ops._ptr(d.get(n)) for n in ("q", "k", "v", "g", "beta", "h0")}, b_gate=ops._ptr(d.get("b")), w_gate=ops._ptr(d.get("w")),
                      o=ops._ptr(o["o"]), hT=ops._ptr(o["hT"]))
        assert native.lib().lethe_gdn_forward(ctypes.byref(a), st) == 0
    for b0, n in ranges if backward else ():
        a = ops._Args(dims=buf.dims, scale=K ** -0.5, saved=buf.saved.data_ptr(), saved_bytes=buf.saved.numel(), status=buf.status.data_ptr(),
                      scratch=buf.scratch.data_ptr(), scratch_bytes=buf.scratch.numel(), l_tokens=L, k_channels=K, lean=min(lean, 1), bh_begin=b0, bh_count=n,
                      **{n: ops._ptr(d.get(n)) for n in ("q", "k", "v", "g", "beta", "h0")}, b_gate=ops._ptr(d.get("b")), w_gate=ops._ptr(d.get("w")),
                      d_o=ops._ptr(d["do"]), dhT=ops._ptr(dhT), **{n: ops._ptr(o.get(n)) for n in ("dq", "dk", "dv", "dg", "dbeta", "dh0")},
                      db_gate=ops._ptr(o.get("db")), dw_gate=ops._ptr(o.get("dw")))
        assert native.lib().lethe_gdn_backward(ctypes.byref(a), st) == 0
    torch.cuda.synchronize()
    ops.check_status(buf.status)


@pytest.mark.gpu
@pytest.mark.parametrize("delta,V,B,H,L,K,states", [
    (1, 128, 2, 10, 130, 128, True), (1, 64, 3, 13, 257, 64, True), (1, 128, 4, 5, 64, 64, False), (2, 128, 2, 10, 192, 128, False),
    (2, 64, 2, 20, 320, 128, True), (0, 128, 2, 23, 130, 128, True), (0, 64, 3, 31, 510, 64, False), (0, 128, 1, 60, 321, 64, True),
    (0, 128, 3, 43, 500, 128, True), (1, 128, 1, 160, 70, 128, False), (0, 64, 1, 180, 700, 128, False)])
def test_bits_of_the_kernels_apart(delta, V, B, H, L, K, states):
    dev, NT = torch.device("cuda"), -(-L // 64)
    inp = make_inputs(B, L, H, K, V, gate="channel", delta=bool(delta), seed=L, mild=True, full=delta == 2, with_h0=states)
    base = {n: t.to(dev) for n, t in inp.items() if t is not None}
    dhT = 0.1 * torch.randn(B, H, K, V, generator=torch.Generator().manual_seed(1)).to(dev) if states else None
    sms = torch.cuda.get_device_properties(dev).multi_processor_count
    got, buf = {}, ops.GdnBuffers(B, 64 * NT, H, 128, V, ops.GATE_CHANNEL, delta, dev)
    Z, sz, off, sz2, off2 = layout(B, H, 64 * NT, V)
    first = (B * H) // 3
    for label, lean, ranges in (("apart", 0, [(0, 0)]), ("joint", 1, [(0, 0)]), ("ranges", 1, [(first, B * H - first), (0, first)]), ("evaluation", 2, [(0, 0)])):
        joint = native.lib().lethe_gdn_joint_scans(ctypes.byref(buf.dims), lean, sms)
        buf.saved.fill_(PATTERN), buf.scratch.fill_(PATTERN)
        nan = lambda t, dt: torch.full(t.shape, float("nan"), dtype=dt, device=dev)
        out = {"o": nan(base["v"], torch.bfloat16), "hT": torch.full((B, H, K, V), float("nan"), device=dev), "dq": nan(base["q"], torch.bfloat16),
               "dk": nan(base["k"], torch.bfloat16), "dv": nan(base["v"], torch.bfloat16), "dg": nan(base["g"], torch.float32)}
        if delta == 1:
            out["dbeta"] = nan(base["beta"], torch.float32)
        if delta == 2:
            out["db"], out["dw"] = nan(base["b"], torch.float32), nan(base["w"], torch.float32)
        if states:
            out["dh0"] = torch.full((B, H, K, V), float("nan"), device=dev)
        run({**base, "out": out}, buf, lean, dhT, L, K, delta, ranges, backward=lean < 2)
        got[label] = out if lean < 2 else {n: out[n] for n in ("o", "hT")}
        # which kernels ran: what goes between the two of a pair is there or not
        rb, hc = (t[o:o + n] for t, o, n in ((buf.scratch, off2["rb"], Z * sz2["rb"]), (buf.saved, off["hc"], (Z + B * H) * sz["hc"])))
        assert bool((rb == PATTERN).all()) == bool(lean == 2 or joint & 2), label
        assert bool((hc == PATTERN).all()) == bool(lean == 2 and joint & 1), label
        assert lean == 0 or joint, "a case for the joint kernels"
    for label, out in got.items():
        for n, t in out.items():
            assert torch.equal(t, got["apart"][n]) and torch.isfinite(t.float()).all(), (label, n)


@pytest.mark.gpu
@pytest.mark.parametrize("delta,V,BH,NT,groups", [(1, 128, 20, 8, 1), (1, 64, 45, 9, 1), (0, 128, 46, 10, 1), (0, 64, 100, 9, 1), (1, 128, 20, 5, 2), (0, 128, 46, 5, 3),
                                                   (1, 128, 20, 8, 3)])
def test_the_captured_step_of_whole_calls_equals_plain_launches_on_every_replay(delta, V, BH, NT, groups):
    K, L, dev = 128, 64 * NT, torch.device("cuda")
    inp = make_inputs(1, L, BH, K, V, gate="channel", delta=bool(delta), seed=NT, mild=True)
    args = [None if inp[n] is None else inp[n].to(dev) for n in ("q", "k", "v", "g", "beta", "h0")]
    do = inp["do"].to(dev)
    ref, buf = (ops.GdnBuffers(1, L, BH, K, V, ops.GATE_CHANNEL, delta, dev) for _ in range(2))
    ops.forward_into(ref, *args, K ** -0.5)
    ops.backward_into(ref, *args, do, None, K ** -0.5)
    sms = torch.cuda.get_device_properties(dev).multi_processor_count
    assert groups > 1 or ops.step_is_chain(ops.GATE_CHANNEL, V, bool(delta), BH, sms, NT)
    graph = ops.GdnStepGraph(buf, *args, do, None, K ** -0.5, groups=groups)
    assert not graph.pipeline and graph.cut == 0 and graph.launches == 4
    names = ["o", "hT", "dq", "dk", "dv", "dg", "dh0"] + (["dbeta"] if delta else [])
    flush = torch.empty(192 << 20, dtype=torch.uint8, device=dev)
    for rep in range(10):
        for n in names:
            getattr(buf, n).fill_(float("nan"))
        if rep == 5:
            buf.saved.fill_(PATTERN), buf.scratch.fill_(PATTERN)
        if rep % 2:
            flush.zero_()
        graph.replay()
        torch.cuda.synchronize()
        ops.check_status(buf.status)
        for n in names:
            assert torch.equal(getattr(buf, n), getattr(ref, n)), (rep, n)
