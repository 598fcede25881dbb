"""The scan kernels that carry the output / scan-input work beside them (``gdn_scan_io.cu``) against the kernels they stand for,
which a call takes that keeps every record (``lean`` 0): the same bits, whatever the number of chunks to the rings."""
import pytest
import torch

from lethe_b200 import ops
from lethe_b200.synth import make_inputs

from .cusource import kernel_body


def test_it_reads_nothing_before_it_waits():
    body = kernel_body("gdn_scan_io.cu", "scan_io_kernel")
    before = body[:body.index("griddep_wait();")]
    assert "p.lay." not in before.replace(before[:before.index("auto rec")], "") and "tma_" not in before and "bulk_" not in before


@pytest.mark.gpu
@pytest.mark.parametrize("NT", [1, 2, 3, 4, 5, 7, 13])
@pytest.mark.parametrize("delta,V,BH", [(1, 64, 38), (1, 128, 19), (2, 128, 20), (0, 64, 50), (0, 128, 46), (1, 64, 150), (0, 64, 180)])
def test_same_bits_as_the_kernels_apart(delta, V, BH, NT):
    if BH > 50 and NT not in (1, 3, 7):
        pytest.skip("more pairs than SMs: a few lengths")
    K, L, dev = 128, 64 * NT, torch.device("cuda")
    inp = make_inputs(1, L, BH, K, V, gate="channel", delta=bool(delta), seed=NT, mild=True, full=delta == 2)
    d = {n: t.to(dev) for n, t in inp.items() if t is not None}
    gates = {"b_gate": d["b"], "w_gate": d["w"]} if delta == 2 else {}
    dhT = 0.1 * torch.randn(1, BH, K, V, generator=torch.Generator().manual_seed(1)).to(dev)
    got = {}
    for lean in (0, 1, 2):
        buf = ops.GdnBuffers(1, L, BH, K, V, ops.GATE_CHANNEL, delta, dev)
        ins = (buf, d["q"], d["k"], d["v"], d["g"], d.get("beta"), d["h0"])
        ops.forward_into(*ins, K ** -0.5, lean=lean, **gates)
        names = ["o", "hT"]
        if lean < 2:
            ops.backward_into(*ins, d["do"], dhT, K ** -0.5, lean=lean, **gates)
            names += ["dq", "dk", "dv", "dg", "dh0"] + (["db", "dw"] if delta == 2 else ["dbeta"] if delta else [])
        ops.check_status(buf.status)
        got[lean] = {n: getattr(buf, n) for n in names}
    for lean in (1, 2):
        for n, t in got[lean].items():
            assert torch.equal(t, got[0][n]), (lean, n)
