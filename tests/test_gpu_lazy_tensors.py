"""Tensors whose memory does not hold their values - a negated view, a tensor of zeros that has no storage - as inputs and as the
gradient of o: the results of the same values written out."""
import pytest
import torch

from lethe_b200 import ops
from lethe_b200.synth import make_inputs

pytestmark = pytest.mark.gpu

FORMS = {"negated": (torch._neg_view, torch.neg), "zeros": (lambda t: torch._efficientzerotensor(t.shape, dtype=t.dtype, device=t.device), torch.zeros_like),
         "strided": (lambda t: t.transpose(1, 2).contiguous().transpose(1, 2), torch.clone), "expanded": (lambda t: t[:1, :1].expand_as(t), lambda t: t[:1, :1].expand_as(t).clone())}


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("form", list(FORMS))
def test_the_gradient_of_o(form, dtype):
    dev, make, plain = torch.device("cuda"), *FORMS[form]
    inp = make_inputs(1, 192, 2, 128, 64, gate="scalar", delta=True, seed=4)
    d = {n: inp[n].to(dev).requires_grad_(True) for n in ("q", "k", "g", "beta", "h0")}
    v = inp["v"].to(dev, dtype).requires_grad_(True)
    do = inp["do"].to(dev, dtype)
    o, _ = ops.gdn_chunk(d["q"], d["k"], v, d["g"], d["beta"], d["h0"])
    wrt = [v, *d.values()]
    got = torch.autograd.grad(o, wrt, make(do), retain_graph=True)
    ref = torch.autograd.grad(o, wrt, plain(do))
    for a, b in zip(got, ref):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_inputs(dtype):
    dev = torch.device("cuda")
    inp = make_inputs(1, 130, 2, 128, 64, gate="scalar", delta=True, seed=5)
    q, k, v = inp["q"].to(dev, dtype), inp["k"].to(dev, dtype), inp["v"].to(dev)
    rest = [inp[n].to(dev) for n in ("g", "beta", "h0")]
    with torch.no_grad():
        for l2 in (False, True):
            got = ops.gdn_chunk(torch._neg_view(-q), torch._neg_view(-k), torch._neg_view(-v), *(torch._neg_view(-t) for t in rest), use_qk_l2norm=l2)
            ref = ops.gdn_chunk(q, k, v, *rest, use_qk_l2norm=l2)
            for a, b in zip(got, ref):
                assert torch.equal(a, b), l2


def test_gates_of_the_six_inputs():
    dev = torch.device("cuda")
    inp = make_inputs(1, 128, 2, 128, 64, gate="channel", delta=True, seed=6, full=True)
    names = ("q", "k", "v", "g", "b", "w")
    ref = ops.gdn2_op(*(inp[n].to(dev) for n in names))
    got = ops.gdn2_op(*(torch._neg_view(-inp[n].to(dev)) for n in names))
    assert torch.equal(got, ref)
