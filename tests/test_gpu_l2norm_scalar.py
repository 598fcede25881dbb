"""Normalisation of q and k inside the prepare kernels for one decay or none, against rows normalised by the kernel of its own.  Both
round the same fp32 values to fp16, whose sums of squares are taken in another order: a few values at a tie differ, and with
them some of the bf16 results, each by a rounding, 2^-8 of its value at most."""
import pytest
import torch

from lethe_b200 import ops
from lethe_b200.synth import make_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gate,delta", [("scalar", True), ("scalar", False), ("none", True), ("none", False)])
@pytest.mark.parametrize("K,V,dtype", [(128, 64, torch.bfloat16), (128, 128, torch.float16), (64, 64, torch.float16), (64, 128, torch.bfloat16)])
@pytest.mark.parametrize("B,H,L", [(1, 1, 1), (2, 3, 191), (1, 160, 200)])
def test_as_rows_normalised_before(gate, delta, K, V, dtype, B, H, L):
    dev = torch.device("cuda")
    inp = make_inputs(B, L, H, K, V, gate=gate, delta=delta, seed=L, mild=True)
    gen = torch.Generator().manual_seed(7)
    q, k = (torch.randn(B, L, H, K, generator=gen).mul_(3.0).to(dev, dtype).requires_grad_(True) for _ in range(2))
    rest = [None if inp[n] is None else inp[n].to(dev).requires_grad_(True) for n in ("v", "g", "beta", "h0")]
    do = inp["do"].to(dev)

    def both(f):
        with torch.no_grad():
            o2, hT2 = f()
        o, hT = f()
        wrt = [q, k] + [t for t in rest if t is not None]
        return [o2, hT2, o.detach(), hT.detach(), *torch.autograd.grad(o, wrt, do)]

    got = both(lambda: ops.gdn_chunk(q, k, *rest, use_qk_l2norm=True))
    ref = both(lambda: ops.gdn_chunk(*ops.l2norm_qk(q, k), *rest))
    for n, (a, b) in enumerate(zip(got, ref)):
        a, b = a.float(), b.float()
        assert (a - b).norm() <= 2 ** -8 * b.norm(), n
    assert torch.equal(got[0], got[2]) and torch.equal(got[1], got[3])


def test_a_row_of_zeros_stays_one():
    dev = torch.device("cuda")
    inp = make_inputs(1, 64, 1, 128, 64, gate="scalar", delta=True, seed=1)
    q, k = (torch.randn(1, 64, 1, 128, device=dev, dtype=torch.bfloat16) for _ in range(2))
    q[:, 5] = 0
    k[:, 6] = 0
    o, _ = ops.gdn_chunk(q, k, *(inp[n].to(dev) for n in ("v", "g", "beta")), use_qk_l2norm=True)
    assert torch.isfinite(o.float()).all() and bool((o[:, 5] == 0).all())
