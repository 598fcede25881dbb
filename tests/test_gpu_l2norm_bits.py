"""One decay or none: normalisation inside the prepare kernels gives the bits of rows normalised by the kernel of its own, so a result
does not depend on where a program has its rows normalised."""
import pytest
import torch

from lethe_b200 import ops
from lethe_b200.synth import make_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gate,delta", [("scalar", True), ("scalar", False), ("none", True), ("none", False)])
@pytest.mark.parametrize("K,V,dtype", [(128, 64, torch.bfloat16), (128, 128, torch.float16), (64, 64, torch.float16), (64, 128, torch.bfloat16)])
@pytest.mark.parametrize("B,H,L", [(1, 8, 1000), (2, 3, 191), (1, 160, 200)])
def test_bits_of_rows_normalised_before(gate, delta, K, V, dtype, B, H, L):
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
        return [o2, hT2, o.detach(), hT.detach(), *torch.autograd.grad(o, [q, k] + [t for t in rest if t is not None], do)]

    got = both(lambda: ops.gdn_chunk(q, k, *rest, use_qk_l2norm=True))
    ref = both(lambda: ops.gdn_chunk(*ops.l2norm_qk(q, k), *rest))
    for n, (a, b) in enumerate(zip(got, ref)):
        assert torch.equal(a, b), n
