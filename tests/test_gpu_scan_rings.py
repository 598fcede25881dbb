"""The state scan without the delta term takes rings of 8, 16 or 32 records by the length of a call and the number of its CTAs, other
ones for parts of the pairs and for ranges of the chunks: the same bits on either side of every line."""
import pytest
import torch

from lethe_b200 import ops
from lethe_b200.synth import make_inputs

pytestmark = pytest.mark.gpu

RANGES = {5: [(0, 4), (4, 1)], 8: [(0, 7), (7, 1)], 9: [(0, 8), (8, 1)], 16: [(0, 7), (7, 9)], 17: [(0, 1), (1, 16)], 33: [(0, 8), (8, 9), (17, 16)]}


@pytest.mark.parametrize("NT", [1, 4, 5, 8, 9, 16, 17, 33])
@pytest.mark.parametrize("V,BH", [(128, 18), (128, 37), (128, 38), (64, 75)])
def test_parts_and_ranges_give_the_bits_of_the_whole(V, BH, NT):
    K, L, dev = 128, 64 * NT, torch.device("cuda")
    inp = make_inputs(1, L, BH, K, V, gate="scalar", delta=False, seed=NT, mild=True)
    d = {n: t.to(dev) for n, t in inp.items() if t is not None}
    dhT = 0.1 * torch.randn(1, BH, K, V, generator=torch.Generator().manual_seed(1)).to(dev)
    args = (d["q"], d["k"], d["v"], d["g"], None, d["h0"])
    whole, parts, ranges = (ops.GdnBuffers(1, L, BH, K, V, ops.GATE_SCALAR, False, dev) for _ in range(3))
    ops.forward_into(whole, *args, K ** -0.5)
    ops.backward_into(whole, *args, d["do"], dhT, K ** -0.5)
    for rng in ((0, 1), (1, BH - 1)):
        ops.forward_into(parts, *args, K ** -0.5, bh_range=rng)
        ops.backward_into(parts, *args, d["do"], dhT, K ** -0.5, bh_range=rng)
    for m in (1, 2, 4):
        for cr in RANGES.get(NT, [(0, 0)]):
            ops.forward_into(ranges, *args, K ** -0.5, m, c_range=cr)
    for m in (1, 2, 4):
        for cr in reversed(RANGES.get(NT, [(0, 0)])):
            ops.backward_into(ranges, *args, d["do"], dhT, K ** -0.5, m, c_range=cr)
    torch.cuda.synchronize()
    for b in (parts, ranges):
        ops.check_status(b.status)
        for n in ("o", "hT", "dq", "dk", "dv", "dg", "dh0"):
            assert torch.equal(getattr(b, n), getattr(whole, n)), n


@pytest.mark.parametrize("V,H", [(64, 149), (128, 75)])
@pytest.mark.parametrize("L", [50, 500, 570, 1030])
def test_parts_of_the_heads_with_64_key_channels(V, H, L):
    dev = torch.device("cuda")
    inp = make_inputs(1, L, H, 64, V, gate="scalar", delta=False, seed=L, mild=True)
    dhT = 0.1 * torch.randn(1, H, 64, V, generator=torch.Generator().manual_seed(2))

    def run(heads):
        cut = lambda n: inp[n][:, heads] if n == "h0" else inp[n][:, :, heads]
        d = {n: cut(n).contiguous().to(dev).requires_grad_(True) for n in ("q", "k", "v", "g", "h0")}
        o, hT = ops.gdn_chunk(d["q"], d["k"], d["v"], d["g"], None, d["h0"])
        grads = torch.autograd.grad((o, hT), list(d.values()), (inp["do"][:, :, heads].to(dev), dhT[:, heads].to(dev)))
        return {"o": o.detach(), "hT": hT.detach(), **{"d" + n: t for n, t in zip(d, grads)}}

    whole = run(slice(0, H))
    for heads in (slice(0, 1), slice(1, H)):
        for n, t in run(heads).items():
            assert torch.equal(t, whole[n][:, heads] if n in ("hT", "dh0") else whole[n][:, :, heads]), n
