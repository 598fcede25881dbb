"""GPU: log decays that are not finite, and ones above zero.  Minus infinity forgets the state; a chunk that cannot form it may answer NaN, as it
does for a NaN, but never with a number that is wrong."""
import pytest
import torch

from lethe_b200 import ops
from lethe_b200.synth import make_inputs
from oracle.gdn_oracle import scale_rel, serial_backward, serial_forward

pytestmark = pytest.mark.gpu
TOL = 5e-3
AT = 70          # the token, in the second of three chunks


@pytest.mark.parametrize("value", [float("-inf"), float("nan")])
@pytest.mark.parametrize("gate,delta,V", [("scalar", True, 64), ("scalar", True, 128), ("scalar", False, 64), ("scalar", False, 128),
                                          ("channel", True, 64), ("channel", True, 128), ("channel", False, 64),
                                          ("channel", False, 128)])
def test_a_finite_result_next_to_a_decay_that_is_not_is_right(gate, delta, V, value):
    B, L, H, K = 1, 192, 2, 128
    inp = make_inputs(B, L, H, K, V, gate=gate, delta=delta, seed=21)
    inp["g"][0, AT, 0] = value                                        # head 0 only
    names = ("q", "k", "v")
    leaves = {n: inp[n].cuda().requires_grad_(n in names) for n in ("q", "k", "v", "g", "beta", "h0") if inp[n] is not None}
    o, hT = ops.gdn_chunk(*(leaves.get(n) for n in ("q", "k", "v", "g", "beta", "h0")))
    grads = torch.autograd.grad(o, [leaves[n] for n in names], inp["do"].cuda())
    f = {n: (None if t is None else t.double()) for n, t in inp.items()}
    args = (f["q"], f["k"], f["v"], f["g"], f["beta"], f["h0"])
    o_ref, hT_ref = serial_forward(*args)[:2]
    gr = serial_backward(*args, f["do"])[2]
    for n, got, want in [("o", o, o_ref), ("hT", hT, hT_ref)] + [("d" + n, t, getattr(gr, "d" + n)) for n, t in zip(names, grads)]:
        got, want = got.detach().double().cpu(), want.double()
        number = torch.isfinite(got)
        assert torch.isfinite(want[number]).all(), n                  # never a number where there is none
        scale = want[torch.isfinite(want)].abs().max()
        assert ((got - want)[number].abs() <= TOL * scale).all(), n
        other = got[:, 1] if n == "hT" else got[:, :, 1]
        assert torch.isfinite(other).all(), n                         # the other head does not see it
        if n == "o":
            assert torch.isfinite(got[:, :64]).all()                  # nor does the chunk before


@pytest.mark.parametrize("gate,delta,V", [("scalar", True, 64), ("scalar", True, 128), ("scalar", False, 128), ("channel", True, 128),
                                          ("channel", False, 64)])
def test_log_decays_of_both_signs(gate, delta, V):
    """A log decay above zero lets the state grow; the token-serial form does, and so do the chunks."""
    B, L, H, K = 1, 192, 2, 128
    inp = make_inputs(B, L, H, K, V, gate=gate, delta=delta, seed=22)
    inp["g"] = 0.05 * torch.randn(inp["g"].shape, generator=torch.Generator().manual_seed(22))
    names = [n for n in ("q", "k", "v", "g", "beta", "h0") if inp[n] is not None]
    leaves = {n: inp[n].cuda().requires_grad_(True) for n in names}
    o, hT = ops.gdn_chunk(*(leaves.get(n) for n in ("q", "k", "v", "g", "beta", "h0")))
    grads = torch.autograd.grad(o, list(leaves.values()), inp["do"].cuda())
    f = {n: (None if t is None else t.double()) for n, t in inp.items()}
    o_ref, hT_ref, gr = serial_backward(f["q"], f["k"], f["v"], f["g"], f["beta"], f["h0"], f["do"])
    errs = {"o": scale_rel(o.detach().double().cpu(), o_ref), "hT": scale_rel(hT.detach().double().cpu(), hT_ref)}
    for n, t in zip(names, grads):
        errs["d" + n] = scale_rel(t.double().cpu(), getattr(gr, "d" + n))
    assert max(errs.values()) <= TOL, errs
