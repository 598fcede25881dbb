"""Sizes at the edges of the kernels' dispatch rules and work splits, against the token-serial fp64 oracle (reference
``gdn_backward.py:16-57``)."""
import pytest
import torch

from lethe_b200 import ops
from lethe_b200.synth import make_inputs
from oracle.gdn_oracle import scale_rel, serial_forward

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
