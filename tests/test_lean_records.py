"""Which records a lean call leaves for a partial one (``kernel_mask``) on the same workspaces: what the contract says, and what it promises."""
import os

import pytest
import torch

from lethe_b200 import ops
from lethe_b200.synth import make_inputs


def test_the_contract_says_which_records_a_lean_call_leaves_out():
    with open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "include", "lethe_gdn.h")) as f:
        text = f.read()
    mask = text[text.index("Profiling aid:"):text.index("uint32_t kernel_mask;")]
    assert "lethe_gdn_joint_scans" in mask and "leaves no RB" in " ".join(mask.split()) and "no Hc" in mask


@pytest.mark.gpu
@pytest.mark.parametrize("delta", [0, 1])
def test_partial_calls_go_on_from_a_full_call_that_leaves_every_record(delta):
    """Kernels run again one by one behind a full call without ``lean``: the same results."""
    K, V, BH, L, dev = 128, 128, 64, 192, torch.device("cuda")
    inp = make_inputs(1, L, BH, K, V, gate="channel", delta=bool(delta), seed=3, mild=True)
    args = [None if inp[n] is None else inp[n].to(dev) for n in ("q", "k", "v", "g", "beta", "h0")]
    do = inp["do"].to(dev)
    buf = ops.GdnBuffers(1, L, BH, K, V, ops.GATE_CHANNEL, delta, dev)
    ops.forward_into(buf, *args, K ** -0.5)
    ops.backward_into(buf, *args, do, None, K ** -0.5)
    names = ["o", "hT", "dq", "dk", "dv", "dg", "dh0"] + (["dbeta"] if delta else [])
    ref = {n: getattr(buf, n).clone() for n in names}
    for again in (lambda: ops.forward_into(buf, *args, K ** -0.5, 4, lean=2), lambda: ops.forward_into(buf, *args, K ** -0.5, 2, lean=1),
                  lambda: ops.backward_into(buf, *args, do, None, K ** -0.5, 2, lean=1), lambda: ops.backward_into(buf, *args, do, None, K ** -0.5, 12)):
        again()
    torch.cuda.synchronize()
    ops.check_status(buf.status)
    for n in names:
        assert torch.equal(getattr(buf, n), ref[n]), n
