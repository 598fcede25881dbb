"""The gate test where every warp looks at one row ahead of its batches (as many rows as one batch of all warps, and more), and just
below: one value that breaks a pattern is found wherever it is, and independent gates are told by any row."""
import pytest
import torch

from lethe_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [64, 128])
@pytest.mark.parametrize("extra", [-1, 0, 1, 20000])
def test_one_value_breaks_a_pattern_wherever_it_is(V, extra):
    dev = torch.device("cuda")
    rows = torch.cuda.get_device_properties(dev).multi_processor_count * 4 * 8 * 4 + extra
    beta = torch.rand(1, rows, 1, 1, device=dev) + 0.25
    g, b, w = (x.expand(1, rows, 1, n).contiguous() for x, n in ((-beta, 128), (beta, 128), (beta, V)))
    assert ops.gate_regime(g, b, w) == (True, True, False)
    for r in (0, 1, 4, 31, rows // 2, rows - 2, rows - 1):
        for t, want in ((g, (False, True, False)), (b, (True, False, False)), (w, (True, False, False))):
            at = (0, r, 0, t.shape[3] - 1)
            old = t[at].item()
            t[at] = old + 0.125
            assert ops.gate_regime(g, b, w) == want, r
            t[at] = old
    zero, one = torch.zeros_like(b), torch.ones_like(w)
    assert ops.gate_regime(g, zero, one) == (True, False, True)
    zero[0, rows - 1, 0, 7] = 1e-30
    assert ops.gate_regime(g, zero, one) == (True, False, False)
    rand = [torch.rand_like(t) for t in (g, b, w)]
    assert ops.gate_regime(*rand) == (False, False, False)
    rand[0] = g                                    # the last of the three only in the batches
    assert ops.gate_regime(*rand) == (True, False, False)
