"""GPU: the slots that gate tests of six-input calls take from a pool and give back."""
import threading

import pytest
import torch

from lethe_b200 import native, ops

pytestmark = pytest.mark.gpu


def _gates(B, L, H, V=64, seed=0):
    gen = torch.Generator().manual_seed(seed)
    g = -torch.rand(B, L, H, 1, generator=gen).expand(B, L, H, 128).contiguous().cuda()
    beta = torch.rand(B, L, H, 1, generator=gen)
    return g, beta.expand(B, L, H, 128).contiguous().cuda(), beta.expand(B, L, H, V).contiguous().cuda()


def test_a_call_refused_after_its_gate_test_gives_the_slot_back():
    """q off the 16-byte grid is refused by the normalisation, behind the gate test's launch."""
    B, L, H = 1, 64, 2
    g, b, w = _gates(B, L, H)
    k = torch.randn(B, L, H, 128, device="cuda", dtype=torch.bfloat16)
    q = torch.zeros(k.numel() + 1, device="cuda", dtype=torch.bfloat16)[1:].view_as(k)
    v = torch.randn(B, L, H, 64, device="cuda", dtype=torch.bfloat16)
    ops.gdn2_op(k, k, v, g, b, w)
    made, free = native.ext().gate_test_slots()
    assert made == free > 0
    for _ in range(3):
        with pytest.raises(ops.GdnError, match="not aligned"):
            ops.gdn2_op(q, k, v, g, b, w)
    assert native.ext().gate_test_slots() == (made, free)


def test_threads_on_streams_of_their_own_share_the_slots():
    """Every thread gets the verdict of its own gates, and there are never more slots than calls in flight."""
    scalar, kda = _gates(2, 128, 3, seed=1), _gates(2, 65, 3, seed=2)
    kda[0][1, 64, 2, 127] += 1e-9 + 1.0
    none = _gates(1, 7, 1, seed=3)
    none[1].zero_(), none[2].fill_(1.0)
    full = _gates(3, 64, 5, V=128, seed=4)
    full[2][2, 63, 4, 127] *= 0.5
    want = [(scalar, (True, True, False)), (kda, (False, True, False)), (none, (True, False, True)), (full, (True, False, False))]
    torch.cuda.synchronize()
    wrong = []

    def work(gates, verdict):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(200):
                got = ops.gate_regime(*gates)
                if got != verdict:
                    wrong.append((got, verdict))

    threads = [threading.Thread(target=work, args=a) for a in want]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    made, free = native.ext().gate_test_slots()
    assert made == free
