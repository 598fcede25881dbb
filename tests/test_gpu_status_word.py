"""GPU: what the PyTorch surface does with the status word.  A kernel whose bounded wait runs out writes its wait site there
(``tests/test_gpu_umma_toolkit.py`` has such a kernel); here the host writes it, and nothing on the GPU goes wrong."""
import ctypes

import pytest
import torch

from lethe_b200 import native, ops
from lethe_b200.synth import make_inputs

from .test_gpu_umma_toolkit import probe_lib

pytestmark = pytest.mark.gpu
SITE = 213


@pytest.fixture
def word():
    w = ctypes.c_int32.from_address(native.ext().status_address(torch.cuda.current_device()))
    torch.cuda.synchronize()
    assert w.value == 0
    yield w
    w.value = 0


def _inputs():
    inp = make_inputs(1, 128, 2, 128, 64, gate="channel", delta=True, seed=4, with_h0=False)
    d = {n: (None if t is None else t.cuda()) for n, t in inp.items()}
    d["b"] = d["beta"][..., None].expand(1, 128, 2, 128).contiguous()
    d["w"] = d["beta"][..., None].expand(1, 128, 2, 64).contiguous()
    return d


CALLS = {
    "gdn_chunk": lambda q, d: ops.gdn_chunk(q, d["k"], d["v"], d["g"], d["beta"])[0],
    "gdn_chunk_full": lambda q, d: ops.gdn_chunk_full(q, d["k"], d["v"], d["g"], d["b"], d["w"])[0],
    "gdn2_op": lambda q, d: ops.gdn2_op(q, d["k"], d["v"], d["g"], d["b"], d["w"]),
}


@pytest.mark.parametrize("call", sorted(CALLS))
def test_an_expired_wait_is_reported_by_the_next_forward_once(word, call):
    d = _inputs()
    want = CALLS[call](d["q"], d)
    word.value = SITE
    with pytest.raises(ops.GdnError, match=f"timed out at site {SITE}"):
        CALLS[call](d["q"], d)
    assert word.value == 0
    assert torch.equal(CALLS[call](d["q"], d), want)


@pytest.mark.parametrize("call", sorted(CALLS))
def test_an_expired_wait_is_reported_by_the_next_backward_from_the_autograd_thread(word, call):
    """The same error type and text, although the thread that raises it does not hold the interpreter lock."""
    d = _inputs()
    q = d["q"].clone().requires_grad_(True)
    o = CALLS[call](q, d)
    (want,) = torch.autograd.grad(o, q, d["do"], retain_graph=True)
    word.value = SITE
    with pytest.raises(ops.GdnError, match=f"timed out at site {SITE}"):
        o.backward(d["do"], retain_graph=True)
    assert word.value == 0 and q.grad is None
    assert torch.equal(torch.autograd.grad(o, q, d["do"])[0], want)


def test_a_kernel_whose_wait_ran_out_reaches_the_next_call_through_the_word(word):
    """The whole way: a test kernel waits, with a short limit, for bytes that nobody sends; its bounded wait leaves the site
    in the surface's word, which lies in host memory, without a copy or an event."""
    d = _inputs()
    trace = torch.zeros(4, dtype=torch.int32, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    assert probe_lib().lethe_probe_starved_wait(ctypes.addressof(word), 100_000, trace.data_ptr(), stream) == 0
    torch.cuda.synchronize()
    assert word.value == 101
    with pytest.raises(ops.GdnError, match="timed out at site 101"):
        CALLS["gdn_chunk"](d["q"], d)
    assert torch.isfinite(CALLS["gdn_chunk"](d["q"], d).float()).all()
