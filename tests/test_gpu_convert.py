"""bf16 <-> fp32 of the six-input surface's fp32 activations: the values of ``Tensor.to``, whatever the length."""
import pytest
import torch

from lethe_b200 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 8, 9, 2047, 2048, 2049, 70001])
def test_same_values_as_torch(n):
    dev = torch.device("cuda")
    x = torch.randn(n, generator=torch.Generator().manual_seed(n)).to(dev)
    x = x * torch.exp2(torch.randint(-140, 120, (n,), generator=torch.Generator().manual_seed(1)).to(dev).float())
    special = torch.tensor([float("inf"), -float("inf"), 0.0, -0.0, 3.3895e38, 1e-40, 1.00390625], device=dev)
    x[:min(n, 7)] = special[:min(n, 7)]
    st = torch.cuda.current_stream().cuda_stream
    h = torch.full((n + 8,), 7.0, dtype=torch.bfloat16, device=dev)
    assert native.lib().lethe_gdn_convert(x.data_ptr(), h.data_ptr(), n, 0, st) == 0
    f = torch.full((n + 8,), 7.0, device=dev)
    assert native.lib().lethe_gdn_convert(h.data_ptr(), f.data_ptr(), n, 1, st) == 0
    assert torch.equal(h[:n], x.bfloat16()) and bool((h[n:] == 7).all())
    assert torch.equal(f[:n], x.bfloat16().float()) and bool((f[n:] == 7).all())


def test_refused():
    x = torch.zeros(64, device="cuda")
    lib, st = native.lib(), torch.cuda.current_stream().cuda_stream
    assert lib.lethe_gdn_convert(None, x.data_ptr(), 8, 1, st) == 1
    assert lib.lethe_gdn_convert(x.data_ptr(), x.data_ptr(), 0, 1, st) == 2
    assert lib.lethe_gdn_convert(x.data_ptr() + 4, x.data_ptr(), 8, 0, st) == 3
