"""What a backward holds at most: its scratch and what the kernels write, and then - the scratch given back - what the kernels wrote
and the results that are made of it.  Not all of it at once."""
import ctypes

import pytest
import torch

from lethe_b200 import native, ops
from lethe_b200.synth import make_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("six", [False, True])
@pytest.mark.parametrize("variant", ["scalar", "kda", "ssd"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_peak_of_a_backward(variant, dtype, six):
    B, L, H, K, V, dev = 2, 2048, 8, 128, 128, torch.device("cuda")
    channel, delta = variant == "kda", variant != "ssd"
    inp = make_inputs(B, L, H, K, V, gate="channel" if channel else "scalar", delta=delta, seed=1, mild=True, with_h0=False)
    d = {n: inp[n].to(dev, dtype) for n in ("q", "k", "v")}
    d["g"] = inp["g"].to(dev)
    if six:
        wide = lambda t, n: t.to(dev).unsqueeze(-1).expand(B, L, H, n).contiguous()
        d["g"] = d["g"] if channel else wide(inp["g"], K)
        d["b"] = wide(inp["beta"], K) if delta else torch.zeros(B, L, H, K, device=dev)
        d["w"] = wide(inp["beta"], V) if delta else torch.ones(B, L, H, V, device=dev)
    elif delta:
        d["beta"] = inp["beta"].to(dev)
    d = {n: t.requires_grad_(True) for n, t in d.items()}
    do = inp["do"].to(dev, dtype)
    call = (lambda: ops.gdn2_op(*d.values(), use_qk_l2norm=True)) if six else (lambda: ops.gdn_chunk(*d.values(), *([] if delta else [None]), use_qk_l2norm=True)[0])
    for _ in range(2):
        o = call()
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        got = torch.autograd.grad(o, list(d.values()), do)
        torch.cuda.synchronize()
        peak = torch.cuda.max_memory_allocated() - before
    N = B * L * H
    dims = ops._Dims(B, H, L, K, V, ops.GATE_CHANNEL if channel else ops.GATE_SCALAR, int(delta))
    scratch = native.lib().lethe_gdn_scratch_bytes(ctypes.byref(dims))
    assert scratch > 32 << 20
    results = sum(t.numel() * t.element_size() for t in got)
    # 16-bit dq, dk, dv and do, and the gradients of the gates
    wrote = N * 2 * (2 * K + V) + N * 4 * ((K if channel else 1) + (2 if delta else 0))
    at_most = max(scratch + wrote + (N * 2 * V if dtype == torch.float32 else 0), wrote + results)
    assert peak <= at_most + (2 << 20), (peak, at_most, scratch, wrote, results)
