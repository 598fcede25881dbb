"""GPU: the differentiable ops under what PyTorch wraps around an autograd function."""
import pytest
import torch
import torch.autograd.forward_ad as fwd_ad

from lethe_b200 import ops
from lethe_b200.synth import make_inputs

pytestmark = pytest.mark.gpu


def _inputs(L=128, V=64, seed=6):
    inp = make_inputs(1, L, 2, 128, V, gate="channel", delta=True, seed=seed)
    d = {n: (None if t is None else t.cuda()) for n, t in inp.items()}
    d["b"] = d["beta"][..., None].expand(1, L, 2, 128).contiguous()
    d["w"] = d["beta"][..., None].expand(1, L, 2, V).contiguous()
    d["bf"], d["wf"] = d["b"] * torch.rand_like(d["b"]), d["w"] * torch.rand_like(d["w"])
    return d


# name: (op on its tensors, their names)
OPS = {
    "gdn_chunk": (lambda *t, **kw: ops.gdn_chunk(*t, **kw)[0], ("q", "k", "v", "g", "beta", "h0")),
    "gdn_chunk_full": (lambda *t, **kw: ops.gdn_chunk_full(*t, **kw)[0], ("q", "k", "v", "g", "bf", "wf", "h0")),
    "gdn2_op": (ops.gdn2_op, ("q", "k", "v", "g", "b", "w")),
    "gdn2_op, independent gates": (ops.gdn2_op, ("q", "k", "v", "g", "bf", "wf")),
}
every_op = pytest.mark.parametrize("name", sorted(OPS))


@every_op
def test_forward_mode_is_refused(name):
    """There is no forward-mode rule: an input with a tangent is refused, not answered without one."""
    op, names = OPS[name]
    d = _inputs()
    for dual in names:
        with fwd_ad.dual_level():
            args = [fwd_ad.make_dual(d[n], torch.ones_like(d[n])) if n == dual else d[n] for n in names]
            with pytest.raises(NotImplementedError, match="forward-mode"):
                op(*args)
            with torch.no_grad(), pytest.raises(NotImplementedError, match="forward-mode"):
                op(*args)
    op(*[d[n] for n in names])




@every_op
@pytest.mark.parametrize("l2norm", [False, True])
def test_hooks_that_move_saved_tensors_see_all_of_them(name, l2norm):
    """Everything the backward needs goes through the hooks, the workspace included, and may come back at any address."""
    op, names = OPS[name]
    d = _inputs()
    kw = dict(use_qk_l2norm=l2norm)
    leaves = [d[n].clone().requires_grad_(True) for n in names]
    want = torch.autograd.grad(op(*leaves, **kw), leaves, d["do"])
    packed = []

    def pack(t):
        packed.append(t.nbytes)
        return t.cpu()

    def unpack(t):                       # 512 bytes past whatever the allocator gives, which is on a 512-byte boundary
        room = torch.empty(t.nbytes + 512, dtype=torch.uint8, device="cuda")
        return room[512:].view(t.dtype).view(t.shape).copy_(t)

    for move in (unpack, lambda t: t.cuda()):
        with torch.autograd.graph.saved_tensors_hooks(pack, move):
            o = op(*leaves, **kw)
        for a, b in zip(torch.autograd.grad(o, leaves, d["do"]), want):
            assert torch.equal(a, b)
    assert max(packed) > 4 * d["q"].nbytes                 # the workspace: 100 KB and more per chunk


@every_op
def test_a_checkpointed_call_keeps_nothing_but_its_inputs_and_output(name):
    from torch.utils.checkpoint import checkpoint
    op, names = OPS[name]
    d = _inputs(L=512)
    leaves = [d[n].clone().requires_grad_(True) for n in names]
    want = torch.autograd.grad(op(*leaves), leaves, d["do"])
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    o = checkpoint(lambda *t: op(*t), *leaves, use_reentrant=False)
    assert torch.cuda.memory_allocated() - before <= o.nbytes + 4096
    for a, b in zip(torch.autograd.grad(o, leaves, d["do"]), want):
        assert torch.equal(a, b)


@every_op
@pytest.mark.filterwarnings("ignore")
def test_a_traced_call_computes(name):
    """torch.jit.trace: other inputs through the trace give what the op gives, and its gradients."""
    op, names = OPS[name]
    d, e = _inputs(), _inputs(seed=7)
    traced = torch.jit.trace(lambda *t: op(*t) * 1, tuple(d[n] for n in names), check_trace=False)
    leaves = [e[n].clone().requires_grad_(True) for n in names]
    again = [e[n].clone().requires_grad_(True) for n in names]
    o, want = traced(*leaves), op(*again)
    assert torch.equal(o, want)
    for a, b in zip(torch.autograd.grad(o, leaves, e["do"]), torch.autograd.grad(want, again, e["do"])):
        assert torch.equal(a, b)
