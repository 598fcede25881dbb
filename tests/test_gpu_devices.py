"""GPU: an input on another device is refused on the host.  Its pointer would fault in a kernel."""
import pytest
import torch

from lethe_b200 import ops
from lethe_b200.synth import make_inputs

pytestmark = pytest.mark.gpu


def _inputs():
    inp = make_inputs(1, 64, 2, 128, 64, gate="channel", delta=True, seed=1)
    d = {n: t.cuda() for n, t in inp.items()}
    d["b"] = d["beta"][..., None].expand(1, 64, 2, 128).contiguous()
    d["w"] = d["beta"][..., None].expand(1, 64, 2, 64).contiguous()
    d["qn"] = d["kn"] = d["q"].half()
    d.update({n + "1": d[n][:, 0].contiguous() for n in ("q", "k", "v", "g", "beta")})
    return d


def _buffers(*t, backward=False):
    buf = ops.GdnBuffers(1, 64, 2, 128, 64, ops.GATE_CHANNEL, True, torch.device("cuda"))
    ops.backward_into(buf, *t, None, 0.1) if backward else ops.forward_into(buf, *t, 0.1)


CALLS = {
    "gdn_chunk": (ops.gdn_chunk, ("q", "k", "v", "g", "beta", "h0")),
    "gdn_chunk_full": (ops.gdn_chunk_full, ("q", "k", "v", "g", "b", "w", "h0")),
    "gdn2_op": (ops.gdn2_op, ("q", "k", "v", "g", "b", "w")),
    "gate_regime": (ops.gate_regime, ("g", "b", "w")),
    "gdn_decode_step": (ops.gdn_decode_step, ("q1", "k1", "v1", "g1", "beta1", "h0")),
    "l2norm_qk": (ops.l2norm_qk, ("q", "k")),
    "l2norm_qk_vjp_raw": (ops.l2norm_qk_vjp_raw, ("q", "k", "qn", "kn")),
    "forward_into": (_buffers, ("q", "k", "v", "g", "beta", "h0")),
    "backward_into": (lambda *t: _buffers(*t, backward=True), ("q", "k", "v", "g", "beta", "h0", "do")),
}


@pytest.mark.parametrize("call,away", [(c, n) for c, (_, names) in sorted(CALLS.items()) for n in names])
def test_an_input_on_the_host_is_refused(call, away):
    f, names = CALLS[call]
    d = _inputs()
    d[away] = d[away].cpu()
    with pytest.raises(ops.GdnError, match="CUDA device"):
        f(*(d[n] for n in names))
