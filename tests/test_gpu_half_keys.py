"""64 key channels without the delta term: the kernels leave the other half of the tiles and records out.  What they give is, bit
for bit, what 128 channels give whose second half is zero."""
import pytest
import torch
import torch.nn.functional as F

from lethe_b200 import ops
from lethe_b200.synth import make_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gate", ["scalar", "none"])
@pytest.mark.parametrize("V", [64, 128])
@pytest.mark.parametrize("B,H,L,f16", [(1, 1, 64, False), (1, 2, 63, True), (2, 3, 1000, False), (1, 40, 130, True), (3, 100, 257, False)])
def test_same_bits_as_padded_keys(gate, V, B, H, L, f16):
    dev = torch.device("cuda")
    inp = make_inputs(B, L, H, 64, V, gate=gate, delta=False, seed=L, mild=True)
    dhT = 0.1 * torch.randn(B, H, 64, V, generator=torch.Generator().manual_seed(2))

    def run(pad):
        wide = lambda t, at: F.pad(t, (0, 0, 0, 64) if at == "rows" else (0, 64)) if pad else t
        d = {"q": wide(inp["q"], ""), "k": wide(inp["k"], ""), "v": inp["v"], "h0": wide(inp["h0"], "rows")}
        if gate == "scalar":
            d["g"] = inp["g"]
        if f16:
            d["q"], d["k"] = d["q"].half(), d["k"].half()
        d = {n: t.to(dev).requires_grad_(True) for n, t in d.items()}
        with torch.no_grad():
            o2, hT2 = ops.gdn_chunk(d["q"], d["k"], d["v"], d.get("g"), None, d["h0"], scale=0.125)
        o, hT = ops.gdn_chunk(d["q"], d["k"], d["v"], d.get("g"), None, d["h0"], scale=0.125)
        grads = torch.autograd.grad((o, hT), list(d.values()), (inp["do"].to(dev), wide(dhT, "rows").to(dev)))
        out = {"o": o.detach(), "hT": hT.detach()[:, :, :64], "o2": o2, "hT2": hT2[:, :, :64]}
        for n, t in zip(d, grads):
            out["d" + n] = t[..., :64] if n in ("q", "k") else t[:, :, :64] if n == "h0" else t
        return out

    got, ref = run(False), run(True)
    for n, t in got.items():
        assert torch.equal(t, ref[n]), n
