"""Keys that resemble one another (behind a SiLU or a ReLU, or around a common direction), where what is rounded once per row adds
up in the gate gradient: 2-norm errors of dg and dbeta against fp64 (reference ``gdn2_assemble.py:102-147`` for the VJP)."""
import pytest
import torch
import torch.nn.functional as F

from lethe_b200 import ops, plugins
from oracle.gdn_oracle import _chunks, chunk_backward, chunk_forward

from .wsview import report

pytestmark = pytest.mark.gpu
B, L, H, K = 1, 512, 4, 128


def half(x):
    return x.half().double()


def tr(x):
    return x.transpose(-1, -2)


def revcum(x):
    return torch.flip(torch.cumsum(torch.flip(x, [-1]), -1), [-1])


def err(got, ref):
    return ((got.double() - ref).norm() / ref.norm()).item()


def inputs(kind, gate, V):
    gen = torch.Generator().manual_seed(5)
    t = {}
    for n in ("q", "k"):
        z = torch.randn(B, L, H, K, generator=gen)
        z = F.silu(z) if kind == "silu" else F.relu(z) if kind == "relu" else z + 2 * torch.randn(1, 1, H, K, generator=gen)
        t[n] = F.normalize(z, dim=-1).bfloat16()
    t["v"], t["do"] = (torch.randn(B, L, H, V, generator=gen).bfloat16() for _ in range(2))
    t["beta"] = torch.randn(B, L, H, generator=gen).sigmoid()
    t["g"] = -0.1 * torch.rand(*((B, L, H, K) if gate == "channel" else (B, L, H)), generator=gen)
    st = chunk_forward(*(t[n].double() for n in ("q", "k", "v", "g", "beta")))
    return t, st, *chunk_backward(st, t["do"].double())


def replay(st, it, do):
    """dg of the scalar gate in fp64 with the roundings of the kernels' operands and records.  The forward's u and w are rounded in
    v_new = u - w h and in dM = -(dbv u^T + dbgk w^T) alike, and the two parts of the gate gradient cancel."""
    doc, bc, gam = _chunks(do, 64), st.beta[..., None], st.G.exp()[..., :1]
    T, A, h, dh = half(st.T), half(st.A), half(st.h[:, :, :-1]), half(it["dh"])
    u, w = half(half(T * tr(bc)) @ st.v), half(half(T * tr(bc * gam)) @ st.k)
    vn = half(u - w @ h)
    x, kdh = tr(A) @ doc, (st.G[..., -1:, :1] - st.G[..., :1]).exp() * (st.k @ dh)
    dv2, dA, dde = half(x + kdh), torch.tril(doc @ tr(vn)), (vn * kdh).sum(-1)
    dG = (st.qs * gam * (doc @ tr(h))).sum(-1) + (dA * A).sum(-1) - (vn * x).sum(-1) - dde
    dG[..., -1] += st.a[..., 0] * (dh * h).sum((-1, -2)) + dde.sum(-1)
    dw = half(-dv2 @ tr(h))
    dbgk = tr(T) @ dw
    dM = -(half(tr(T) @ dv2) @ tr(u) + half(dbgk) @ tr(w))
    e = bc * torch.tril(dM, -1) * st.ratio[..., 0] * (st.k @ tr(st.k))
    return revcum(dG + e.sum(-1) - e.sum(-2) + (bc * gam * dbgk * st.k).sum(-1))


def textbook(st, T, dv2, dw, form):
    """dg and dbeta of K#2 alone, scalar gate, with -T^T dT T^T through ``form`` (what becomes of dT and dT T^T)."""
    bc, gam = st.beta[..., None], st.G.exp()[..., :1]
    dbv, dbgk = tr(T) @ dv2, tr(T) @ dw
    dT = form(dv2 @ tr(bc * st.v) + dw @ tr(bc * gam * st.k))
    m = torch.tril(-(tr(T) @ form(dT @ tr(T))), -1) * st.ratio[..., 0] * (st.k @ tr(st.k))
    p = gam[..., 0] * (dbgk * st.k).sum(-1)
    e = bc * m
    return revcum(e.sum(-1) - e.sum(-2) + st.beta * p), (dbv * st.v).sum(-1) + p + m.sum(-1)


@pytest.mark.parametrize("gate", ["scalar", "channel"])
@pytest.mark.parametrize("V", [64, 128])
@pytest.mark.parametrize("kind", ["silu", "relu", "direction"])
def test_gate_gradients_of_the_op(kind, V, gate):
    t, st, gr, it = inputs(kind, gate, V)
    d = {n: t[n].cuda().requires_grad_(True) for n in ("q", "k", "v", "g", "beta")}
    o, _ = ops.gdn_chunk(*(d[n] for n in ("q", "k", "v", "g", "beta")), None)
    dg, dbeta = torch.autograd.grad(o, (d["g"], d["beta"]), t["do"].cuda())
    errs = {"dg": err(dg.cpu(), gr.dg), "dbeta": err(dbeta.cpu(), gr.dbeta)}
    report(f"{kind} keys, gate={gate} V={V}", errs)
    assert max(errs.values()) <= 2 ** -9, errs              # four roundings to half an fp16 unit on the way, 2^-11 each
    if gate == "scalar" and kind != "silu":
        # 1.2: what the replay leaves out (fp32 sums, the recurrences' own roundings, 5 to 11 %).  dM from dT, or from dbv v^T and
        # dbgk k^T, has smaller errors by itself and 1.25 to 1.3 here
        ref = gr.dg.transpose(1, 2).reshape(st.beta.shape)
        assert errs["dg"] <= 1.2 * err(replay(st, it, t["do"].double()), ref), errs


@pytest.mark.parametrize("V", [64, 128])
@pytest.mark.parametrize("kind", ["silu", "relu", "direction"])
def test_gate_gradients_of_k2_alone(kind, V):
    """K#2 by itself has no v_new to cancel against: its error is to be that of the textbook product with fp16 dT and dT T^T."""
    t, st, gr, it = inputs(kind, "scalar", V)
    T, dv2, dw = half(st.T), half(it["dv2"]), half(it["dw"])
    dg_ref, db_ref = textbook(st, T, dv2, dw, lambda x: x)
    dg_16, db_16 = textbook(st, T, dv2, dw, half)
    f = lambda x: x.float().cuda()      # noqa: E731
    _, _, dbeta, dg = plugins.k2_fn(f(st.k), f(st.v), f(st.beta), f(st.G[..., 0] / plugins.LN2), f(T), f(dw), f(dv2))
    errs = {"dg": err(dg.cpu(), dg_ref), "dbeta": err(dbeta.cpu(), db_ref)}
    bound = {"dg": 1.15 * err(dg_16, dg_ref), "dbeta": 1.15 * err(db_16, db_ref)}      # 15 %: fp32 sums and the decays' exp
    report(f"K#2 alone, {kind} keys V={V}", {**errs, **{n + " bound": b for n, b in bound.items()}})
    assert errs["dg"] <= bound["dg"] and errs["dbeta"] <= bound["dbeta"], (errs, bound)
