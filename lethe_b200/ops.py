"""PyTorch surface of the B200 chunked gated-delta-rule path.

``gdn_chunk`` is the differentiable op.  It keeps the argument meaning of the reference project's op
(``gdn2_op``, ``src/lethe/kernels/ops/gdn_layer.py:99-111``: token-major ``[B, L, H, D]`` tensors,
``scale`` applied to q, optional L2 normalisation of q and k) and adds what the reference only has in
its chunkwise references: an initial state in and the final state out
(``src/lethe/kernels/references/gdn2_chunkwise.py:77,157-158``).

PyTorch supplies device memory, the stream and autograd bookkeeping; every number is computed by the
CUDA library behind ``lethe_b200.native`` (there is no other path: a missing library raises).  The
differentiable ops and the decode step are one call each into the native binding (``csrc/torch_ops.cpp``).
"""

from __future__ import annotations

import ctypes
from typing import NamedTuple

import torch
from torch import Tensor
from torch.autograd.function import once_differentiable

from . import native

GATE_NONE, GATE_SCALAR, GATE_CHANNEL = 0, 1, 2


class _Dims(ctypes.Structure):
    _fields_ = [(n, ctypes.c_int32) for n in ("B", "H", "L", "K", "V", "gate", "delta")]


class _Args(ctypes.Structure):
    _fields_ = [
        ("dims", _Dims), ("scale", ctypes.c_float),
        ("q", ctypes.c_void_p), ("k", ctypes.c_void_p), ("v", ctypes.c_void_p),
        ("g", ctypes.c_void_p), ("beta", ctypes.c_void_p), ("h0", ctypes.c_void_p),
        ("o", ctypes.c_void_p), ("hT", ctypes.c_void_p),
        ("d_o", ctypes.c_void_p), ("dhT", ctypes.c_void_p),
        ("dq", ctypes.c_void_p), ("dk", ctypes.c_void_p), ("dv", ctypes.c_void_p),
        ("dg", ctypes.c_void_p), ("dbeta", ctypes.c_void_p), ("dh0", ctypes.c_void_p),
        ("saved", ctypes.c_void_p), ("saved_bytes", ctypes.c_size_t),
        ("scratch", ctypes.c_void_p), ("scratch_bytes", ctypes.c_size_t),
        ("status", ctypes.c_void_p), ("kernel_mask", ctypes.c_uint32),
        ("dbeta_write", ctypes.c_void_p),
        ("b_gate", ctypes.c_void_p), ("w_gate", ctypes.c_void_p),
        ("db_gate", ctypes.c_void_p), ("dw_gate", ctypes.c_void_p),
        ("bh_begin", ctypes.c_uint32), ("bh_count", ctypes.c_uint32), ("qk_f16", ctypes.c_uint32),
        ("c_begin", ctypes.c_uint32), ("c_count", ctypes.c_uint32),
        ("l_tokens", ctypes.c_uint32), ("k_channels", ctypes.c_uint32),
        ("lean", ctypes.c_uint32),
        ("l2_eps", ctypes.c_float), ("q_norm", ctypes.c_void_p), ("k_norm", ctypes.c_void_p),
    ]


def _workspace(nbytes: int, dev) -> Tensor:
    """Byte buffer whose first element is 1024-byte aligned (the tile images inside need it)."""
    raw = torch.empty(nbytes + 1024, dtype=torch.uint8, device=dev)
    off = (-raw.data_ptr()) % 1024
    return raw[off:off + nbytes]


def _ptr(t: Tensor | None):
    return None if t is None else t.data_ptr()


class GdnError(RuntimeError):
    pass


def _check(rc: int) -> None:
    if rc != 0:
        msg = native.lib().lethe_gdn_strerror(rc).decode()
        raise GdnError(f"lethe_gdn: {msg} (code {rc})")


def check_status(status: Tensor) -> None:
    """Raise if a device-side wait of an earlier call gave up (synchronises)."""
    code = int(status.item())
    if code != 0:
        raise GdnError(f"lethe_gdn: device-side wait timed out at site {code}; results are invalid")


def _same_device(q: Tensor, *tensors) -> None:
    """A pointer from somewhere else would fault in a kernel."""
    if not q.is_cuda:
        raise GdnError("lethe_gdn: inputs must live on a CUDA device (there is no CPU path)")
    for t in tensors:
        if t is not None and t.device != q.device:
            raise GdnError(f"lethe_gdn: all tensors must live on one CUDA device ({q.device} and {t.device})")


def _prep16(t: Tensor) -> Tensor:
    return t.to(torch.bfloat16).contiguous()


class GdnBuffers:
    """Every buffer one forward + backward of a fixed problem size needs, allocated once.  The C
    library allocates nothing: callers that must not allocate per step (a training loop, the
    benchmark) keep one of these and call ``forward_into`` / ``backward_into``."""

    def __init__(self, B, L, H, K, V, gate: int, delta: bool, device, backward: bool = True,
                 saved: Tensor | None = None, status: Tensor | None = None, qk_dtype=torch.bfloat16):
        L_ = native.lib()
        # delta: False / True (one beta per token-head), or 2 for the full op's per-channel gates b, w
        self.dims = _Dims(B, H, L, K, V, gate, int(delta))
        full = int(delta) == 2
        nsaved = L_.lethe_gdn_saved_bytes(ctypes.byref(self.dims))
        if nsaved == 0:
            raise GdnError(f"lethe_gdn: unsupported sizes B={B} H={H} L={L} K={K} V={V} "
                           "(need K = 128, V in {64, 128}, L a multiple of 64)")
        bf, f32 = torch.bfloat16, torch.float32
        self.saved = _workspace(nsaved, device) if saved is None else saved
        self.status = torch.zeros(1, dtype=torch.int32, device=device) if status is None else status
        self.o = torch.empty(B, L, H, V, dtype=bf, device=device)
        self.hT = torch.empty(B, H, K, V, dtype=f32, device=device)
        self.scratch = None
        self.db = self.dw = None
        if backward:
            self.scratch = _workspace(L_.lethe_gdn_scratch_bytes(ctypes.byref(self.dims)), device)
            self.dq = torch.empty(B, L, H, K, dtype=qk_dtype, device=device)     # the type of q, k
            self.dk = torch.empty(B, L, H, K, dtype=qk_dtype, device=device)
            self.dv = torch.empty(B, L, H, V, dtype=bf, device=device)
            gshape = (B, L, H, K) if gate == GATE_CHANNEL else (B, L, H)
            self.dg = torch.empty(gshape, dtype=f32, device=device) if gate != GATE_NONE else None
            self.dbeta = torch.empty(B, L, H, dtype=f32, device=device) if (delta and not full) else None
            self.db = torch.empty(B, L, H, K, dtype=f32, device=device) if full else None
            self.dw = torch.empty(B, L, H, V, dtype=f32, device=device) if full else None
            self.dbeta_write = None      # set to a [B, L, H] fp32 tensor to get the erase / write split
            self.dh0 = torch.empty(B, H, K, V, dtype=f32, device=device)


def forward_into(buf: GdnBuffers, q, k, v, g, beta, h0, scale: float, kernel_mask: int = 0, *,
                 b_gate=None, w_gate=None, bh_range: tuple[int, int] = (0, 0),
                 c_range: tuple[int, int] = (0, 0), lean: bool = False) -> None:
    """Enqueue the forward kernels on the current stream; results land in ``buf.o`` / ``buf.hT``.
    ``b_gate [B,L,H,K]`` / ``w_gate [B,L,H,V]`` (fp32) replace ``beta`` for buffers made with ``delta=2``.
    ``bh_range = (begin, count)`` restricts the call to those (batch, head) pairs (count 0: all),
    ``c_range = (begin, count)`` to those 64-token chunks of every sequence (the scans carry their state from
    one range to the next: forward ranges in ascending order).  ``lean``: workspace records that no kernel of the
    forward or the backward reads are not written (2: nor what only a backward reads); calls with ``kernel_mask`` that go on
    from a full one need it made without ``lean``."""
    _same_device(q, k, v, g, beta, h0, b_gate, w_gate, buf.saved)
    a = _Args(dims=buf.dims, scale=scale, q=_ptr(q), k=_ptr(k), v=_ptr(v), g=_ptr(g), beta=_ptr(beta),
              h0=_ptr(h0), o=_ptr(buf.o), hT=_ptr(buf.hT), saved=_ptr(buf.saved),
              saved_bytes=buf.saved.numel(), status=_ptr(buf.status), kernel_mask=kernel_mask,
              b_gate=_ptr(b_gate), w_gate=_ptr(w_gate), bh_begin=bh_range[0], bh_count=bh_range[1],
              qk_f16=int(q.dtype == torch.float16), c_begin=c_range[0], c_count=c_range[1], lean=int(lean))
    _check(native.lib().lethe_gdn_forward(ctypes.byref(a), torch.cuda.current_stream(q.device).cuda_stream))


def backward_into(buf: GdnBuffers, q, k, v, g, beta, h0, do, dhT, scale: float, kernel_mask: int = 0, *,
                  b_gate=None, w_gate=None, bh_range: tuple[int, int] = (0, 0),
                  c_range: tuple[int, int] = (0, 0), lean: bool = False) -> None:
    """Enqueue the backward kernels; gradients land in ``buf.dq`` ... ``buf.dh0`` (``buf.db`` / ``buf.dw``
    for the per-channel gates of buffers made with ``delta=2``).  ``kernel_mask``, ranges and ``lean`` as in the forward."""
    _same_device(q, k, v, g, beta, h0, do, dhT, b_gate, w_gate, buf.saved)
    a = _Args(dims=buf.dims, scale=scale, q=_ptr(q), k=_ptr(k), v=_ptr(v), g=_ptr(g), beta=_ptr(beta),
              h0=_ptr(h0), d_o=_ptr(do), dhT=_ptr(dhT), dq=_ptr(buf.dq), dk=_ptr(buf.dk), dv=_ptr(buf.dv),
              dg=_ptr(buf.dg), dbeta=_ptr(buf.dbeta), dh0=_ptr(buf.dh0), saved=_ptr(buf.saved),
              saved_bytes=buf.saved.numel(), scratch=_ptr(buf.scratch), scratch_bytes=buf.scratch.numel(),
              status=_ptr(buf.status), kernel_mask=kernel_mask, dbeta_write=_ptr(buf.dbeta_write),
              b_gate=_ptr(b_gate), w_gate=_ptr(w_gate), db_gate=_ptr(buf.db), dw_gate=_ptr(buf.dw),
              bh_begin=bh_range[0], bh_count=bh_range[1], qk_f16=int(q.dtype == torch.float16),
              c_begin=c_range[0], c_count=c_range[1], lean=int(lean))
    if buf.dq.dtype != q.dtype:
        raise GdnError("lethe_gdn: dq / dk buffers must have the type of q / k (make GdnBuffers with qk_dtype=)")
    _check(native.lib().lethe_gdn_backward(ctypes.byref(a), torch.cuda.current_stream(q.device).cuda_stream))


def default_cut(gate: int, V: int, NT: int, BH: int, sms: int) -> int:
    """Chunk index at which ``GdnStepGraph`` cuts every sequence: near half of its ``NT`` chunks, on a multiple of
    as many chunks as two CTAs per SM (scalar gate or none, d_v = 64) or one (otherwise) cover when every one of
    the ``BH`` (batch, head) pairs takes the same number; half where that is nothing or everything.  ``sms``: SMs.

    That unit was a wave of the chunk kernels when they ran one CTA per chunk.  They are persistent now, with one
    to four CTAs per SM, and no wave ends at the cut: the unit is where the cut lies, not a reason for it.  ``step_is_cut``
    has what a cut here is worth."""
    if NT < 8:
        return 0
    per_sm = 2 if (gate != GATE_CHANNEL and V == 64) else 1
    unit = (sms * per_sm) // BH                  # chunks of every (batch, head) pair
    if unit == 0 or unit >= NT:
        return NT // 2
    cut = max(1, int(NT / 2 / unit + 0.5)) * unit
    if cut >= NT:
        cut -= unit
    return cut if cut > 0 else NT // 2


def default_bwd_cuts(gate: int, V: int, delta: bool, NT: int, BH: int, sms: int, cut: int) -> tuple:
    """Where the backward is cut: at the forward's cut, and - scalar gate, d_v = 64, two units of ``default_cut`` at
    most - once more at half a unit, so that the last main kernel, which has nothing to hide behind, is short.
    That cut was placed when Stage B and the WY VJP were kernels of their own.  Replay in us without / with it, where it is
    made: 16 x 32 107 / 107, 8 x 64 113 / 122, 4 x 128 147 / 147.  Elsewhere a second cut at half of the first costs 1 to
    9 % (d_v = 128, 16 x 32 136 / 147; channel-wise 179 / 189; 64 x 64 763 / 797).  So it is worth nothing any more."""
    if not cut:
        return ()
    two_per_sm = gate != GATE_CHANNEL and V == 64 and delta
    unit = (sms * 2) // BH
    if two_per_sm and unit >= 2 and cut == unit and unit < NT <= 2 * unit:
        return (unit // 2, cut)
    return (cut,)


def step_is_cut(gate: int, delta: bool, NT: int, BH: int, sms: int) -> bool:
    """Whether ``GdnStepGraph`` cuts the sequences at all when it is not told.  A cut adds launches and gives up the scan of a whole
    sequence: without the delta term, and with the channel-wise gate while a CTA of its kernels has one chunk, that costs more than
    the overlap gives.  Replay in us, not cut / cut, BH x NT: SSD, d_v = 64, 4 x 32 33 / 41, 16 x 32 53 / 61, 64 x 16 91 / 98, 36 x 47 131 / 136;
    d_v = 128, 16 x 32 74 / 85, 32 x 64 231 / 240, 64 x 64 445 / 463; GLA 4 x 32 39 / 53, 16 x 32 82 / 91, 64 x 16 132 / 154, d_v = 128 32 x 64
    318 / 326; KDA 4 x 32 73 / 76, d_v = 128, 3 x 128 202 / 187, 4 x 64 125 / 129, 8 x 37 113 / 134, 16 x 32 171 / 179, 16 x 64 285 / 293; d_v = 64, 4 x 128
    209 / 173, 16 x 128 451 / 513; scalar 4 x 16 51 / 61, 4 x 32 64 / 62, 4 x 64 94 / 87, 4 x 256 324 / 273, 8 x 32 77 / 72, 8 x 128 231 / 192, 16 x 32
    109 / 107, 16 x 128 333 / 377, 36 x 47 260 / 264, 64 x 64 553 / 544; d_v = 128, 4 x 128 196 / 166, 8 x 32 86 / 92, 8 x 128 261 / 304, 16 x 32 138 / 136,
    64 x 64 714 / 763.

    Few pairs with long sequences are cut with the channel-wise gate, too: the serial scan is most of their step.  KDA, not cut / cut, d_v = 64:
    1 x 64 94 / 92, 1 x 256 255 / 239, 2 x 96 135 / 121, 3 x 64 113 / 96, 3 x 96 138 / 141, 4 x 48 100 / 90, 4 x 64 115 / 102, 4 x 72 121 / 127, but 6 x 48 104 /
    113, 8 x 32 92 / 101, 2 x 32 70 / 74; d_v = 128: 1 x 192 213 / 194, 2 x 128 172 / 151, 3 x 48 92 / 89, 4 x 40 100 / 102, 4 x 56 117 / 109.

    Otherwise the rule goes by the number of chunks in all, and is coarser than its figures.  A cut gains up to 17 % where the pairs are so few that both
    scans keep 8 columns per CTA (up to 8 pairs of d_v = 64, 4 of 128) and the sequences have 32 chunks or more, where the serial scan is
    what there is to hide; elsewhere it gives 2 % at best and costs up to 19 %.  The rule still cuts there - every scalar gate with the delta term, the
    channel-wise one from two chunks per SM on, and SSD from 4096 chunks on - as it did before whole sequences had shorter scans."""
    if not delta:
        return NT * BH >= 4096
    return gate != GATE_CHANNEL or NT * BH >= 2 * sms or (BH <= 4 and NT >= 40)


def joint_scans(gate: int, V: int, delta: bool, BH: int, sms: int, NT: int = 64) -> int:
    """Which scans of a whole lean call the library launches with the kernel beside them in one: 1 forward, 2 adjoint (bits)."""
    dims = _Dims(1, BH, 64 * NT, 128, V, gate, int(delta))
    return native.lib().lethe_gdn_joint_scans(ctypes.byref(dims), 1, sms)


def step_is_chain(gate: int, V: int, delta: bool, BH: int, sms: int, NT: int = 64) -> bool:
    """Whether one chain of whole calls is the faster captured step: where forward and backward take the scans that have the output,
    or their input, beside them (``joint_scans``).  Replay in us, overlapped with a cut / without / chain, BH x NT: KDA, d_v = 64, 64 x 16
    237 / 227 / 227, 64 x 64 799 / 791 / 777; d_v = 128 32 x 64 514 / 505 / 511, 64 x 64 975 / 923 / 904; GLA, d_v = 128, 64 x 16 181 / 173 / 164, 64 x 64
    613 / 609 / 562, 32 x 64 (not this) 326 / 318 / 326.

    Not below 8 chunks, where nothing is ever cut: the overlap hides more than the launches cost (without a cut / chain: KDA, d_v = 64, 38 x 7 84 /
    92, 100 x 1 59 / 62; d_v = 128, 100 x 2 98 / 104; GLA, d_v = 64, 100 x 2 49 / 57; d_v = 128, 46 x 4 55 / 61, 256 x 6 255 / 279)."""
    return NT >= 8 and joint_scans(gate, V, delta, BH, sms, NT) == 3


class GdnStepGraph:
    """Forward + backward of one fixed problem, captured once into a CUDA graph and replayed.

    A training step at fixed shapes calls the library with the same pointers every time; replaying the
    captured kernels removes the launch gaps between them.  Two ways to fill the SMs the serial state scans
    leave idle (a scan occupies V / 64 to V / 8 CTAs per (batch, head) pair), both bitwise
    equal to the plain chain:

    ``pipeline`` (default, but where ``step_is_chain``): only the serial chain of the step - prepare, forward scan, adjoint scan, Stage B
    and WY - stays on one stream; the output kernel and the kernel that builds the adjoint scan's input run
    on other streams of the graph beside the scans (the adjoint scan needs neither the outputs nor the
    forward scan).  ``cut`` (default: ``default_cut`` where ``step_is_cut``, about half of the chunks, for sequences of at least 8
    chunks; 0 = no cut) splits every sequence into an early and a late segment of
    chunks (``c_range`` of the C ABI): the late segment is prepared under the forward scan of the early one,
    and its Stage B and WY kernels run under the adjoint scan of the early one.  The scans hand their fp32
    state from segment to segment through the workspace.  ``bwd_cuts`` (default: ``default_bwd_cuts``) cuts the backward at
    places of its own; every further segment adds a scan prologue to the serial chain.

    ``groups > 1``: the (batch, head) pairs are cut into that many ranges and every range runs its own
    kernel chain on its own stream inside the graph (the pairs are independent recurrences).

    Inputs are read from, and results written to, the tensors given here: copy new data into them between
    replays.  Results land in ``buf`` as with ``forward_into`` / ``backward_into``.
    """

    def __init__(self, buf: GdnBuffers, q, k, v, g, beta, h0, do, dhT, scale: float, *, b_gate=None, w_gate=None,
                 groups: int = 1, pipeline: bool | None = None,
                 cut: int | None = None, bwd_cuts=None):
        self.buf = buf
        self._keep = (q, k, v, g, beta, h0, do, dhT, b_gate, w_gate)
        dev = q.device
        BH = buf.dims.B * buf.dims.H
        NT = buf.dims.L // 64
        groups = max(1, min(int(groups), BH))
        bounds = [BH * i // groups for i in range(groups + 1)]
        ranges = [(bounds[i], bounds[i + 1] - bounds[i]) for i in range(groups)]
        self.groups = groups
        if pipeline is None:
            pipeline = groups == 1 and not (cut is None and bwd_cuts is None and self._is_chain(buf, BH, NT, dev))
        self.pipeline = bool(pipeline) and groups == 1
        if cut is None:
            cut = self._default_cut(buf, NT, BH, dev)
        self.cut = int(cut) if self.pipeline and 0 < int(cut) < NT else 0
        self.segments = 2 if self.cut else 1
        if bwd_cuts is None or not self.pipeline:
            bwd_cuts = self._default_bwd_cuts(buf, NT, BH, dev, self.cut)
        self.bwd_cuts = tuple(sorted(int(c) for c in bwd_cuts))
        # kernels of one replay (and range of pairs)
        self.launches = 3 * (self.segments + len(self.bwd_cuts) + 1)
        if not self.pipeline:
            self.launches = 6 - self._joint_scans(buf, BH, NT, dev).bit_count()
        if any(c <= 0 or c >= NT for c in self.bwd_cuts) or len(set(self.bwd_cuts)) != len(self.bwd_cuts):
            raise GdnError(f"lethe_gdn: backward cuts {self.bwd_cuts} must be distinct chunk indices inside (0, {NT})")
        gates = dict(b_gate=b_gate, w_gate=w_gate, lean=True)

        def chain(rng):
            forward_into(buf, q, k, v, g, beta, h0, scale, bh_range=rng, **gates)
            backward_into(buf, q, k, v, g, beta, h0, do, dhT, scale, bh_range=rng, **gates)

        side = torch.cuda.Stream(device=dev)
        self._streams = [torch.cuda.Stream(device=dev) for _ in range(max(groups - 1, 2))]

        def fwd(mask, cr):
            forward_into(buf, q, k, v, g, beta, h0, scale, mask, c_range=cr, **gates)

        def bwd(mask, cr):
            backward_into(buf, q, k, v, g, beta, h0, do, dhT, scale, mask, c_range=cr, **gates)

        def mark(st):
            e = torch.cuda.Event()
            e.record(st)
            return e

        def pipelined():
            # The serial chain of a step is prepare(first segment) -> forward scan -> adjoint scan -> Stage B and
            # WY of the first segment; `side` carries exactly that.  Everything else hangs off it by events:
            # `other` prepares the later segment and builds the adjoint scan's input while the forward scan
            # runs, computes the outputs behind the scan, and runs Stage B / WY of the later segment under the
            # adjoint scan of the first; `third` computes the output of the last segment while the adjoint scan
            # has already started.  Every edge into a kernel with the programmatic-dependency attribute, the ones
            # from events too, is a programmatic one in the captured graph: such a kernel may start while the ones
            # it depends on still run, and waits for them itself.  Until then it reads the caller's tensors and
            # records of prepare only (the adjoint scan: P), and whatever the cuts, a kernel that has waited for
            # prepare lies in between (tests/test_launch_order_cpu.py goes through the schedule).
            other, third = self._streams[0], self._streams[1]
            segs = [(0, self.cut), (self.cut, NT - self.cut)] if self.segments == 2 else [(0, NT)]
            S = len(segs)
            # the backward may be cut at other places than the forward (its ranges only have to be visited in
            # descending order): boundaries self.bwd_cuts, ascending
            bb = [0] + list(self.bwd_cuts) + [NT]
            bsegs = [(bb[i], bb[i + 1] - bb[i]) for i in range(len(bb) - 1)]
            SB = len(bsegs)
            e_p, e_f, e_o = ([None] * S for _ in range(3))
            e_r, e_a = ([None] * SB for _ in range(2))
            with torch.cuda.stream(side):
                fwd(1, segs[0])
                e_p[0] = mark(side)
            other.wait_event(e_p[0])
            with torch.cuda.stream(other):
                for i in range(1, S):
                    fwd(1, segs[i])                          # prepare of the later segment: under the first scan
                    e_p[i] = mark(other)
                for i in reversed(range(SB)):
                    bwd(1, bsegs[i])                         # input of the adjoint scan: needs prepare and do only
                    e_r[i] = mark(other)
            for i in range(S):                               # forward scan, segment after segment
                if i:
                    side.wait_event(e_p[i])
                with torch.cuda.stream(side):
                    fwd(2, segs[i])
                    e_f[i] = mark(side)
            for i in range(S):                               # outputs behind the scan, off the serial chain
                st = third if i == S - 1 else other
                st.wait_event(e_f[i])
                with torch.cuda.stream(st):
                    fwd(4, segs[i])
                    e_o[i] = mark(st)
            for i in reversed(range(SB)):                    # adjoint scan straight behind the forward scan
                side.wait_event(e_r[i])
                with torch.cuda.stream(side):
                    bwd(2, bsegs[i])
                    e_a[i] = mark(side)
            for n, i in enumerate(reversed(range(1, SB))):   # Stage B / WY of the later segments: under the adjoint scan
                st = other if n % 2 == 0 else third
                st.wait_event(e_a[i])
                for e in e_o:
                    st.wait_event(e)
                with torch.cuda.stream(st):
                    bwd(12, bsegs[i])
            for e in e_o:
                side.wait_event(e)
            with torch.cuda.stream(side):
                bwd(12, bsegs[0])
            side.wait_event(mark(other))
            side.wait_event(mark(third))

        def step():
            if self.pipeline:
                pipelined()
                return
            if groups == 1:
                chain((0, 0))
                return
            fork = torch.cuda.Event()
            fork.record(side)
            joins = []
            for i, rng in enumerate(ranges):
                st = side if i == 0 else self._streams[i - 1]
                if i:
                    st.wait_event(fork)
                with torch.cuda.stream(st):
                    chain(rng)
                if i:
                    e = torch.cuda.Event()
                    e.record(st)
                    joins.append(e)
            for e in joins:
                side.wait_event(e)

        side.wait_stream(torch.cuda.current_stream(dev))
        with torch.cuda.stream(side):
            chain((0, 0))               # first call outside the capture: one-time driver look-ups and attributes
            side.synchronize()
            check_status(buf.status)
            self.graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(self.graph, stream=side):
                step()
        torch.cuda.current_stream(dev).wait_stream(side)

    @staticmethod
    def _default_cut(buf, NT: int, BH: int, dev) -> int:
        sms = torch.cuda.get_device_properties(dev).multi_processor_count
        if not step_is_cut(buf.dims.gate, buf.dims.delta != 0, NT, BH, sms):
            return 0
        return default_cut(buf.dims.gate, buf.dims.V, NT, BH, sms)

    @staticmethod
    def _joint_scans(buf, BH: int, NT: int, dev) -> int:
        sms = torch.cuda.get_device_properties(dev).multi_processor_count
        return joint_scans(buf.dims.gate, buf.dims.V, buf.dims.delta != 0, BH, sms, NT)

    @staticmethod
    def _is_chain(buf, BH: int, NT: int, dev) -> bool:
        sms = torch.cuda.get_device_properties(dev).multi_processor_count
        return step_is_chain(buf.dims.gate, buf.dims.V, buf.dims.delta != 0, BH, sms, NT)

    @staticmethod
    def _default_bwd_cuts(buf, NT: int, BH: int, dev, cut: int) -> tuple:
        sms = torch.cuda.get_device_properties(dev).multi_processor_count
        return default_bwd_cuts(buf.dims.gate, buf.dims.V, buf.dims.delta != 0, NT, BH, sms, cut)

    def replay(self) -> None:
        """Enqueue the captured step on the current stream."""
        self.graph.replay()


def _gate_code(g: Tensor | None) -> int:
    return GATE_NONE if g is None else (GATE_SCALAR if g.dim() == 3 else GATE_CHANNEL)


def gdn_forward_raw(q, k, v, g, beta, h0, scale: float):
    """One forward call of the library.  Inputs must be CUDA tensors: q, k (both bf16 or both fp16) and
    v (bf16) contiguous ``[B, L, H, D]``; g, beta, h0 fp32.  Returns ``(o, hT, saved, status)`` in fresh
    buffers."""
    B, L, H, K = q.shape
    buf = GdnBuffers(B, L, H, K, v.shape[-1], _gate_code(g), beta is not None, q.device, backward=False)
    forward_into(buf, q, k, v, g, beta, h0, scale)
    return buf.o, buf.hT, buf.saved, buf.status


def gdn_backward_raw(q, k, v, g, beta, h0, do, dhT, saved, status, scale: float):
    """One backward call of the library.  Returns ``(dq, dk, dv, dg, dbeta, dh0, scratch)``."""
    B, L, H, K = q.shape
    buf = GdnBuffers(B, L, H, K, v.shape[-1], _gate_code(g), beta is not None, q.device,
                     saved=saved, status=status, qk_dtype=q.dtype)
    backward_into(buf, q, k, v, g, beta, h0, do, dhT, scale)
    return buf.dq, buf.dk, buf.dv, buf.dg, buf.dbeta, buf.dh0, buf.scratch


L2_IN_F32, L2_NORM_F16 = 1, 2       # flags of the C calls


def _l2_working(q: Tensor, k: Tensor) -> tuple[Tensor, Tensor, bool]:
    """q, k as the normalisation kernels read them: both bf16 if both came as bf16, else both fp32."""
    f32 = not (q.dtype == torch.bfloat16 and k.dtype == torch.bfloat16)
    dt = torch.float32 if f32 else torch.bfloat16
    return q.to(dt).contiguous(), k.to(dt).contiguous(), f32


def l2norm_qk_raw(q: Tensor, k: Tensor, eps: float = 1e-6, norm_dtype=torch.float16) -> tuple[Tensor, Tensor]:
    """``x * rsqrt(sum x^2 + eps)`` over the last axis of q and of k in one launch (epsilon placed as in
    the reference, ``gdn_backward.py:9-10``).  The rows are formed in fp32 and rounded once: to fp16 by
    default (the operand type of the GDN kernels, which then read them unchanged; the reference rounds
    at the same point, ``gdn2_bwd_dhu_l3.py:477-479``), or to bf16 with ``norm_dtype=torch.bfloat16``."""
    _same_device(q, k)
    if q.shape != k.shape:
        raise GdnError("lethe_gdn: q and k must have the same shape")
    if norm_dtype not in (torch.float16, torch.bfloat16):
        raise GdnError("lethe_gdn: normalised rows are fp16 or bf16")
    qc, kc, f32 = _l2_working(q, k)
    qn, kn = torch.empty_like(qc, dtype=norm_dtype), torch.empty_like(kc, dtype=norm_dtype)
    D = q.shape[-1]
    flags = (L2_IN_F32 if f32 else 0) | (L2_NORM_F16 if norm_dtype == torch.float16 else 0)
    _check(native.lib().lethe_gdn_l2norm_qk(qc.data_ptr(), kc.data_ptr(), qn.data_ptr(), kn.data_ptr(),
                                            qc.numel() // D, D, flags, eps,
                                            torch.cuda.current_stream(q.device).cuda_stream))
    return qn, kn


def l2norm_qk_vjp_raw(q: Tensor, k: Tensor, dqn: Tensor, dkn: Tensor, eps: float = 1e-6) -> tuple[Tensor, Tensor]:
    """Gradients with respect to q and k given those with respect to the normalised rows (fp16 or bf16,
    as the backward kernels wrote them).  Returned in the working type of q, k (bf16 or fp32)."""
    _same_device(q, k, dqn, dkn)
    qc, kc, f32 = _l2_working(q, k)
    f16 = dqn.dtype == torch.float16 and dkn.dtype == torch.float16
    if f16:
        dqn, dkn = dqn.contiguous(), dkn.contiguous()
    else:
        dqn, dkn = _prep16(dqn), _prep16(dkn)
    dq, dk = torch.empty_like(qc), torch.empty_like(kc)
    D = q.shape[-1]
    flags = (L2_IN_F32 if f32 else 0) | (L2_NORM_F16 if f16 else 0)
    _check(native.lib().lethe_gdn_l2norm_qk_vjp(qc.data_ptr(), kc.data_ptr(), dqn.data_ptr(), dkn.data_ptr(),
                                                dq.data_ptr(), dk.data_ptr(), qc.numel() // D, D, flags, eps,
                                                torch.cuda.current_stream(q.device).cuda_stream))
    return dq, dk


class _L2NormQK(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, eps):
        ctx.save_for_backward(q, k)
        ctx.eps = eps
        return l2norm_qk_raw(q, k, eps)

    @staticmethod
    @once_differentiable
    def backward(ctx, dqn, dkn):
        q, k = ctx.saved_tensors
        dqn = torch.zeros_like(q, dtype=torch.float16) if dqn is None else dqn
        dkn = torch.zeros_like(k, dtype=torch.float16) if dkn is None else dkn
        dq, dk = l2norm_qk_vjp_raw(q, k, dqn, dkn, ctx.eps)
        return dq.to(q.dtype), dk.to(k.dtype), None


def l2norm_qk(q: Tensor, k: Tensor, eps: float = 1e-6) -> tuple[Tensor, Tensor]:
    """Differentiable L2 normalisation of q and k over the channel axis (one kernel each way).  Returns
    fp16 rows, which ``gdn_chunk`` / ``gdn_chunk_full`` take as they are."""
    return _L2NormQK.apply(q, k, eps)


class _Traced(torch.autograd.Function):
    """A call under ``torch.jit.trace``.  The tracer records the tensor operations that it sees, which of a native call are
    only the allocations of its results; an autograd function it records as a call, so this one stands around it."""

    @staticmethod
    def forward(ctx, call, scale, l2norm, *tensors):
        inner = [None if t is None else t.detach().requires_grad_(t.requires_grad) for t in tensors]
        with torch.enable_grad():
            out = getattr(native.ext(), call)(*inner, scale, l2norm)
        outs = (out,) if isinstance(out, Tensor) else out
        ctx.outs, ctx.inner = outs, [t for t in inner if t is not None and t.requires_grad]
        ctx.wanted = [t is not None and t.requires_grad for t in inner]
        detached = tuple(t.detach() for t in outs)
        return detached[0] if isinstance(out, Tensor) else detached

    @staticmethod
    @once_differentiable
    def backward(ctx, *grads):
        got = iter(torch.autograd.grad(ctx.outs, ctx.inner, grads, retain_graph=True, allow_unused=True))
        return (None, None, None, *(next(got) if w else None for w in ctx.wanted))


def gdn_chunk(q: Tensor, k: Tensor, v: Tensor, g: Tensor | None, beta: Tensor | None,
              h0: Tensor | None = None, *, scale: float | None = None,
              use_qk_l2norm: bool = False) -> tuple[Tensor, Tensor]:
    """Chunked gated delta rule, differentiable.  Returns ``(o [B,L,H,V], h_T [B,H,K,V] fp32)``.

    ``g``: per-token log decay, ``[B,L,H]`` (scalar gate), ``[B,L,H,K]`` (channel-wise) or None.
    ``beta``: ``[B,L,H]`` (erase and write gate) or None for the variants without the delta term
    (linear attention, GLA, SSD).  Gradients flow to q, k, v, g, beta and h0 (first order only: the
    backward is not itself differentiable, asking for a second derivative raises).  ``L`` need not be a
    multiple of the chunk length and d_k may be 64 or 128: the kernels read what is missing from a chunk
    as zeros, which is exact (a token with k = v = q = 0, g = 0 and beta = 0 leaves the state untouched).
    q and k are read as bf16, or as fp16 when both are given as fp16; with ``use_qk_l2norm`` they are normalised
    in fp32 and rounded once to fp16.
    """
    if not q.is_cuda:
        raise GdnError("lethe_gdn: inputs must live on a CUDA device (there is no CPU path)")
    scale = q.shape[-1] ** -0.5 if scale is None else scale
    if torch._C._is_tracing():
        return _Traced.apply("chunk", float(scale), bool(use_qk_l2norm), q, k, v, g, beta, h0)
    return native.ext().chunk(q, k, v, g, beta, h0, scale, use_qk_l2norm)


class _DecodeArgs(ctypes.Structure):
    _fields_ = [("B", ctypes.c_int32), ("H", ctypes.c_int32), ("K", ctypes.c_int32), ("V", ctypes.c_int32),
                ("gate", ctypes.c_int32), ("delta", ctypes.c_int32), ("scale", ctypes.c_float),
                ("q", ctypes.c_void_p), ("k", ctypes.c_void_p), ("v", ctypes.c_void_p),
                ("g", ctypes.c_void_p), ("beta", ctypes.c_void_p), ("state", ctypes.c_void_p),
                ("o", ctypes.c_void_p), ("in_f32", ctypes.c_uint32)]


def gdn_decode_step(q: Tensor, k: Tensor, v: Tensor, g: Tensor | None, beta: Tensor | None, state: Tensor,
                    *, scale: float | None = None) -> Tensor:
    """One token of the recurrence for every (batch, head) pair, for generation: the body of the
    reference's token loop (``src/lethe/kernels/references/gdn_backward.py:45-53``).

    ``q, k [B,H,K]``, ``v [B,H,V]``; ``g [B,H]`` (scalar gate), ``[B,H,K]`` (channel-wise) or None;
    ``beta [B,H]`` or None (no delta term); ``state [B,H,K,V]`` fp32 contiguous, **updated in place**
    (start from the ``h_T`` that ``gdn_chunk`` returned for the prompt).  Returns ``o [B,H,V]`` bf16.
    Not differentiable.  K must be 128, V 64 or 128.
    """
    return native.ext().decode_step(q, k, v, g, beta, state, state.shape[2] ** -0.5 if scale is None else scale)


def gdn_chunk_full(q: Tensor, k: Tensor, v: Tensor, g: Tensor, b: Tensor, w: Tensor, h0: Tensor | None = None, *,
                   scale: float | None = None, use_qk_l2norm: bool = False) -> tuple[Tensor, Tensor]:
    """The reference's full six-input recurrence with an initial state in and the final state out:
    ``g, b [B,L,H,K]`` (log decay and erase gate per key channel), ``w [B,L,H,V]`` (write gate per value
    channel).  Returns ``(o, h_T)``; gradients flow to all seven inputs (first order only)."""
    scale = q.shape[-1] ** -0.5 if scale is None else scale
    if torch._C._is_tracing():
        return _Traced.apply("chunk_full", float(scale), bool(use_qk_l2norm), q, k, v, g, b, w, h0)
    return native.ext().chunk_full(q, k, v, g, b, w, h0, scale, use_qk_l2norm)


# ------------------------------------------------------------------------------------------------
# The reference's own six-input surface
# ------------------------------------------------------------------------------------------------
def gate_regime(g: Tensor, b: Tensor, w: Tensor) -> tuple[bool, bool, bool]:
    """``(scalar_gate, one_beta, no_delta)`` of a six-input call, decided as the reference decides
    (``src/lethe/kernels/cute/gdn2_backward.py:53-60``): BITWISE equality along the channel axis, never
    a tolerance - a gate that is merely close to constant is a channel-wise gate.  One kernel and one
    host read for all five tests.

    scalar_gate: g is one value per token-head broadcast over the key channels;
    one_beta:    b and w are the same one value per token-head broadcast over their channels;
    no_delta:    b = 0 everywhere and w = 1 everywhere (no erase term, unit write gate)."""
    m = native.ext().gate_regime(g, b, w)
    return bool(m & 1), bool(m & 2), bool(m & 4)


def gdn2_op(q: Tensor, k: Tensor, v: Tensor, g: Tensor, b: Tensor, w: Tensor, *, scale: float | None = None,
            use_qk_l2norm: bool = True) -> Tensor:
    """Drop-in for the reference's ``gdn2_op`` (same argument list, same defaults, returns ``o``).
    First-order gradients only: the backward pass is not differentiable (the reference falls back to its
    eager path for that case, ``cute/gdn2_backward.py:92``; here a second derivative raises).

    The kernels cover the regimes the reference's native path covers (``cute/gdn2_backward.py:53-60,102-134``
    and ``cute/gdn2_family.py``): ``b`` and ``w`` both equal to one beta per token-head (gated delta rule,
    KDA), or ``b = 0, w = 1`` (no delta term); ``g`` constant over the channels (scalar gate) or not.  Independent
    per-channel ``b`` / ``w`` run the full recurrence of ``gdn_chunk_full``.  Gradients of broadcast gates are
    spread evenly over the channels, as the reference's scalar assembly does (``gdn2_assemble.py:343-345``);
    ``grad_b`` carries the erase part and ``grad_w`` the write part of the beta gradient
    (``gdn2_assemble.py:150-181``)."""
    if not q.is_cuda:
        raise GdnError("lethe_gdn: inputs must live on a CUDA device (there is no CPU path)")
    scale = q.shape[-1] ** -0.5 if scale is None else scale
    if torch._C._is_tracing():
        return _Traced.apply("six_inputs", float(scale), bool(use_qk_l2norm), q, k, v, g, b, w)
    return native.ext().six_inputs(q, k, v, g, b, w, scale, use_qk_l2norm)


class Gdn2Grads(NamedTuple):
    """Field for field the reference's result type (``src/lethe/kernels/references/gdn_backward.py:58-67``)."""
    grad_q: Tensor
    grad_k: Tensor
    grad_v: Tensor
    grad_g: Tensor
    grad_b: Tensor
    grad_w: Tensor
    grad_initial_state: Tensor | None


def gdn2_backward(q: Tensor, k: Tensor, v: Tensor, g: Tensor, b: Tensor, w: Tensor, do: Tensor, *,
                  scale: float | None = None, use_qk_l2norm: bool = True, fwd_stash=None,
                  rescale_do: bool = True) -> Gdn2Grads:
    """Drop-in for the reference's backward entry point ``gdn2_backward``
    (``src/lethe/kernels/ops/gdn_backward.py:16-57``: same positional arguments, same keywords, same
    result type), which is what its autograd function calls (``ops/gdn_layer.py:69-96``) and what its
    verifier harness takes as the candidate (``verifier/op_harness.py:714-733``).  The six gradients
    come back in the dtypes of the inputs they belong to.

    The reference function gets the inputs only, so the forward is recomputed here (the reference does
    the same, ``cute/gdn2_assemble.py:261-263``); ``fwd_stash`` is accepted and ignored.

    ``rescale_do``: the backward is linear in ``do``, and ``do`` enters the tensor cores as fp16.  With
    this flag (default) ``do`` is first divided by a power of two near its largest magnitude and the
    gradients are multiplied back, so that upstream gradients far outside the fp16 range (1e6, 1e-6)
    neither saturate nor fall into the subnormals.  Exact (a power of two), all on the device, no
    host synchronisation."""
    if do.requires_grad:
        raise GdnError("lethe_gdn: the backward is not differentiable (do.requires_grad): there is no eager "
                       "fallback to route a second derivative to (the reference declines its native path in "
                       "this case, cute/gdn2_backward.py:92)")
    do = do.detach()
    mult = None
    if rescale_do:
        amax = do.abs().amax().float()
        amax = torch.where(torch.isfinite(amax) & (amax > 0), amax, torch.ones_like(amax))
        mult = torch.exp2(torch.round(torch.log2(amax)))          # power of two: scaling is exact
        do = (do.float() / mult).to(do.dtype if do.dtype != torch.float16 else torch.float32)
    leaves = [t.detach().requires_grad_(True) for t in (q, k, v, g, b, w)]
    with torch.enable_grad():
        o = gdn2_op(*leaves, scale=scale, use_qk_l2norm=use_qk_l2norm)
    grads = torch.autograd.grad(o, leaves, do.to(o.dtype))
    if mult is not None:
        grads = tuple((t.float() * mult).to(t.dtype) for t in grads)
    return Gdn2Grads(*grads, None)
