"""CPU: the order of the captured step's kernels.

A kernel launched with the programmatic-dependency attribute may start while the kernels it depends on still run - in a
captured graph that holds for every edge into it, the ones that come from events included - and reads some records before
it waits for them.  Which ones is taken from the sources here; the schedule of ``ops.GdnStepGraph`` is run against
stand-ins for streams and events; and every pair of kernels that touch the same record of the same chunk, one of them
writing, has to be in order, whatever the cuts.  No run could show this reliably: the early reader usually wins its race."""
import re
from types import SimpleNamespace

import pytest
import torch

from lethe_b200 import ops

from .cusource import block, kernel_body, source

MAIN = 12      # Stage B and the WY VJP


def early_reads(name, kernel, after_scan=False, adjoint=None):
    """Records that a kernel reads before its first wait for the kernel before it (as text: every branch counts, but for
    what a call does only when it has launched the adjoint scan itself)."""
    body = kernel_body(name, kernel)
    if adjoint is not None:                    # scan_mma_kernel: which of its producer's two waits comes first
        assert "if (!ADJOINT) griddep_wait();" in body and "if (ADJOINT) griddep_wait();" in body
        body = body.replace("if (%sADJOINT) griddep_wait();" % ("!" if adjoint else ""), "")
    for m in list(re.finditer(r"const unsigned char\* (\w+) = ([^;]*);", body)):        # a pointer is no read
        body = re.sub(r"\b%s\b" % m.group(1), "(%s)" % m.group(2), body.replace(m.group(0), ""))
    body = body[:body.index("griddep_wait();")]
    if not after_scan:
        body = re.sub(r"if \(p\.after_scan\) \w+\(a\);", "", body)
    lambdas = {}
    for m in reversed(list(re.finditer(r"auto (\w+) = \[&\]", body))):
        inner, end = block(body, m.end())
        lambdas[m.group(1)] = inner
        body = body[:m.start()] + body[end:]
    text = body
    for _ in list(lambdas):                    # what is called, and what that calls
        for n, inner in list(lambdas.items()):
            if re.search(r"\b%s\(" % n, text):
                text += lambdas.pop(n)
    return {r for r in re.findall(r"\bp\.lay\.(\w+)", text) if not r.startswith("sz_")}


def adjoint_early():
    """Of either kernel with a product: scan_kernel's P, as asserted below, and what scan_mma_kernel reads."""
    return {"p"} | early_reads("gdn_scan.cu", "scan_mma_kernel", adjoint=True)


def test_what_the_kernels_read_before_they_wait():
    """Before its wait a kernel may read the caller's tensors and what the prepare kernel wrote: the calls that need a
    chunk's other records all lie between prepare and the reader, on any stream."""
    for main in (("gdn_bwd_main.cu", "bwd_sc_kernel"), ("gdn_cw_bwd.cu", "bwd_cw_kernel")):
        assert early_reads(*main) == {"ta"}
        # in one call with the adjoint scan also what is older than that scan
        assert early_reads(*main, after_scan=True) <= {"ta", "vn", "hc", "dv2"}
    backward = source("capi.cu")
    backward = backward[backward.index("int lethe_gdn_backward("):]
    assert re.search(r"if \(\(m & 2u\) && \(e = launch_scan\(p, true, st\)\)\) return e;\s*p\.after_scan = \(m & 2u\) \? 1 : 0;\s*"
                     r"if \(m & 12u\)", backward)
    assert sum(s.count("after_scan =") for s in map(source, ("capi.cu", "gdn_bwd_main.cu", "gdn_cw_bwd.cu"))) == 1
    assert early_reads("gdn_fwd.cu", "output_kernel") == {"qg", "w", "ta", "u"}
    for name, kernel in (("gdn_fwd.cu", "prepare_kernel"), ("gdn_fwd.cu", "prepare_nodelta_kernel"),
                         ("gdn_scan.cu", "scan_nodelta_kernel")):
        assert early_reads(name, kernel) == set(), kernel
    for name, kernel, launch in (("gdn_bwd_pre.cu", "bwd_pre_kernel", r"bwd_pre_kernel<[^;]*<<<"),
                                 ("gdn_cw_fwd.cu", "prepare_cw_kernel", r"\bkern<<<")):
        assert "griddep_wait" not in kernel_body(name, kernel)             # launched plainly: nothing to wait for
        assert re.search(launch, source(name)) and "launch_dependent" not in source(name)
    # the scans' warp that streams P does not wait in the adjoint (on warp-level products it brings the decays along)
    assert "if (!(ADJOINT && warp == kStateWarps)) {" in kernel_body("gdn_scan.cu", "scan_kernel")
    assert early_reads("gdn_scan.cu", "scan_mma_kernel", adjoint=False) == set()
    assert adjoint_early() == {"p", "ad"}


# ---- stand-ins ---------------------------------------------------------------------------------------------------
class Kernel:
    def __init__(self, what, chunks, deps):
        self.what, self.chunks = what, chunks
        self.before = set()            # complete when it starts: what the kernels it depends on have waited for
        for k in deps:
            self.before |= k.all
        self.all = self.before | deps  # complete once it has waited


class Recorder:
    """torch.cuda as far as the step graph uses it."""

    def __init__(self):
        self.kernels, self.stack = [], [self.Stream(self)]

    class Stream:
        def __init__(self, rec):
            self.rec, self.last, self.full = rec, None, set()

        def wait_event(self, e):
            self.full |= e.nodes

        def wait_stream(self, other):
            pass

        def synchronize(self):
            pass

    class Event:
        nodes = frozenset()

        def record(self, st):
            self.nodes = frozenset(st.full | ({st.last} if st.last else set()))

    def launch(self, what, chunks):
        st = self.stack[-1]
        st.last, st.full = Kernel(what, chunks, st.full | ({st.last} if st.last else set())), set()
        self.kernels.append(st.last)


def schedule(monkeypatch, NT, cut, bwd_cuts, gate=ops.GATE_SCALAR, V=64):
    rec = Recorder()

    class Scope:
        def __init__(self, st=None):
            self.st = st

        def __enter__(self):
            rec.stack.append(self.st or rec.stack[-1])

        def __exit__(self, *a):
            rec.stack.pop()

    class Capture(Scope):
        def __init__(self, graph, stream):
            super().__init__(stream)
            rec.kernels.clear()                    # the call ahead of the capture is over by now
            for st in rec.streams:
                st.last, st.full = None, set()
            rec.side = stream

    rec.streams = []

    def stream(device=None):
        rec.streams.append(Recorder.Stream(rec))
        return rec.streams[-1]

    monkeypatch.setattr(torch.cuda, "Stream", stream)
    monkeypatch.setattr(torch.cuda, "Event", Recorder.Event)
    monkeypatch.setattr(torch.cuda, "stream", Scope)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda dev=None: rec.stack[0])
    monkeypatch.setattr(torch.cuda, "CUDAGraph", lambda: None)
    monkeypatch.setattr(torch.cuda, "graph", Capture)
    monkeypatch.setattr(ops, "check_status", lambda s: None)

    def calls(names, mask_at):
        def call(*args, **kwargs):
            mask = args[mask_at] if len(args) > mask_at else 0
            c0, cn = kwargs.get("c_range", (0, 0))
            for bit, what in names:
                if not mask or mask & bit:
                    rec.launch(what, range(c0, c0 + (cn or NT)))
        return call

    monkeypatch.setattr(ops, "forward_into", calls(((1, "prepare"), (2, "scan"), (4, "output")), 8))
    monkeypatch.setattr(ops, "backward_into", calls(((1, "pre"), (2, "adjoint"), (MAIN, "main")), 10))
    t = torch.empty(0)
    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda dev: SimpleNamespace(multi_processor_count=148))
    buf = SimpleNamespace(dims=SimpleNamespace(B=2, H=8, L=64 * NT, V=V, gate=gate, delta=1), status=None)
    ops.GdnStepGraph(buf, t, t, t, t, t, None, t, None, 1.0, cut=cut, bwd_cuts=bwd_cuts)
    return rec


# records a kernel reads early, reads after its wait, writes; "carry" and "end" belong to no chunk
READS = {"prepare": set(), "scan": {"p", "r", "ad", "carry_f"}, "output": {"qg", "w", "ta", "u", "hc"},
         "pre": {"ta", "w", "qg"}, "adjoint": {"p", "ad", "rb", "carry_b"}, "main": {"ta", "vn", "hc", "dh", "w", "u"}}
WRITES = {"prepare": {"ta", "w", "u", "p", "r", "ad", "qg"}, "scan": {"hc", "carry_f"}, "output": {"vn", "o"},
          "pre": {"rb"}, "adjoint": {"dh", "carry_b"}, "main": {"dq", "dv2", "dw"}}
SEQUENCE = {"carry_f", "carry_b"}


def check(rec, NT, early):
    def touches(k, record):
        return {0} if record in SEQUENCE else set(k.chunks)

    for n, a in enumerate(rec.kernels):
        for b in rec.kernels[n + 1:]:              # in the order of capture
            for record in (WRITES[a.what] & (READS[b.what] | WRITES[b.what])) | (READS[a.what] & WRITES[b.what]):
                if touches(a, record) & touches(b, record):
                    assert a in b.all, (a.what, a.chunks, b.what, b.chunks, record)
                    if record in early.get(b.what, ()):
                        assert a in b.before, ("early", a.what, a.chunks, b.what, b.chunks, record)
    side = rec.side
    end = side.full | ({side.last} if side.last else set())
    assert set(rec.kernels) == end | {k for e in end for k in e.all}          # the capture joins every stream
    for what in READS:                                                         # every chunk, once
        assert sorted(c for k in rec.kernels if k.what == what for c in k.chunks) == list(range(NT)), what


CUTS = [(32, None, None), (64, None, None), (1, None, None), (32, 18, (9, 18)), (32, 18, (18,)), (16, 0, None), (16, 0, (4,)), (16, 0, (4, 9)), (16, 0, (2, 7, 11)), (16, 8, None),
        (16, 8, (3,)), (16, 8, (12,)), (16, 8, (3, 9)), (16, 5, (2, 7, 11, 14)), (16, 1, (1,)), (16, 15, (15,)), (16, 15, (1, 2, 3, 4)),
        (8, 4, (1, 2, 3, 4, 5, 6, 7))]


@pytest.mark.parametrize("NT,cut,bwd_cuts", CUTS)
def test_no_kernel_of_the_captured_step_reads_what_may_still_be_written(monkeypatch, NT, cut, bwd_cuts):
    main = early_reads("gdn_bwd_main.cu", "bwd_sc_kernel") | early_reads("gdn_cw_bwd.cu", "bwd_cw_kernel")
    early = {"output": early_reads("gdn_fwd.cu", "output_kernel"), "adjoint": adjoint_early(), "main": main}
    check(schedule(monkeypatch, NT, cut, bwd_cuts), NT, early)


@pytest.mark.parametrize("early,writer", [({"main": {"ta", "vn"}}, "output"), ({"adjoint": {"p", "rb"}}, "pre")])
def test_the_check_sees_a_reader_that_starts_too_soon(monkeypatch, early, writer):
    """A main kernel that read v_new before its wait would race with the output kernels, at the default cuts too; an adjoint scan
    that read its input, with the kernel that makes it."""
    with pytest.raises(AssertionError, match="'early', '%s'" % writer):
        check(schedule(monkeypatch, 32, None, None), 32, early)
