"""CPU: the order of the kernels of whole calls, with either scan apart from the kernel beside it or joint with it, and with q and k
normalised on the way: what each reads before it waits for the kernel before it is taken from the sources, reads through tensor
maps included (``test_launch_order_cpu.py`` has the captured step's schedule, and names records only)."""
import itertools
import re

import pytest

from .cusource import block, kernel_body, source
from .test_launch_order_cpu import Kernel, early_reads


def early_text(name, kernel, wait="griddep_wait();"):
    """What a kernel may execute before its wait, called lambdas included."""
    body = kernel_body(name, kernel)
    body = body[:body.index(wait)]
    lambdas = {}
    for m in reversed(list(re.finditer(r"auto (\w+) = \[&\]", body))):
        inner, end = block(body, m.end())
        lambdas[m.group(1)] = inner
        body = body[:m.start()] + body[end:]
    text = body
    for _ in list(lambdas):
        for n, inner in list(lambdas.items()):
            if re.search(r"\b%s\(" % n, text):
                text += lambdas.pop(n)
    return text


def early_maps(name, kernel):
    """Tensors read through a map before the wait: q, k, v, do, g."""
    loads = re.findall(r"\btma_(?:load|prefetch)_4d\(([^;]*)\);", early_text(name, kernel))
    return {m for a in loads for m in re.findall(r"&m(q|k|v|do|g|io)\b", a)}


NORMALISED = {"q": "q_norm", "k": "k_norm"}


def early(what):
    """Records and normalised rows that a kernel of a whole call reads before its wait."""
    if what == "output":
        return early_reads("gdn_fwd.cu", "output_kernel") | {NORMALISED[m] for m in early_maps("gdn_fwd.cu", "output_kernel") if m in NORMALISED}
    if what == "main":
        got = set()
        for main in (("gdn_bwd_main.cu", "bwd_sc_kernel"), ("gdn_cw_bwd.cu", "bwd_cw_kernel")):
            got |= early_reads(*main, after_scan=True) | {NORMALISED[m] for m in early_maps(*main) if m in NORMALISED}
        return got
    if what == "adjoint":
        return {"p"} | early_reads("gdn_scan.cu", "scan_mma_kernel", adjoint=True)
    if what in ("joint scan", "joint adjoint"):
        return early_reads("gdn_scan_io.cu", "scan_io_kernel") | {"map " + m for m in early_maps("gdn_scan_io.cu", "scan_io_kernel")}
    if what == "scan":
        return early_reads("gdn_scan.cu", "scan_mma_kernel", adjoint=False) | early_reads("gdn_scan.cu", "scan_nodelta_kernel")
    return set()


WRITES = {"prepare": {"ta", "w", "u", "p", "r", "ad", "qg", "q_norm", "k_norm"}, "scan": {"hc"}, "output": {"vn", "o"},
          "joint scan": {"hc", "vn", "o"}, "pre": {"rb"}, "adjoint": {"dh"}, "joint adjoint": {"dh"}, "main": {"dq", "dk", "dv2", "dw"}, "vjp": {"dx"}}


def chain(fwd_joint, adj_joint):
    names = ["prepare"] + (["joint scan"] if fwd_joint else ["scan", "output"])
    return names + (["joint adjoint"] if adj_joint else ["pre", "adjoint"]) + ["main", "vjp"]


@pytest.mark.parametrize("fwd_joint,adj_joint", list(itertools.product((False, True), repeat=2)))
def test_what_is_read_early_is_older_than_the_kernel_before(fwd_joint, adj_joint):
    done, last = [], None
    for what in chain(fwd_joint, adj_joint):
        k = Kernel(what, (0,), {last} if last else set())
        for a in done:
            if WRITES[a.what] & early(what):
                assert a in k.before, (a.what, what, WRITES[a.what] & early(what))
        done.append(k)
        last = k


def test_the_joint_scans_read_nothing_early():
    text = early_text("gdn_scan_io.cu", "scan_io_kernel")
    assert early("joint scan") == set()
    assert not re.search(r"p\.lay\.|tma_|bulk_|ldg|p\.(q|k|v|d_o|g|beta|h0|dhT)\b", text)


def test_what_the_other_kernels_read_through_maps_early():
    assert early_maps("gdn_fwd.cu", "output_kernel") == {"q", "v"}
    assert early_maps("gdn_bwd_main.cu", "bwd_sc_kernel") <= {"q", "k", "v", "do"}
    assert early_maps("gdn_cw_bwd.cu", "bwd_cw_kernel") <= {"q", "k", "v", "do", "g"}
    assert early("output") >= {"q_norm", "ta"} and "k_norm" not in early("output")
    # the output kernel's q is the normalised one where prepare has made it
    assert re.search(r"p\.l2_eps > 0\.f && p\.gate != LETHE_GATE_CHANNEL\) \{\s*mq = mn\.q;", source("capi.cu"))


def test_the_vjp_reads_the_gradients_behind_its_wait_and_rows_that_are_older_than_the_backward():
    body = kernel_body("gdn_l2norm.cu", "l2norm_qk_kernel")
    before, after = body.split('asm volatile("griddepcontrol.wait;" ::: "memory");')
    assert "load8<IN>(p.x[t]" in before and "p.dy" not in before and "store8" not in before
    assert "load8_16(p.dy[t]" in after
    ops = source("torch_ops.cpp")
    first = ops[ops.index("variable_list first_order("):]
    at = {s: first.index(s) for s in ("q_in.unpack(self)", "k_in.unpack(self)", "run_backward(", "LETHE_L2_EARLY", "lethe_gdn_l2norm_qk_vjp(")}
    assert max(at["q_in.unpack(self)"], at["k_in.unpack(self)"]) < at["run_backward("] < at["LETHE_L2_EARLY"] < at["lethe_gdn_l2norm_qk_vjp("]
    # rows that had to be converted behind the backward are not read early
    assert re.search(r"if \(qc\.data_ptr\(\) == q_raw\.data_ptr\(\) && kc\.data_ptr\(\) == k_raw\.data_ptr\(\)\) flags \|= LETHE_L2_EARLY;", first)


@pytest.mark.parametrize("what,record,names", [("output", "q_norm", ["prepare", "output"]), ("main", "vn", ["prepare", "joint scan", "main"])])
def test_the_check_sees_a_kernel_too_few_between(what, record, names):
    last, done = None, []
    for n in names:
        last = Kernel(n, (0,), {last} if last else set())
        done.append(last)
    writer = next(k for k in done if record in WRITES[k.what])
    assert record in early(what) and writer not in last.before
