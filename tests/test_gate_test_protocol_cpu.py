"""CPU: the hand-over of the gate test's two device words.  The host gives a slot back as soon as it sees the verdict, and
the next call may use it on another stream; no run shows a missing fence reliably, so the order is read from the source."""
import re

from .cusource import kernel_body


def test_the_words_are_cleared_and_fenced_before_the_verdict_appears():
    body = kernel_body("gdn_gates.cu", "gate_regime_kernel")
    verdict = [m.start() for m in re.finditer(r"\(p\.flags\)\s*=", body)]
    assert len(verdict) == 1
    clears = [m.start() for m in re.finditer(r"atomicExch\(p\.work|p\.work\[1\]\s*=", body)]
    assert len(clears) == 2 and max(clears) < verdict[0]
    assert "p.work" not in body[verdict[0]:]
    assert "__threadfence_system()" in body[max(clears):verdict[0]]
