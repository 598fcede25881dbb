"""CPU: the reference arm of the benchmark runs the reference's own code or says that it cannot."""
import json
import sys

import bench
from oracle import make_ref


def test_the_reference_arm_is_unavailable_without_the_reference(monkeypatch, capsys):
    """Never a number of this repository's own port under the reference's name."""
    monkeypatch.setattr(make_ref, "import_reference", lambda: None)
    monkeypatch.setattr(sys, "argv", ["bench.py", "--impl", "reference", "--steps", "1", "--warmup", "1"])
    monkeypatch.delenv("RANK", raising=False)
    bench.main()
    lines = capsys.readouterr().out.strip().splitlines()
    assert len(lines) == 1
    line = json.loads(lines[0])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
