"""bench.py's reference arm on a machine without the reference's library: one line
that says so, and exit code 0."""
import json
import os
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.dirname(HERE))
import bench  # noqa: E402
from oracle import ref_lib  # noqa: E402


def test_reference_arm_without_the_library(monkeypatch, capsys):
    monkeypatch.setattr(ref_lib, "LIB_PATH", os.path.join(HERE, "no_such_library.so"))
    monkeypatch.setattr(ref_lib, "_lib", None)
    monkeypatch.setattr(sys, "argv", ["bench.py", "--impl", "reference", "--gpus", "1", "--steps", "2", "--warmup", "3"])
    assert bench.main() == 0
    line = json.loads(capsys.readouterr().out.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
