"""The rules that fit a launch's tile to a block's shared memory
(launch_rules.hpp), checked on the CPU over every grid size and both element
sizes (tests/cpp/launch_rules_check.cpp)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_launch_rules(tmp_path):
    exe = tmp_path / "launch_rules_check"
    csrc = os.path.join(ROOT, "mlfma_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{csrc}", os.path.join(ROOT, "tests", "cpp", "launch_rules_check.cpp"),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and "ALL OK" in out.stdout, out.stdout + out.stderr
