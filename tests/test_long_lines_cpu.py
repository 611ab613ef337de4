"""Line plans of sets whose lines are longer than a 32-bit product of tile counts can count (cc_plan.cpp line_groups)."""
import os
import subprocess

from conftest import ROOT

EXE = os.path.join(ROOT, "tests", "_build", "long_line_check")


def test_long_lines_are_shared_out():
    os.makedirs(os.path.dirname(EXE), exist_ok=True)
    subprocess.run(["g++", "-std=c++17", "-O2", "-o", EXE, os.path.join(ROOT, "tests", "long_line_check.cpp"),
                    os.path.join(ROOT, "modules_b200", "csrc", "cc_plan.cpp")], check=True)
    # six lines of nj column tiles: nj * nj / 4 passes 2^31 from nj = 92682 on
    halves = [1000, 365000, 372000, 500000]
    r = subprocess.run([EXE], input="".join(f"{h} 6\n" for h in halves), capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.split() == [w for h in halves for w in ("ok=1", f"nj={h // 4 + 1}")]
