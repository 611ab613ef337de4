"""32-bit particle indices of the line kernels at the limit up to which they are used (cc_plan.h kLineMaxParticles)."""
import os
import subprocess

from conftest import ROOT

EXE = os.path.join(ROOT, "tests", "_build", "line_limit_check")


def test_particle_indices_stay_in_range():
    os.makedirs(os.path.dirname(EXE), exist_ok=True)
    subprocess.run(["g++", "-std=c++17", "-O2", "-o", EXE, os.path.join(ROOT, "tests", "line_limit_check.cpp")], check=True)
    r = subprocess.run([EXE], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
