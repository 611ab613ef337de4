"""CPU run of the line kernels' index arithmetic (tests/line_check.cpp): bounds, every output written once, and the sums
equal to direct ones, over cubic stealthy sets, skew and shifted sets (line centres), repeats, gaps and dense boxes."""
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT, load_golden

EXE = os.path.join(ROOT, "tests", "_build", "line_check")


@pytest.fixture(scope="module")
def line_check():
    os.makedirs(os.path.dirname(EXE), exist_ok=True)
    src = os.path.join(ROOT, "tests", "line_check.cpp")
    plan = os.path.join(ROOT, "modules_b200", "csrc", "cc_plan.cpp")
    subprocess.run(["g++", "-std=c++17", "-O2", "-o", EXE, src, plan], check=True)
    return EXE


def _run(exe, ksets):
    text = []
    for modes, V in ksets:
        modes = np.asarray(modes, np.int64).reshape(len(V), -1)
        text.append(f"{modes.shape[1]} {len(V)}")
        for m, v in zip(modes, V):
            text.append(" ".join(str(int(x)) for x in m) + f" {float(v)!r}")
    r = subprocess.run([exe], input="\n".join(text) + "\n", capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return [int(line.split("ok=")[1].split()[0]) for line in r.stdout.splitlines()]


def test_lines_stealthy_sets(ccgpu, line_check):
    ks = [ccgpu.stealthy_kset(d, np.eye(d) * N ** (1.0 / d), N, chi, t)
          for d, N, chi, t in [(2, 100, 0.30, 0), (2, 1000, 0.05, 3), (2, 7001, 0.37, 3), (2, 100000, 0.49, 0),
                               (3, 100, 0.10, 0), (3, 300, 0.30, 3), (3, 2000, 0.45, 0), (3, 20000, 0.20, 3)]]
    assert all(_run(line_check, ks))


def test_lines_other_sets(line_check):
    rng = np.random.default_rng(3)
    ks = []
    for name in ["lattice_2d_skew", "lattice_3d_skew", "fd_2d_skew", "lattice_1d"]:
        r = load_golden(name)
        ks.append((r["modes"], r["V"]))
    for d in (2, 3):
        box = np.stack(np.meshgrid(*[np.arange(-6, 7)] * d, indexing="ij"), -1).reshape(-1, d)
        ks.append((rng.permutation(box), rng.uniform(-1, 1, len(box))))                 # a full box, zero mode included
        ks.append((box + np.array([3, -40, 1000][:d]), np.ones(len(box))))              # far from the origin: centres
        skew = box.copy()
        skew[:, -1] += 5 * skew[:, 0]
        ks.append((skew, np.ones(len(skew))))                                           # centres that follow the prefix
        ks.append((rng.integers(-3, 4, (2000, d)), rng.uniform(0, 1, 2000)))            # repeats
        gaps = box[(box[:, -1] % 5 != 0) & (rng.random(len(box)) < 0.8)]
        ks.append((gaps, rng.uniform(0, 1, len(gaps))))                                 # gaps in the lines
        ks.append((rng.integers(-10 ** 6, 10 ** 6, (300, d)), np.ones(300)))            # isolated modes: segment kernels
        line = np.zeros((5000, d), np.int64)
        line[:, d - 1] = np.arange(-2500, 2500)
        ks.append((line, np.ones(5000)))                                                # one long line: segment kernels
    ok = _run(line_check, ks)
    assert ok[3] == 0 and ok[4] and ok[5] and ok[6] and ok[7]
