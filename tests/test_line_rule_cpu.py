"""Which sets and particle counts take the line kernels (cc_plan.cpp lines_preferred), at sets where one side is well ahead:
timings of both on B200 are in the comments."""
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

EXE = os.path.join(ROOT, "tests", "_build", "line_rule_check")


@pytest.fixture(scope="module")
def rule():
    os.makedirs(os.path.dirname(EXE), exist_ok=True)
    subprocess.run(["g++", "-std=c++17", "-O2", "-o", EXE, os.path.join(ROOT, "tests", "line_rule_check.cpp"),
                    os.path.join(ROOT, "modules_b200", "csrc", "cc_plan.cpp")], check=True)

    def run(modes, counts):
        modes = np.asarray(modes)
        text = f"{modes.shape[1]} {len(modes)} {len(counts)}\n{' '.join(map(str, counts))}\n"
        text += "\n".join(" ".join(map(str, m)) for m in modes.tolist()) + "\n"
        r = subprocess.run([EXE], input=text, capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
        return r.stdout.split()
    return run


def _ball(d, r):
    ax = np.arange(-r, r + 1)
    m = np.stack(np.meshgrid(*[ax[r:]] + [ax] * (d - 1), indexing="ij"), -1).reshape(-1, d)
    first = np.where(m[:, 0] != 0, m[:, 0], m[:, 1] if d == 2 else np.where(m[:, 1] != 0, m[:, 1], m[:, 2]))
    return m[((m ** 2).sum(1) <= r * r) & (first > 0)]


def _lines(d, count, half):
    m = np.zeros((2 * half + 1, d), int)
    m[:, -1] = np.arange(-half, half + 1)
    return np.concatenate([m + np.eye(d, dtype=int)[0] * i for i in range(1, count + 1)])


@pytest.mark.parametrize("d,N,chi", [(2, 100, 0.05), (2, 100, 0.30), (2, 500, 0.49), (2, 7001, 0.37), (2, 100000, 0.49),
                                     (3, 100, 0.05), (3, 300, 0.49), (3, 2000, 0.45), (3, 20000, 0.20), (3, 30000, 0.49)])
def test_stealthy_sets_take_lines(ccgpu, rule, d, N, chi):
    modes, _ = ccgpu.stealthy_kset(d, np.eye(d) * N ** (1.0 / d), N, chi)
    assert rule(modes, [N]) == ["11"]


def test_few_particles_with_very_many_modes(rule):
    # segments against lines, us: N = 100 41 / 108, 300 60 / 111, 3000 385 / 194; rho alone, N = 100 26 / 40
    assert rule(_ball(2, 250), [1, 100, 3000]) == ["00", "00", "11"]
    # 100 32 / 67, 300 46 / 69, 1000 105 / 79; rho alone, N = 100 20 / 28
    assert [x[0] for x in rule(_ball(3, 30), [100, 300, 1000])] == ["0", "0", "1"]
    # 100 28 / 62, 300 44 / 64, 1000 120 / 68, 5000 525 / 122
    assert [x[0] for x in rule(_lines(2, 16, 1000), [100, 300, 1000, 5000])] == ["0", "0", "1", "1"]
    # 100 18 / 61, 1000 45 / 67, 20000 574 / 352; rho alone 100 11 / 16, 5000 72 / 44
    assert rule(_lines(2, 5, 1000), [100, 1000, 5000, 20000])[0] == "00"
    assert rule(_lines(2, 5, 1000), [20000])[0] == "11"
    # one row of short lines: 100 17 / 9, 5000 30 / 17
    assert rule(_lines(2, 16, 60), [1, 100, 5000, 20000]) == ["11"] * 4
    # and sets without a line plan
    assert rule(_lines(2, 2, 300), [100]) == ["-"]
