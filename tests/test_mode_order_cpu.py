"""The planner's order of the modes (cc_plan.cpp mode_order): packed keys sorted by digits, and comparisons where the keys do
not fit 64 bits, give one segment per run of eight and one slot per distinct mode, whatever the order of the input."""
import os
import subprocess

import numpy as np

from conftest import ROOT

EXE = os.path.join(ROOT, "tests", "_build", "mode_order_check")


def _segments(modes):
    """Segments of the distinct modes: runs of up to 8 consecutive last indices."""
    u = np.unique(modes, axis=0)
    count = length = 0
    for i in range(len(u)):
        follows = i and (u[i, :-1] == u[i - 1, :-1]).all() and u[i, -1] == u[i - 1, -1] + 1
        if follows and length < 8:
            length += 1
        else:
            count, length = count + 1, 1
    return count


def test_order():
    os.makedirs(os.path.dirname(EXE), exist_ok=True)
    subprocess.run(["g++", "-std=c++17", "-O1", "-o", EXE, os.path.join(ROOT, "tests", "mode_order_check.cpp"),
                    os.path.join(ROOT, "modules_b200", "csrc", "cc_plan.cpp")], check=True)
    text, want = "", []
    for d in (1, 2, 3):
        for spread in (1, 3, 1 << 10, (1 << 20) - 1, (1 << 20), (1 << 31) - 1):   # 3D: 63 bits, 66, 99
            rng = np.random.default_rng(d)
            near = np.stack(np.meshgrid(*[np.arange(-5, 6)] * d, indexing="ij"), -1).reshape(-1, d)
            modes = rng.permutation(np.concatenate([rng.integers(-spread, spread + 1, (150, d)), near, near[::2],
                                                    [[-spread] * d, [spread] * d]]))
            V = rng.integers(1, 9, len(modes)).astype(float)
            for o in (np.arange(len(modes)), np.lexsort(modes.T[::-1])):
                text += f"{d} {len(V)}\n" + "".join(" ".join(map(str, m)) + f" {v}\n" for m, v in zip(modes[o].tolist(), V[o]))
                want.append([_segments(modes), len(np.unique(modes, axis=0)), V.sum()])
    r = subprocess.run([EXE], input=text, capture_output=True, text=True, check=True)
    assert [[float(x) for x in line.split()] for line in r.stdout.splitlines()] == want
