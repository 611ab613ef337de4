"""What a handle's first evaluations take: the arrays of the line plan are there from the first FP64 evaluation on, not from the
handle's creation (sets evaluated in mixed precision alone never need them)."""
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

# (in a process of its own: what earlier handles gave back to the driver counts for nothing)
MEASURE = """
import numpy as np, torch
import modules_b200 as cc
d, N, count = 2, 20000, 80
basis = np.eye(d) * N ** (1.0 / d)
modes, V = cc.stealthy_kset(d, basis, N, 0.2)
nslot = cc.CCPotential(d, basis, modes, V).plan_info(N)["nseg"] * 8
torch.cuda.synchronize()
def handles(m):
    before = torch.cuda.mem_get_info()[0]
    made = [cc.CCPotential(d, basis, modes[:m], V[:m]) for _ in range(count)]
    return made, (before - torch.cuda.mem_get_info()[0]) / count
used, _ = handles(1)        # (take up what the first handle gave back)
small, apart = handles(1)   # what a handle takes apart from its set (a stream)
pots, each = handles(len(V))
print(each - apart, nslot, len(V), count)
"""


def test_handles_hold_no_line_arrays_before_fp64(gpu):
    r = subprocess.run([sys.executable, "-c", MEASURE], capture_output=True, text=True, cwd=ROOT, timeout=300)
    assert r.returncode == 0, r.stderr
    each, nslot, M, count = (float(x) for x in r.stdout.split())
    # slots: rho, u and a weight; modes: rho and a slot number; segments 20 bytes; tables and rounding a tenth
    expected = 1.1 * (nslot * 40 + M * 20 + nslot / 8 * 20)
    print(f"{each:.0f} bytes a handle, expected {expected:.0f} (and up to 4 MB for all)")
    assert each <= expected + (4 << 20) / count


def test_first_fp64_evaluation_after_mixed_ones(gpu):
    d, N = 2, 2000
    basis = np.eye(d) * N ** (1.0 / d)
    modes, V = gpu.stealthy_kset(d, basis, N, 0.2)
    frac = np.random.default_rng(1).random((N, d))
    a, b = gpu.CCPotential(d, basis, modes, V), gpu.CCPotential(d, basis, modes, V)
    a.set_configuration(frac)
    b.set_configuration(frac)
    b.energy(gpu.PREC_MIXED)
    b.energy_and_forces(gpu.PREC_MIXED)
    (E0, F0), (E1, F1) = a.energy_and_forces(), b.energy_and_forces()
    assert E0 == E1 and np.array_equal(F0, F1)
