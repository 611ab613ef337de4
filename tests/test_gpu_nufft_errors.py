"""NUFFT evaluations after one that ended with an error half way (its particles spread, their grid not yet taken): the
results are those of a handle that saw no error, bit for bit (the path repeats bitwise)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [1, 2, 3])
def test_nufft_after_a_failed_evaluation(gpu, d):
    N = 900
    if d == 1:
        modes, V = np.arange(1, 41, dtype=np.int32).reshape(-1, 1), np.ones(40)
    else:
        modes, V = gpu.stealthy_kset(d, np.eye(d), N, 0.1)
    p = gpu.CCPotential(d, np.eye(d), modes, V)
    p.set_path(gpu.PATH_NUFFT)
    p.set_configuration(np.random.default_rng(d).random((N, d)))
    E0, F0 = p.energy_and_forces()
    # A refused allocation (more configurations than any GPU holds; nothing of the buffers is read) leaves its error behind,
    # which the next evaluation meets after its first launch.
    one = (ctypes.c_double * 1)()
    at = ctypes.cast(one, ctypes.c_void_p)
    assert p._lib.cc_energy_grad_many(p.handle, 1 << 40, N, at, at, None, gpu.PREC_FP64) < 0
    try:
        p.energy()
    except gpu.CCError:
        pass
    E1, F1 = p.energy_and_forces()
    assert E1 == E0 and np.array_equal(F1, F0)
    E2, F2 = p.energy_and_forces()   # and those of the captured evaluation
    assert E2 == E0 and np.array_equal(F2, F0)
