"""A refused allocation fails its own call, and no other: the next one on any handle works."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("path", ["split", "nufft"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_the_next_call_works(gpu, path, precision):
    d, N = 2, 500
    modes, V = gpu.stealthy_kset(d, np.eye(d), N, 0.2)
    p = gpu.CCPotential(d, np.eye(d), modes, V)
    p.set_path(gpu.PATH_NUFFT if path == "nufft" else gpu.PATH_SPLIT)
    prec = gpu.PREC_MIXED if precision == "mixed" else gpu.PREC_FP64
    p.set_configuration(np.random.default_rng(1).random((N, d)))
    E, F = p.energy_and_forces(prec)
    re, im = p.rho(prec)
    one = (ctypes.c_double * 1)()
    at = ctypes.cast(one, ctypes.c_void_p)

    def refused():   # more configurations than any GPU holds; nothing of the buffers is read
        assert p._lib.cc_energy_grad_many(p.handle, 1 << 40, N, at, at, None, prec) < 0

    refused()
    E1, F1 = p.energy_and_forces(prec)
    assert E1 == E and np.array_equal(F1, F)
    refused()
    re1, im1 = p.rho(prec)
    assert np.array_equal(re1, re) and np.array_equal(im1, im)
