"""The S2 form on the line kernels (targets per cell, the weights of combined sub-configurations) against the numpy restatement
of the reference's formulas in test_s2.py, which needs no reference library: particle counts around the tiles of 8 to 32,
sets with and without line centres, repeated modes, sub-configurations of every one of these sizes, many configurations in
one call. Tolerance: test_s2.py's, 1e-10 of its rounding scales."""
import numpy as np
import pytest

from test_s2 import RTOL, case, multiconfig_restatement, restatement, tol_scales

pytestmark = pytest.mark.gpu


def _set(d, N, shifted, seed):
    basis, frac, modes, V, S0 = case(d, N, 7 if d == 2 else 4, seed)
    if shifted:   # lines that lie off the origin and follow the prefix: line centres
        modes = modes.copy()
        modes[:, -1] += 4 * modes[:, 0] + 9
    return basis, frac, modes, V, S0


def _has_lines(gpu, d, basis, modes, V):
    """Sets with a line plan evaluate FP64 without force splits (plan_info names one)."""
    return gpu.CCPotential(d, basis, modes, V).plan_info(4000)["nksplit"] == 1


@pytest.mark.parametrize("shifted", [False, True])
@pytest.mark.parametrize("N", [1, 7, 8, 9, 25, 33, 129, 1200])
@pytest.mark.parametrize("d", [2, 3])
def test_s2_against_restatement(gpu, d, N, shifted):
    basis, frac, modes, V, S0 = _set(d, N, shifted, 100 + N)
    assert _has_lines(gpu, d, basis, modes, V)
    E0, F0, re, im, dS, k = restatement(basis, frac, modes, V, S0, -0.25)
    sE, sF = tol_scales(V, dS, re, im, k, N)
    p = gpu.CCPotential(d, basis, modes, V, -0.25, S0=S0)
    p.set_configuration(frac)
    for _ in range(3):   # direct, then captured
        E, F = p.energy_and_forces()
        assert abs(E - E0) <= RTOL * sE
        assert np.abs(F - F0).max() <= RTOL * sF
    assert p.energy() == E
    gre, gim = p.rho()
    assert max(np.abs(gre - re).max(), np.abs(gim - im).max()) <= RTOL * N


def test_s2_repeated_modes_against_restatement(gpu):
    basis, frac, modes, V, S0 = _set(2, 800, False, 77)
    rng = np.random.default_rng(5)
    pick = rng.choice(len(modes), 12, replace=False)
    modes = np.vstack([modes, modes[pick], modes[pick[:4]]])
    V = np.concatenate([V, rng.uniform(0.1, 1.0, 12), rng.uniform(-0.05, 0.5, 4)])
    S0 = np.concatenate([S0, rng.uniform(0.0, 2.0, 16)])
    E0, F0, re, im, dS, k = restatement(basis, frac, modes, V, S0, 0.2)
    sE, sF = tol_scales(V, dS, re, im, k, len(frac))
    p = gpu.CCPotential(2, basis, modes, V, 0.2, S0=S0)
    p.set_configuration(frac)
    E, F = p.energy_and_forces()
    assert abs(E - E0) <= RTOL * sE
    assert np.abs(F - F0).max() <= RTOL * sF


@pytest.mark.parametrize("Np", [1, 8, 9, 33, 400])
@pytest.mark.parametrize("d,nsub,shifted", [(2, 3, False), (3, 4, False), (2, 2, True)])
def test_multiconfig_against_restatement(gpu, d, nsub, shifted, Np):
    basis, frac, modes, V, S0 = _set(d, nsub * Np, shifted, 300 + nsub + Np)
    E0, F0, re, im, dS, k = multiconfig_restatement(basis, frac, modes, V, S0, 0.125, nsub)
    sE, sF = tol_scales(V, dS, np.sqrt((re * re + im * im).sum(0)), 0 * dS, k, Np)
    p = gpu.CCPotential(d, basis, modes, V, 0.125, S0=S0, nsub=nsub)
    p.set_configuration(frac)
    for _ in range(3):
        E, F = p.energy_and_forces()
        assert abs(E - E0) <= RTOL * sE
        assert np.abs(F - F0).max() <= RTOL * sF
    assert p.energy() == E


@pytest.mark.parametrize("d,nsub", [(2, 1), (3, 1), (2, 2)])
def test_s2_many_is_bitwise_single(gpu, d, nsub):
    """Several at a time for the S2 form, one at a time for sub-configurations."""
    basis, _, modes, V, S0 = _set(d, 200, False, 9)
    p = gpu.CCPotential(d, basis, modes, V, 0.1, S0=S0, nsub=nsub)
    frac = np.random.default_rng(8).random((70, 200, d))
    E, F = p.energy_grad_many(frac)
    for i in (0, 1, 2, 3, 63, 64, 69):
        p.set_configuration(frac[i])
        e, f = p.energy_and_forces()
        assert e == E[i] and np.array_equal(f, F[i])
