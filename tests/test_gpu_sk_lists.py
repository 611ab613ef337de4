"""S(k) on one list of wavevectors after another, and the two ways its values leave the GPU: the pinned result buffer where it
holds no forces and the list fits it, else a copy of their own. All give the same bits; none touches the cached forces."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _circle(d, r):
    g = np.stack(np.meshgrid(*[np.arange(-r, r + 1)] * d, indexing="ij"), -1).reshape(-1, d)
    return g[((g ** 2).sum(1) <= r * r) & (g != 0).any(1)].astype(np.int32)


def _handle(gpu, d, N, seed=1):
    p = gpu.CCPotential(d, np.eye(d) * N ** (1.0 / d), _circle(d, 2), np.ones(len(_circle(d, 2))))
    p.set_configuration(np.random.default_rng(seed).random((N, d)))
    return p


@pytest.mark.parametrize("d,r", [(2, 30), (3, 8)])
def test_lists_in_turn(gpu, d, r):
    """Longer, shorter, permuted and repeated lists with one handle, in both precisions, against a new handle each."""
    rng = np.random.default_rng(2)
    full = _circle(d, r)
    p = _handle(gpu, d, 700)
    lists = [full[:40], full, full[: len(full) // 3], rng.permutation(full), np.concatenate([full[:90], full[:90]]), full[:1],
             full + np.array([0] * (d - 1) + [11], np.int32), np.array([[10 ** 6] * d, [-10 ** 6] * d], np.int32), full]
    for precision in (gpu.PREC_FP64, gpu.PREC_MIXED, gpu.PREC_FP64):
        for k in lists:
            S = p.structure_factor(k, precision)
            assert np.array_equal(S, _handle(gpu, d, 700).structure_factor(k, precision))
            assert np.array_equal(S, p.structure_factor(k, precision))


@pytest.mark.parametrize("K", [100, 1500])   # below and above N * d
def test_both_routes_and_the_cached_forces(gpu, K):
    d, N = 2, 500
    k = np.concatenate([_circle(d, 12)] * 4)[:K]
    p = _handle(gpu, d, N)
    S0 = p.structure_factor(k)           # no forces cached: the result buffer where K fits it
    E, F = p.energy_and_forces()
    S1 = p.structure_factor(k)           # forces cached
    assert np.array_equal(S0, S1)
    assert all(np.array_equal(p.force(i), F[i]) for i in (0, 1, N // 2, N - 1))
    frac = np.random.default_rng(1).random((N, d))
    phase = 2 * np.pi * frac @ k.T.astype(float)
    want = np.abs(np.exp(1j * phase).sum(0)) ** 2 / N
    # a phase errs by |k.r| 2^-53 < 2e-14, rho by N times that, S by 2 |rho| / N times rho's error with |rho| <= N
    assert np.abs(S0 - want).max() <= 2 * N * 2e-14


def test_a_new_list_costs_little_more_than_its_plan(gpu):
    """Buffers stay from one list to the next: a new list of 2500 wavevectors takes five times a repeated one (0.18 ms;
    46 times when every list had its buffers allocated anew)."""
    d, N = 2, 7001
    full = _circle(d, 40)
    full = full[(full[:, 0] > 0) | ((full[:, 0] == 0) & (full[:, 1] > 0))]
    p = _handle(gpu, d, N)
    new, again = [], []
    for i in range(12):
        k = np.random.default_rng(i).permutation(full)[: len(full) - 40]
        for times in (new, again):
            t = time.perf_counter()
            p.structure_factor(k)
            times.append(time.perf_counter() - t)
    print(f"new list {np.median(new) * 1e6:.0f} us, again {np.median(again) * 1e6:.0f} us")
    assert np.median(new[2:]) <= 16 * np.median(again[2:])
