"""Both sides of the rule between the line and the segment kernels (cc_plan.cpp lines_preferred): sets with many force phases at
particle counts on either side, single and in batches, against the plain-C oracle. Tolerance: that of test_gpu_lines.py with
the phases of longer lines: |k.r| up to 2 pi 400 adds 400 / 130 times its 2e-13 to a phase, so rho errs by 2e-12 N at most and
energies and forces by 4e-12 of their scales."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _lines(d, count, half):
    m = np.zeros((2 * half + 1, d), int)
    m[:, -1] = np.arange(-half, half + 1)
    return np.concatenate([m + np.eye(d, dtype=int)[0] * i for i in range(1, count + 1)])


def _disc(r):
    g = np.stack(np.meshgrid(np.arange(r + 1), np.arange(-r, r + 1), indexing="ij"), -1).reshape(-1, 2)
    return g[((g ** 2).sum(1) <= r * r) & ((g[:, 0] > 0) | (g[:, 1] > 0))]


@pytest.mark.parametrize("d,modes,few,many", [(2, _lines(2, 8, 400), 40, 6000), (3, _lines(3, 8, 500), 100, 12000),
                                              (2, _disc(160), 100, 1500)])
def test_both_sides(gpu, d, modes, few, many):
    V = np.random.default_rng(1).uniform(0, 1, len(modes))
    basis = np.eye(d)
    k = oracle.lattice_k(basis, modes)
    kmax = np.sqrt((np.asarray(k) ** 2).sum(1)).max()
    p = gpu.CCPotential(d, basis, modes, V)
    p.set_path(gpu.PATH_SPLIT)
    assert p.plan_info(few)["nksplit"] > 1 and p.plan_info(many)["nksplit"] == 1   # segments, lines
    fracs = [np.random.default_rng(N).random((N, d)) for N in (few, many)]
    want = [oracle.port_eval(d, basis, f, k, V) for f in fracs]

    def check(E, F, N, w):
        assert abs(E - w[0]) <= 4e-12 * V.sum() * N * N
        assert np.abs(F - w[1]).max() <= 4e-12 * 4 * V.sum() * N * kmax

    for f, w in zip(fracs, want):
        p.set_configuration(f)
        for _ in range(3):
            E, F = p.energy_and_forces()
            check(E, F, len(f), w)
        assert p.energy() == E
        re, im = p.rho()
        assert max(np.abs(re - w[2]).max(), np.abs(im - w[3]).max()) <= 2e-12 * len(f)
        S = p.structure_factor(modes)
        assert np.abs(S - (w[2] ** 2 + w[3] ** 2) / len(f)).max() <= 2 * 2e-12 * len(f)
    b = gpu.CCBatch([p, p, p], [few, many, few])
    b.set_positions([fracs[0], fracs[1], fracs[0]])
    E, F = b.energy_and_forces()
    for i in (0, 1, 2):
        check(E[i], F[i], len(fracs[i % 2]), want[i % 2])
    assert E[0] == E[2] and np.array_equal(F[0], F[2])
    one = gpu.CCBatch([p], [few])
    one.set_positions([fracs[0]])
    e, f = one.energy_and_forces()
    assert e[0] == E[0] and np.array_equal(f[0], F[0])   # an instance's results do not depend on the others
