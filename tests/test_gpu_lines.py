"""The line kernels (cc_lines.cuh: FP64 energies and forces as contractions on the FP64 matrix unit) where they can go
wrong: particle counts around the tiles of 8 to 32 particles and the splits of 8, sets whose lines need centres, sets of one
row, of several groups and of several force phases, and sets that fall back to the segment kernels, against the plain-C
oracle.

Tolerance: a phase is at most 11 + 2 products of table entries (each within 2 ulp) away from sincospi, so |d exp| <= 15
products x 2.2e-16 x sqrt(2) < 5e-15; the oracle forms k.r in Cartesian coordinates, an error of at most |k.r| 2^-53 x d
(below 2e-13 for the largest |k.r| here, 2 pi 130 x 2). rho is a sum of N phases: 5e-13 N; energies and forces follow with a
factor 2 and the sums' own rounding: 1e-12 of their scales (E ~ sum|V| N^2 / vol, F ~ 4 sum|V| N kmax / vol)."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _box(d, m):
    g = np.stack(np.meshgrid(*[np.arange(-m, m + 1)] * d, indexing="ij"), -1).reshape(-1, d)
    first = np.array([next((x for x in n if x != 0), 0) for n in g])
    return g[first > 0]


def _set(gpu, d, kind):
    rng = np.random.default_rng(7)
    if kind == "stealthy":
        return gpu.stealthy_kset(d, np.eye(d) * 400 ** (1 / d), 400, 0.45, 3)
    if kind == "centres":      # lines that follow the prefix and lie off the origin
        m = _box(d, 5)
        m[:, -1] += 4 * m[:, 0] + 9
        return m, rng.uniform(-1, 1, len(m))
    if kind == "one line row":
        m = _box(2, 3) if d == 2 else _box(3, 1)
        return m, rng.uniform(0, 1, len(m))
    if kind == "phases":       # tables beyond one force phase, several rho groups (2D)
        m = _box(2, 130)
        m = m[(m ** 2).sum(1) <= 130 ** 2]
        return m, rng.uniform(0, 1, len(m))
    m = np.concatenate([_box(d, 6), _box(d, 3), _box(d, 2)[::-1]])   # repeats, in any order
    p = rng.permutation(len(m))
    return m[p], rng.uniform(-1, 1, len(m))


@pytest.mark.parametrize("N", [1, 7, 8, 9, 16, 17, 24, 25, 32, 33, 129, 1200, 2500])
@pytest.mark.parametrize("d,kind", [(2, "stealthy"), (3, "stealthy"), (2, "centres"), (3, "centres"), (2, "one line row"),
                                    (3, "one line row"), (3, "repeats"), (2, "phases")])
def test_lines_against_oracle(gpu, d, kind, N):
    modes, V = _set(gpu, d, kind)
    if kind == "phases" and N not in (1, 25, 129):
        pytest.skip("the oracle takes its time on this set")
    basis = np.eye(d) * 2.0
    basis[-1, 0] = 0.3          # a skew cell
    frac = np.random.default_rng(N).random((N, d))
    frac[0] = 0.0               # the edges of the cell
    frac[-1] = 1.0 - 2.0 ** -53
    p = gpu.CCPotential(d, basis, modes, V, 0.25)
    p.set_path(gpu.PATH_SPLIT)
    p.set_configuration(frac)
    E, F = p.energy_and_forces()
    E0 = p.energy()
    re, im = p.rho()
    k = oracle.lattice_k(basis, modes)
    Eo, Fo, ro, io = oracle.port_eval(d, basis, frac, k, V, 0.25)
    vol, sumV = abs(np.linalg.det(basis)), np.abs(V).sum()
    kmax = np.sqrt((np.asarray(k) ** 2).sum(1)).max()
    assert max(np.abs(re - ro).max(), np.abs(im - io).max()) <= 5e-13 * N
    assert abs(E - Eo) <= 1e-12 * sumV * N * N / vol
    assert np.abs(F - Fo).max() <= 1e-12 * 4 * sumV * N * kmax / vol
    assert E0 == E              # the energy alone, summed in the same order
    E2, F2 = p.energy_and_forces()
    assert E2 == E and np.array_equal(F2, F)


def test_sets_that_stay_on_the_segment_kernels(gpu):
    """Isolated modes (no lines to speak of) and 1D sets have no line plan; their results agree with the oracle too."""
    rng = np.random.default_rng(2)
    for d in (1, 2, 3):
        modes = rng.integers(-40, 41, (300, d))
        V = rng.uniform(0, 1, 300)
        frac = rng.random((257, d))
        p = gpu.CCPotential(d, np.eye(d), modes, V)
        p.set_configuration(frac)
        E, F = p.energy_and_forces()
        k = oracle.lattice_k(np.eye(d), modes)
        Eo, Fo, _, _ = oracle.port_eval(d, np.eye(d), frac, k, V)
        assert abs(E - Eo) <= 1e-12 * V.sum() * 257 ** 2
        assert np.abs(F - Fo).max() <= 1e-12 * 4 * V.sum() * 257 * np.sqrt((np.asarray(k) ** 2).sum(1)).max()


@pytest.mark.parametrize("d,M", [(1, 1), (2, 255), (2, 256), (3, 257), (3, 8193)])
def test_mc_moves_against_whole_energies(gpu, d, M):
    """Trial moves at the edges of the kernel's blocks of 256 modes and beyond 32 blocks: dE is the difference of the whole
    energies (to their rounding, 1e-12 of the energy scale), accepted moves accumulate, and an evaluation in between (which
    writes the same result buffer) changes nothing."""
    rng = np.random.default_rng(M)
    modes = rng.integers(-9, 10, (M, d))
    V = rng.uniform(0, 1, M)
    N = 40
    frac = rng.random((N, d))
    p = gpu.CCPotential(d, np.eye(d), modes, V)
    q = gpu.CCPotential(d, np.eye(d), modes, V)
    p.set_configuration(frac)
    q.set_configuration(frac)
    E = q.energy()
    cur = frac.copy()
    for step in range(6):
        j = int(rng.integers(N))
        new = rng.random(d)
        dE = p.try_move(cur[j], new)
        assert p.try_move(cur[j], new) == dE   # a second trial of the same move repeats bitwise
        trial = cur.copy()
        trial[j] = new
        q.set_configuration(trial)
        assert abs(dE - (q.energy() - E)) <= 1e-12 * V.sum() * N * N
        if step % 2 == 0:
            p.accept_move()
            cur, E = trial, q.energy()
        if step == 3:
            p.energy_and_forces()


@pytest.mark.parametrize("d,N,chi", [(2, 12000, 0.20), (2, 100000, 0.20), (3, 30000, 0.05), (3, 60000, 0.05), (3, 30000, 0.45)])
def test_auto_path(gpu, d, N, chi):
    """AUTO: FP64 takes the NUFFT path only where mixed precision's rule (the segment kernels') does, and not where the
    line kernels are faster; either way its results are those of the path that it names, bit by bit."""
    basis = np.eye(d) * N ** (1 / d)
    modes, V = gpu.stealthy_kset(d, basis, N, chi)
    p = gpu.CCPotential(d, basis, modes, V)
    p.set_configuration(np.random.default_rng(N).random((N, d)))
    fp64, mixed = p.eval_path(N), p.eval_path(N, gpu.PREC_MIXED)
    assert fp64 == mixed or (fp64, mixed) == ("split", "nufft")
    expect = {(2, 12000): "split", (2, 100000): "nufft", (3, 30000): {0.05: "split", 0.45: "nufft"}.get(chi), (3, 60000): "split"}
    assert fp64 == expect[d, N]
    E, F = p.energy_and_forces()
    p.set_path(gpu.PATH_NUFFT if fp64 == "nufft" else gpu.PATH_SPLIT)
    E1, F1 = p.energy_and_forces()
    assert E == E1 and np.array_equal(F, F1)


def test_batch_tiles_teams(gpu):
    """A batch with many force tiles (two teams of warps per tile of 48 particles, several tiles per item, twice the
    particles per rho item): bitwise what each instance gives in a batch of one, and the single evaluation to 1e-12 of
    the scales. Particle counts around the tiles of 24 and 48 and the rho items of 64 and 128; the last set's tables
    are too long for teams."""
    shapes = [(d, N, 0.4) for d in (2, 3) for N in (23, 24, 25, 47, 48, 49, 97, 433, 640, 641, 1279, 1280, 1281)]
    shapes += [(2, 20001, 0.02), (3, 15000, 0.02), (2, 6000, 0.9)]
    assert sum((N + 23) // 24 for _, N, _ in shapes) >= 1.5 * 296
    rng = np.random.default_rng(3)
    pots, fracs = [], []
    for d, N, chi in shapes:
        basis = np.eye(d) * N ** (1 / d)
        modes, V = gpu.stealthy_kset(d, basis, N, chi, 3)
        pots.append(gpu.CCPotential(d, basis, modes, V))
        fracs.append(rng.random((N, d)))
    b = gpu.CCBatch(pots, [N for _, N, _ in shapes])
    b.set_positions(fracs)
    E, F = b.energy_and_forces()
    for k, (d, N, _) in enumerate(shapes):
        one = gpu.CCBatch([pots[k]], [N])
        one.set_positions([fracs[k]])
        e1, f1 = one.energy_and_forces()
        assert e1[0] == E[k] and np.array_equal(f1[0], F[k]), (d, N)
        pots[k].set_path(gpu.PATH_SPLIT)
        pots[k].set_configuration(fracs[k])
        e, f = pots[k].energy_and_forces()
        modes, V = gpu.stealthy_kset(d, np.eye(d) * N ** (1 / d), N, shapes[k][2], 3)
        kmax = 2 * np.pi * np.sqrt((np.asarray(modes, float) ** 2).sum(1)).max() / N ** (1 / d)
        assert abs(E[k] - e) <= 1e-12 * V.sum() * N
        assert np.abs(F[k] - f).max() <= 1e-12 * 4 * V.sum() * kmax
