"""The work that users of this framework have it do, case by case, through its public entry points.

Every configuration is N uniform random points in a periodic cube of unit density (side N^(1/d)) with a stealthy
constraint set (the command-line program's Types 0 and 3), at the sizes of the benchmark, the tests and the served
stream: N = 100 to 100000, d = 2 and 3, chi = 0.05 to 0.49. The kinds:

  host    one configuration bound from host memory, its energy and forces read back (an optimiser's objective)
  device  one evaluation of resident positions, results left on the device (a driver with its own GPU state)
  pool    resident configurations evaluated one after another in one replayed CUDA graph (the benchmark's headline)
  many    configurations from pinned host memory in one call (an ensemble on the host)
  batch   uneven independent configurations in one batch, positions in, energies and forces out
  relax   the first steps of a batched minimisation, from random starts to an evaluation limit
  sk      S(k) of a configuration on every wavevector of a circle (the structure factor)
  s2      the S2 form (targets for S(k)), always by direct sums
  mc      a Monte Carlo sweep: bind, then trial moves of which every second one is accepted
"""
import math

import numpy as np
import torch

import modules_b200 as cc


def listed():
    return [
        # the smallest job: a 2D ground-state search of 100 points asks for one objective at a time
        dict(name="host 2d n100", kind="host", d=2, N=100, chi=0.30, v=0),
        # the headline configuration, evaluated alone
        dict(name="device 3d n2000", kind="device", d=3, N=2000, chi=0.45, v=0, prec="fp64"),
        # the headline measurement: resident configurations one after another
        dict(name="pool 3d n2000", kind="pool", d=3, N=2000, chi=0.45, v=0, count=32),
        # an ensemble in pinned host memory
        dict(name="many 3d n2000", kind="many", d=3, N=2000, chi=0.45, v=0, count=128),
        # an ordinary 2D evaluation by direct sums, at a size nobody tuned for
        dict(name="device 2d n7001", kind="device", d=2, N=7001, chi=0.37, v=3, prec="fp64"),
        # the same size range in mixed precision (the first stage of a precision schedule)
        dict(name="device 3d n3001 mixed", kind="device", d=3, N=3001, chi=0.25, v=0, prec="mixed"),
        # the large 2D workload, M = 40002 wavevectors
        dict(name="device 2d n100000", kind="device", d=2, N=100000, chi=0.20, v=0, prec="fp64"),
        # uneven independent configurations
        dict(name="batch 60", kind="batch", count=60, nmin=200, nmax=5000),
        # the first steps of a batch of ground-state searches
        dict(name="relax 48", kind="relax", count=48, nmin=200, nmax=5000, evals=16),
        # the structure factor of the large 2D configuration
        dict(name="sk 2d n100000", kind="sk", d=2, N=100000, chi=0.20),
        # targets for S(k) in 3D
        dict(name="s2 3d n20000", kind="s2", d=3, N=20000, chi=0.20),
        # one Monte Carlo sweep
        dict(name="mc 3d n2000", kind="mc", d=3, N=2000, chi=0.45, v=0, moves=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "device", "device", "pool", "many", "batch", "relax", "sk", "s2", "mc"])
    d = rng.choice([2, 3])
    chi = round(rng.uniform(0.05, 0.49), 3)
    v = rng.choice([0, 3])
    if kind == "host":
        return dict(kind=kind, d=d, N=_log(rng, 100, 20000), chi=chi, v=v)
    if kind == "device":
        prec = rng.choice(["fp64", "fp64", "fp64", "mixed"])
        return dict(kind=kind, d=d, N=_log(rng, 100, 5000 if prec == "mixed" else 100000 if d == 2 else 30000), chi=chi,
                    v=v, prec=prec)
    if kind == "pool":
        return dict(kind=kind, d=d, N=_log(rng, 200, 5000), chi=chi, v=v, count=rng.randint(8, 40))
    if kind == "many":
        return dict(kind=kind, d=d, N=_log(rng, 200, 5000), chi=chi, v=v, count=rng.randint(16, 128))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(6, 60), nmin=200, nmax=_log(rng, 800, 5000))
    if kind == "relax":
        return dict(kind=kind, count=rng.randint(6, 48), nmin=200, nmax=_log(rng, 800, 5000), evals=rng.randint(4, 16))
    if kind == "sk":
        return dict(kind=kind, d=d, N=_log(rng, 200, 100000 if d == 2 else 50000), chi=round(rng.uniform(0.05, 0.20), 3))
    if kind == "s2":
        return dict(kind=kind, d=d, N=_log(rng, 200, 20000), chi=round(rng.uniform(0.05, 0.40), 3))
    return dict(kind=kind, d=d, N=_log(rng, 200, 5000), chi=chi, v=v, moves=rng.randint(16, 64))


# ---- inputs ------------------------------------------------------------------------------------------------------
def _half_space(d, want):
    """Half-space integer vectors by (|n|^2, index): the first `want` and the rest of the last shell, |n|^2 of each,
    and |n|^2 of the first shell left out."""
    r = int(math.ceil({2: math.sqrt(2 * want / math.pi), 3: (1.5 * want / math.pi) ** (1 / 3)}[d])) + 3
    ax = np.arange(-r, r + 1, dtype=np.int32)
    n = np.stack(np.meshgrid(*[ax[r:]] + [ax] * (d - 1), indexing="ij"), -1).reshape(-1, d)
    first = np.where(n[:, 0] != 0, n[:, 0], n[:, 1] if d == 2 else np.where(n[:, 1] != 0, n[:, 1], n[:, 2]))
    n = n[first > 0]
    n2 = (n.astype(np.int64) ** 2).sum(1)
    o = np.lexsort(tuple(n[:, e] for e in range(d - 1, -1, -1)) + (n2,))
    n, n2 = n[o], n2[o]
    M = int(np.searchsorted(n2, n2[want - 1], side="right"))
    return np.ascontiguousarray(n[:M]), n2[:M], int(n2[M])


def _constraints(d, N, chi, v):
    """(modes, V) of a stealthy set by the command-line program's rule, without its code (for exact())."""
    n, n2, nx = _half_space(d, int(math.ceil(chi * N * d)))
    return n, (np.ones(len(n)) if v == 0 else (1.0 - np.sqrt(n2 / nx)) ** 2)


def _frac(N, d, seed):
    return np.random.default_rng(seed).random((N, d))


def _pool(case, seed):
    return np.random.default_rng(seed).random((case["count"], case["N"], case["d"]))


def _instances(case, seed):
    """The uneven instances of a batch: shapes by the case alone, positions by the seed. v = (1 - |k|/K)^2."""
    rng = np.random.default_rng(case["count"] * 7919 + case["nmax"])
    pos = np.random.default_rng(seed)
    out = []
    for _ in range(case["count"]):
        d = int(rng.choice([2, 3]))
        n = int(round(math.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"])))))
        out.append((d, n, float(rng.uniform(0.10, 0.49)), pos.random((n, d))))
    return out


def _s2_targets(modes):
    """Targets of a hyperuniform S(k) ~ k^2 and equal weights."""
    n2 = (modes.astype(np.float64) ** 2).sum(1)
    return np.ones(len(modes)), 0.8 * n2 / n2.max()


def _moves(case, seed):
    rng = np.random.default_rng(seed + 1)
    who = rng.integers(0, case["N"], case["moves"])
    return who, rng.normal(0.0, 0.1 / case["N"] ** (1 / case["d"]), (case["moves"], case["d"]))


def _potential(case):
    d, N = case["d"], case["N"]
    basis = np.eye(d) * N ** (1.0 / d)
    modes, V = cc.stealthy_kset(d, basis, N, case["chi"], case["v"])
    return cc.CCPotential(d, basis, modes, V)


def _resident(case, seed):
    return torch.from_numpy(_frac(case["N"], case["d"], seed)).cuda()


# ---- what a user's program has in hand, and one pass ----------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind in ("batch", "relax"):
        s["pots"], Ns = [], []
        s["fracs"] = []
        for d, n, chi, frac in _instances(case, seed):
            s["pots"].append(_potential(dict(d=d, N=n, chi=chi, v=3)))
            Ns.append(n)
            s["fracs"].append(frac)
        s["batch"] = cc.CCBatch(s["pots"], Ns)
        return s
    d, N = case["d"], case["N"]
    if kind == "s2":
        modes, _ = _constraints(d, N, case["chi"], 0)
        V, S0 = _s2_targets(modes)
        s["pot"] = cc.CCPotential(d, np.eye(d) * N ** (1.0 / d), modes, V, S0=S0)
    elif kind == "sk":
        modes, _ = _constraints(d, N, case["chi"], 0)
        s["modes"] = modes
        s["pot"] = cc.CCPotential(d, np.eye(d) * N ** (1.0 / d), modes[:1], np.ones(1))
    else:
        s["pot"] = _potential(case)
    pot = s["pot"]
    if kind in ("device", "s2"):
        s["prec"] = cc.PREC_MIXED if case.get("prec") == "mixed" else cc.PREC_FP64
        s["frac"] = _resident(case, seed)
        s["E"] = torch.zeros(1, dtype=torch.float64, device="cuda")
        s["F"] = torch.zeros(N, d, dtype=torch.float64, device="cuda")
    elif kind == "pool":
        s["frac"] = torch.from_numpy(_pool(case, seed)).cuda()
        s["E"] = torch.zeros(case["count"], dtype=torch.float64, device="cuda")
        s["F"] = torch.zeros(case["count"], N, d, dtype=torch.float64, device="cuda")
        pot.set_independent_positions(True)
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()

        def sweep(n):
            for i in range(n):
                pot.energy_grad_device(N, s["frac"][i].data_ptr(), s["E"][i:i + 1].data_ptr(), s["F"][i].data_ptr(),
                                       stream=stream.cuda_stream)
        sweep(1)
        stream.synchronize()
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["graph"], stream=stream):
            sweep(case["count"])
    elif kind == "many":
        def pinned(*shape):
            return torch.zeros(*shape, dtype=torch.float64, pin_memory=True).numpy()
        s["frac"] = pinned(case["count"], N, d)
        s["frac"][:] = _pool(case, seed)
        s["E"], s["F"] = pinned(case["count"]), pinned(case["count"], N, d)
    else:
        s["frac"] = _frac(N, d, seed)
        if kind == "mc":
            who, step = _moves(case, seed)
            s["moves"] = []
            at = {}
            for k in range(case["moves"]):   # every second move is accepted
                j = int(who[k])
                old = at.get(j, s["frac"][j])
                new = (old + step[k]) % 1.0
                if k % 2 == 0:
                    at[j] = new
                s["moves"].append((old, new))
    return s


def run(s):
    kind, pot = s["case"]["kind"], s.get("pot")
    if kind == "host":
        pot.set_configuration(s["frac"])
        return pot.energy_and_forces()
    if kind in ("device", "s2"):
        pot.energy_grad_device(s["case"]["N"], s["frac"].data_ptr(), s["E"].data_ptr(), s["F"].data_ptr(),
                               precision=s["prec"])
        return s["E"], s["F"]
    if kind == "pool":
        s["graph"].replay()
        return s["E"], s["F"]
    if kind == "many":
        return pot.energy_grad_many(s["frac"], E=s["E"], F=s["F"])
    if kind == "batch":
        s["batch"].set_positions(s["fracs"])
        return s["batch"].energy_and_forces()
    if kind == "relax":
        x, E, evals, iters, status = s["batch"].minimize(s["fracs"], max_evals=s["case"]["evals"])
        return x, E, evals, iters, status
    if kind == "sk":
        pot.set_configuration(s["frac"])
        return pot.structure_factor(s["modes"])
    pot.set_configuration(s["frac"])
    dE = np.empty(len(s["moves"]))
    for k, (old, new) in enumerate(s["moves"]):
        dE[k] = pot.try_move(old, new)
        if k % 2 == 0:
            pot.accept_move()
    return dE


# ---- what a pass cannot do without --------------------------------------------------------------------------------
def _eval_work(d, N, chi, copies=1, rho_only=False):
    """Positions in, forces out, the constraint set (16 bytes a vector) read once. Arithmetic: per particle and vector
    one real multiply-add per component of rho and two per component pair of the forces when the vectors +m and -m of a
    lattice line share the cosine and sine (4 + 8 flops); or, where that is less, fast transforms of the particles
    spread onto a grid of twice the range (14 points an axis)."""
    M = math.ceil(chi * N * d)
    direct = (4.0 if rho_only else 12.0) * N * M
    K = math.sqrt(2 * M / math.pi) if d == 2 else (1.5 * M / math.pi) ** (1 / 3)
    grid = (4 * K + 2) ** d
    fast = N * 14.0 ** d * (2 if rho_only else 2 + 2 * d) + 2.5 * grid * math.log2(grid) * (1 if rho_only else 1 + d)
    return dict(bytes=float(copies) * N * d * 8 * (1 if rho_only else 2) + M * 16, flops=copies * min(direct, fast))


def work(case):
    kind = case["kind"]
    if kind in ("batch", "relax"):
        w = [_eval_work(d, n, chi) for d, n, chi, _ in _instances(case, 0)]
        k = case.get("evals", 1)
        return dict(bytes=sum(x["bytes"] for x in w), flops=k * sum(x["flops"] for x in w))
    d, N, chi = case["d"], case["N"], case["chi"]
    if kind == "mc":
        w = _eval_work(d, N, chi, rho_only=True)
        M = math.ceil(chi * N * d)
        return dict(bytes=w["bytes"] + 40.0 * M * case["moves"], flops=w["flops"] + 30.0 * M * case["moves"])
    return _eval_work(d, N, chi, case.get("count", 1), rho_only=kind == "sk")


# ---- the same in 64 bits, by plain direct sums --------------------------------------------------------------------
def _phases(frac, modes):
    """cos and sin of 2 pi n.s, particles x modes."""
    t = torch.zeros(len(frac), len(modes), dtype=torch.float64, device=frac.device)
    for e in range(frac.shape[1]):
        p = frac[:, e:e + 1] * modes[None, :, e]
        t += p - torch.round(p)
    t *= 2 * math.pi
    return torch.cos(t), torch.sin(t)


def _rho(frac, modes):
    re = torch.zeros(len(modes), dtype=torch.float64, device=frac.device)
    im = torch.zeros_like(re)
    step = max(1, (1 << 26) // max(1, len(modes)))
    for j in range(0, len(frac), step):
        c, s = _phases(frac[j:j + step], modes)
        re += c.sum(0)
        im += s.sum(0)
    return re, im


def _forces(frac, modes, wr, wi, scale):
    """scale * sum_k Im((wr - i wi) exp(i k.r)) n_k"""
    F = torch.empty_like(frac)
    step = max(1, (1 << 26) // max(1, len(modes)))
    for j in range(0, len(frac), step):
        c, s = _phases(frac[j:j + step], modes)
        F[j:j + step] = scale * ((s * wr - c * wi) @ modes)
    return F


def _gpu(x):
    return torch.from_numpy(np.ascontiguousarray(x, dtype=np.float64)).to("cuda" if torch.cuda.is_available() else "cpu")


def _exact_eval(frac, modes, V):
    """(E, F) of ShiftedCCPotential in a cube of unit density."""
    N, d = frac.shape
    f, n, w = _gpu(frac), _gpu(modes), _gpu(V)
    re, im = _rho(f, n)
    E = float((w * (re * re + im * im)).sum()) / N
    F = _forces(f, n, w * re, w * im, 2.0 / N * 2 * math.pi / N ** (1.0 / d))
    return E, F.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "relax":
        return None
    if kind == "batch":
        E, F = [], []
        for d, n, chi, frac in _instances(case, seed):
            e, f = _exact_eval(frac, *_constraints(d, n, chi, 3))
            E.append(e)
            F.append(f)
        return np.array(E), F
    d, N = case["d"], case["N"]
    modes, V = _constraints(d, N, case["chi"], case.get("v", 0))
    if kind in ("pool", "many"):
        r = [_exact_eval(f, modes, V) for f in _pool(case, seed)]
        return np.array([e for e, _ in r]), np.stack([f for _, f in r])
    frac = _frac(N, d, seed)
    if kind == "host":
        return _exact_eval(frac, modes, V)
    if kind == "device":
        E, F = _exact_eval(frac, modes, V)
        return np.array([E]), F
    f, n = _gpu(frac), _gpu(modes)
    re, im = _rho(f, n)
    if kind == "sk":
        return ((re * re + im * im) / N).cpu().numpy()
    if kind == "s2":
        V, S0 = (_gpu(x) for x in _s2_targets(modes))
        ds = (re * re + im * im) / N - S0
        F = _forces(f, n, V * ds * re, V * ds * im, 4.0 / N * 2 * math.pi / N ** (1.0 / d))
        return np.array([float((V * ds * ds).sum())]), F.cpu().numpy()
    who, step = _moves(case, seed)
    w, at, dE = _gpu(V), {}, np.empty(case["moves"])
    for k in range(case["moves"]):
        j = int(who[k])
        old = at.get(j, frac[j])
        new = (old + step[k]) % 1.0
        c, s = _phases(_gpu(np.stack([old, new])), n)
        dr, di = c[1] - c[0], s[1] - s[0]
        dE[k] = float((w * (2 * (re * dr + im * di) + dr * dr + di * di)).sum()) / N
        if k % 2 == 0:
            at[j] = new
            re, im = re + dr, im + di
    return dE
