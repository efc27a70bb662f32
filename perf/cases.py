"""Performance cases of the library: what a path-integral Monte Carlo run has it do.

`listed()` gives the named cases, `draw(rng)` one more case of the same
ranges, `prepare(case, seed)` what a program holds before the call (contexts,
tables, paths, seeded streams), `run(state)` one pass through the public entry
points, `work(case)` the bytes and operations one pass cannot do without, and
`exact(case, seed)` the values of a pass in 64 bits by plain numpy / torch.

Kinds of pass:
  single   one ShortRange SingleAction: the drop-in's smallest call
  stages   one move driven from the host: Kinetic and ShortRange of the NEW and
           the OLD copy at every level, LongRange at the lowest, AcceptCopy
  energy   the energy estimator of the whole path
  gofr     one g(r) sample of the whole path and its read-out
  moves    BisectionBlocks on the device, one ShiftMove, the path read back
  batch    a block of moves on many uneven independent chains

Systems: "lj", Lennard-Jones helium with a 1-D DavidPA table (offdiag > 0: with
off-diagonal u_kj terms; rcut > 0: truncated there, else the table ends at half
the box); "tricubic", the same liquid with a PAtricubicFit; "coulomb", jellium
at r_s = 4 with the optimized Ewald breakup.  Units: Angstrom and Kelvin
(jellium: bohr and Rydberg).
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import pimcplusplus_b200 as P

LAMBDA_HE, RHO_HE = 6.0596, 0.02186
EPS, SIGMA, R_MIN = 10.22, 2.556, 1.5
KCUT, KNOTS, Z1Z2 = 1.2, 49, 2.0


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # The smallest call of a program that keeps its own move loop and replaces one action by the
        # library's: 64 atoms, one moved atom, a window of 8 links.  Latency of a call.
        dict(name="single-lj64", kind="single", system="lj", n=64, m=40, temp=2.0, levels=3, level=0, active=1,
             offdiag=0, rcut=0.0, npts=1000, precision="fp64"),
        # One move of such a program on the benchmark liquid: 16 action calls from 16 links down, and the copy.
        dict(name="stages-tricubic512", kind="stages", system="tricubic", n=512, m=128, temp=1.5, levels=4, active=1,
             nq=200, ny=50, nt=50),
        # The same on jellium, whose lowest stage also updates rho_k and sums over its 510 k-vectors.
        dict(name="stages-jellium128", kind="stages", system="coulomb", n=128, m=64, levels=3, active=1),
        # The energy sample after each block of moves: the whole path, all pairs, of the benchmark liquid, ...
        dict(name="energy-tricubic512", kind="energy", system="tricubic", n=512, m=128, temp=1.5, levels=4, nq=200,
             ny=50, nt=50),
        # ... of jellium (rho_k of every slice recomputed), ...
        dict(name="energy-jellium128", kind="energy", system="coulomb", n=128, m=64, levels=3),
        # ... and of a large chain with a truncated potential: the largest call.
        dict(name="energy-lj4096", kind="energy", system="lj", n=4096, m=256, temp=1.0, levels=5, offdiag=0,
             rcut=2.5 * SIGMA, npts=1000),
        # The pair correlation sample beside it, on the default grid of 100 bins to the box side.
        dict(name="gofr-lj512", kind="gofr", system="lj", n=512, m=128, temp=1.5, levels=4, offdiag=0, rcut=0.0,
             npts=1000, end=0.0, points=101),
        # A small chain as an input file runs it: the reference's sequential schedule, the library's own launch shape.
        dict(name="moves-lj64", kind="moves", system="lj", n=64, m=40, temp=2.0, levels=3, offdiag=0, rcut=0.0,
             npts=1000, schedule="sequential", steps=64, blocks=8, cluster=0, threads=0, precision="fp64", skin=0.0),
        # One chain of the benchmark liquid on all of the GPU: concurrent slice windows, tricubic tables.
        dict(name="moves-tricubic512", kind="moves", system="tricubic", n=512, m=128, temp=1.5, levels=4, nq=200,
             ny=50, nt=50, schedule="windows", steps=128, blocks=2, cluster=16, threads=512, precision="fp64", skin=0.0),
        # Jellium with the long-range action in the lowest stage of every move.
        dict(name="moves-jellium128", kind="moves", system="coulomb", n=128, m=64, levels=3, schedule="windows",
             steps=16, blocks=16, cluster=8, threads=512, precision="fp64", skin=0.0),
        # A large chain with neighbour lists, in mixed precision.
        dict(name="moves-lj4096", kind="moves", system="lj", n=4096, m=256, temp=1.0, levels=5, offdiag=0,
             rcut=2.5 * SIGMA, npts=1000, schedule="windows", steps=16, blocks=4, cluster=16, threads=512,
             precision="mixed", skin=2.5),
        # Many uneven chains at once (clones, or a scan over temperatures and densities): throughput.
        dict(name="batch-512", kind="batch", chains=512, max_n=512, max_m=128, steps=4, blocks=2, precision="mixed"),
    ]


def _log(rng, lo, hi):
    """A whole number of [lo, hi], spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _draw_lj(rng, n_hi, m_lo, m_hi):
    return dict(system="lj", n=_log(rng, 16, n_hi), m=_log(rng, m_lo, m_hi), temp=round(rng.uniform(1.0, 4.0), 3),
                offdiag=rng.choice([0, 0, 1, 2]), rcut=rng.choice([0.0, 2.5 * SIGMA]), npts=_log(rng, 100, 2000))


def _draw_tricubic(rng, n_hi, m_lo, m_hi):
    return dict(system="tricubic", n=_log(rng, 16, n_hi), m=_log(rng, m_lo, m_hi), temp=round(rng.uniform(1.0, 4.0), 3),
                nq=_log(rng, 40, 200), ny=rng.randint(12, 50), nt=rng.randint(12, 50))


def _draw_coulomb(rng, m_lo, m_hi):
    return dict(system="coulomb", n=rng.randint(24, 160), m=_log(rng, m_lo, m_hi))


def draw(rng):
    kind = rng.choice(["single", "stages", "energy", "gofr", "moves", "batch"])
    if kind == "batch":
        return dict(kind=kind, chains=_log(rng, 24, 512), max_n=rng.choice([64, 128, 256, 512]),
                    max_m=rng.choice([32, 64, 128]), steps=rng.randint(1, 4), blocks=rng.randint(1, 2),
                    precision=rng.choice(["fp64", "mixed"]))
    if kind == "gofr":
        c = _draw_lj(rng, 2048, 8, 128)
        c.update(kind=kind, levels=1, offdiag=0, end=rng.choice([0.0, 0.5]), points=_log(rng, 20, 1001))
        return c
    system = rng.choice(["lj", "lj", "tricubic", "coulomb"])
    levels = rng.randint(1, 3 if system == "coulomb" else 5)
    m_lo = (2 << levels) + 1
    c = {"lj": lambda: _draw_lj(rng, 2048 if kind == "energy" else 4096, m_lo, 256),
         "tricubic": lambda: _draw_tricubic(rng, 512, m_lo, 128),
         "coulomb": lambda: _draw_coulomb(rng, m_lo, 128)}[system]()
    c.update(kind=kind, levels=levels)
    if kind == "single":
        c.update(level=rng.randrange(levels), active=rng.choice([1, 1, 2, 5]), precision=rng.choice(["fp64", "mixed"]))
    elif kind == "stages":
        c.update(active=1)
    elif kind == "moves":
        windows = rng.random() < 0.6
        c.update(schedule="windows" if windows else "sequential", steps=rng.randint(4, 32), blocks=rng.randint(1, 6),
                 precision=rng.choice(["fp64", "mixed"]), skin=0.0)
        c["cluster"], c["threads"] = rng.choice([(0, 0), (1, 128), (4, 256), (8, 256), (8, 512), (16, 512)])
        if system == "lj":
            c.update(offdiag=0 if c["precision"] == "mixed" else c["offdiag"])
            if c["rcut"] > 0.0 and c["n"] >= 512:
                c.update(skin=2.5)
                if windows and rng.random() < 0.4:
                    c.update(schedule="proposals", cluster=rng.choice([2, 4, 8]), threads=256)
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _box(case):
    if case["system"] == "coulomb":
        return (4.0 * math.pi / 3.0 * case["n"]) ** (1.0 / 3.0) * 4.0
    return (case["n"] / RHO_HE) ** (1.0 / 3.0)


def _tau(case):
    return 8.0 / case["m"] if case["system"] == "coulomb" else 1.0 / (case["temp"] * case["m"])


def _lambda(case):
    return 1.0 if case["system"] == "coulomb" else LAMBDA_HE


def _bridge(rng, n, m, rms):
    """n closed Brownian paths of m links (row m = row 0), each coordinate of the given rms about row 0's."""
    w = np.zeros((m + 1, n, 3))
    np.cumsum(rng.normal(0.0, rms * math.sqrt(6.0 / m), (m, n, 3)), axis=0, out=w[1:])
    w -= (np.arange(m + 1) / m)[:, None, None] * w[-1]
    return w


def _path(rng, n, m, box, rms):
    """A liquid start: the sites of a cubic lattice, jittered, each with its own closed path."""
    side = int(math.ceil(n ** (1.0 / 3.0) - 1e-9))
    at = (np.arange(n) * side ** 3) // n
    ijk = np.stack([at // (side * side), (at // side) % side, at % side], axis=1)
    a = box / side
    return ((ijk + 0.5 + 0.1 * (rng.random((n, 3)) * 2.0 - 1.0)) * a - 0.5 * box)[None] + _bridge(rng, n, m, rms)


def _case_path(case, rng):
    return _path(rng, case["n"], case["m"], _box(case), 1.5 if case["system"] == "coulomb" else 0.5)


def _lj(r):
    s6 = (SIGMA / r) ** 6
    return 4.0 * EPS * (s6 * s6 - s6)


def _david(case):
    """(grid start, end, ukj, dukj) of a primitive LJ table, [level][point][column], column 0 the potential."""
    tau, nlev, npts, od = _tau(case), case["levels"] + 1, case["npts"], case["offdiag"]
    end = min(case["rcut"], _box(case) / 2) if case["rcut"] > 0.0 else _box(case) / 2
    r = np.linspace(R_MIN, end, npts)
    v = _lj(r) - (_lj(end) if case["rcut"] > 0.0 else 0.0)
    u = np.zeros((nlev, npts, 1 + (od + 1) * (od + 2) // 2))
    du = np.zeros_like(u)
    u[:, :, 0] = du[:, :, 0] = v
    for lev in range(nlev):
        u[lev, :, 1] = tau * 2.0 ** lev * v
        for col in range(2, u.shape[2]):
            f = 1e-3 / col ** 2 * np.exp(-(r / SIGMA) ** 2)
            u[lev, :, col], du[lev, :, col] = tau * 2.0 ** lev * f, f
    u[:, -1] = du[:, -1] = 0.0
    return R_MIN, end, u, du


@functools.lru_cache(maxsize=4)
def _tricubic_nodes(box, tau, nlev, nq, ny, nt):
    q = np.linspace(0.0, box / 2, nq)[:, None, None]
    y, t = np.linspace(0.0, 1.0, ny)[None, :, None], np.linspace(0.0, 1.0, nt)[None, None, :]
    z = y * 2.0 * q
    s = z + t * (2.0 * q - z)
    base = 0.5 * (_lj(np.maximum(q + 0.5 * z, R_MIN)) + _lj(np.maximum(q - 0.5 * z, R_MIN)))
    f = base + s * s * np.exp(-(q / SIGMA) ** 2)
    umat = np.stack([tau * 2.0 ** b * f for b in range(nlev)])
    dumat = np.stack([f] * nlev)
    pot = (R_MIN, box * math.sqrt(3.0) / 2.0 + 1.0, 2000)
    return (0.0, box / 2, nq), (0.0, 1.0, ny), (0.0, 1.0, nt), umat, dumat, pot, _lj(np.linspace(*pot))


def _nodes(case):
    return _tricubic_nodes(_box(case), _tau(case), case["levels"], case["nq"], case["ny"], case["nt"])


def _moved(case, path, rng):
    """Moved atoms, first slice, and the path with their interior slices of one window sampled anew."""
    span = 1 << case["levels"]
    slice1 = int(rng.integers(0, case["m"] - span + 1))
    act = [int(i) for i in rng.choice(case["n"], case["active"], replace=False)]
    new = path.copy()
    new[slice1:slice1 + span + 1, act] += _bridge(rng, len(act), span, 0.2)
    return act, slice1, slice1 + span, new


def _context(case, path):
    box = _box(case)
    d = P.PathData(case["n"], case["m"] + 1, [box] * 3, _tau(case), _lambda(case))
    if case["system"] == "lj":
        start, end, u, du = _david(case)
        d.pa_david(P.GRID_LINEAR, start, end, u, du, 0, case["offdiag"])
    elif case["system"] == "tricubic":
        q, y, t, umat, dumat, pot, v = _nodes(case)
        d.pa_tricubic(q, y, t, _tau(case), umat, dumat, pot, v)
    else:
        d.pa_coulomb(Z1Z2, case["levels"])
        d.setup_kvecs(KCUT)
        d.longrange_coulomb(KNOTS)
    d.set_path(path)
    return d


def _chains(case, rng):
    """Uneven chains: 1/16 .. all of max_n atoms, 1/8 .. all of max_m slices (the set's sizes go with the case), 1-4 K."""
    out, sizes = [], np.random.default_rng(case["chains"])
    for i in range(case["chains"]):
        n = max(16, case["max_n"] >> int(sizes.integers(0, 5)))
        m = max(8, case["max_m"] >> int(sizes.integers(0, 4)))
        levels = min(4, int(math.log2(m)) - 1)
        tau = 1.0 / (rng.uniform(1.0, 4.0) * m)
        box = (n / rng.uniform(0.018, 0.024)) ** (1.0 / 3.0)
        r = np.linspace(R_MIN, box / 2, 1000)
        u00 = (tau * 2.0 ** np.arange(levels + 1))[:, None] * _lj(r)
        u00[:, -1] = 0.0
        out.append(dict(N=n, slices=m + 1, box=[box] * 3, tau=tau, lam=LAMBDA_HE, num_levels=levels,
                        steps_per_block=case["steps"], seed=int(rng.integers(1, 1 << 40)), grid=(R_MIN, box / 2, 1000),
                        u00=u00, path=_path(rng, n, m, box, 0.3)))
    return out


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    st = dict(case=case)
    if case["kind"] == "batch":
        st["batch"] = P.BatchChains(_chains(case, rng), precision=P.MIXED if case["precision"] == "mixed" else P.FP64,
                                    threads_per_cta=512, max_split=2)
        return st
    path = _case_path(case, rng)
    d = st["d"] = _context(case, path)
    if case["kind"] in ("single", "stages"):
        st["act"], st["slice1"], st["slice2"], new = _moved(case, path, rng)
        d.set_path(new, P.NEWMODE)
        precision = P.MIXED if case.get("precision") == "mixed" else P.FP64
        st["short"], st["kin"] = P.ShortRangeClass(d, precision), P.KineticClass(d)
        if case["system"] == "coulomb":
            d.calc_rhok()
            st["long"] = P.LongRangeClass(d)
        d.SetMode(P.NEWMODE)
    elif case["kind"] == "gofr":
        d.gofr_setup(0.0, case["end"] * _box(case), case["points"])
    elif case["kind"] == "moves":
        sched = {"sequential": P.SEQUENTIAL, "windows": P.WINDOWS, "proposals": P.PROPOSALS}[case["schedule"]]
        st["bb"] = P.BisectionBlock(d, case["levels"], case["steps"],
                                    precision=P.MIXED if case["precision"] == "mixed" else P.FP64,
                                    cluster_ctas=case["cluster"], threads_per_cta=case["threads"], schedule=sched,
                                    use_longrange=case["system"] == "coulomb", neighbor_skin=case["skin"])
        st["bb"].seed(seed)
        st["host"] = torch.empty(path.shape, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    return {"single": _run_single, "stages": _run_stages, "energy": _run_energy, "gofr": _run_gofr, "moves": _run_moves,
            "batch": _run_batch}[state["case"]["kind"]](state)


def _run_single(st):
    return np.float64(st["short"].SingleAction(st["slice1"], st["slice2"], st["act"], st["case"]["level"]))


def _run_stages(st):
    d, a, s1, s2 = st["d"], st["act"], st["slice1"], st["slice2"]
    short, kin, lrange = [], [], []
    for level in range(st["case"]["levels"] - 1, -1, -1):
        for mode in (P.NEWMODE, P.OLDMODE):
            d.SetMode(mode)
            kin.append(st["kin"].SingleAction(s1, s2, a, level))
            short.append(st["short"].SingleAction(s1, s2, a, level))
            if level == 0 and "long" in st:
                lrange.append(st["long"].SingleAction(s1, s2, a, level))
    d.AcceptCopy(s1, s2, a)
    return dict(kinetic=np.array(kin), short=np.array(short), long=np.array(lrange))


def _run_energy(st):
    e = st["d"].energy()
    return {k: np.float64(e[k]) for k in ("kinetic", "du_short", "du_long", "v_short", "total")}


def _run_gofr(st):
    st["d"].gofr_accumulate()
    hist, g, samples = st["d"].gofr_get()
    return dict(hist=hist.astype(np.int64), g=g, samples=samples)


def _trace(rec):
    return {k: np.ascontiguousarray(rec[k]) for k in ("slice1", "ptcl", "accepted", "stages_passed")}


def _run_moves(st):
    c = st["case"]
    rec, stats = st["bb"].MakeMoves(c["blocks"])
    shift = st["d"].ShiftMove()
    out = _trace(rec)
    # the mixed path's dS are sums of single-precision terms
    out["dS"] = rec["dS"].astype(np.float32 if c["precision"] == "mixed" else np.float64)
    out["counts"] = np.array([stats[k] for k in ("moves", "accepted", "stages_attempted", "pair_evals")])
    out["shift"] = shift
    out["path"] = st["d"].get_path(out=st["host"])
    return out


def _run_batch(st):
    b = st["batch"]
    rec, stats = b.run(st["case"]["blocks"], trace=True)
    out = _trace(rec)
    out["counts"] = np.array([stats[k] for k in ("moves", "accepted", "stages_attempted", "pair_evals")])
    out["path"] = np.concatenate([b.path(i).reshape(-1) for i in range(0, b.n, max(1, b.n // 8))])
    return out


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
# Operations of one pair-link: the two minimum-image distances (24 each), q, z, s^2 (12), and the table (1-D: two
# cubic splines, 40; tricubic: three Hermite bases and 64 products, 200; Coulomb: two quintics and a division, 40).
_PAIR = {"lj": 100, "tricubic": 260, "coulomb": 100}


def _table_bytes(case, levels, evals):
    """Table bytes a pass reads: at most the whole levels', at most what its evaluations touch."""
    if case["system"] == "lj":
        return min(levels * case["npts"] * 16, evals * 64)
    if case["system"] == "tricubic":
        return min(levels * case["nq"] * case["ny"] * case["nt"] * 64, evals * 512)
    return min(levels * 1000 * 48, evals * 96)


def _num_k(case):
    return int(0.5 * 4.0 / 3.0 * math.pi * (KCUT * _box(case) / (2.0 * math.pi)) ** 3)


def _reach(case):
    """Share of all pairs that a table reaches: a 1-D table is zero from its end on."""
    if case["system"] != "lj":
        return 1.0
    end = min(case["rcut"], _box(case) / 2) if case["rcut"] > 0.0 else _box(case) / 2
    return 4.0 / 3.0 * math.pi * (end / _box(case)) ** 3


def work(case):
    if case["kind"] == "batch":
        # mean chain: N over five halvings of max_n, M over four of max_m; levels of it; about half of the stages
        n, m = case["max_n"] * 31 / 80, case["max_m"] * 15 / 32
        moves = case["chains"] * case["steps"] * case["blocks"]
        return dict(bytes=case["chains"] * (16000 + n * m * 24),
                    flops=moves * n * min(16, m / 2) * _PAIR["lj"])
    n, m, kind = case["n"], case["m"], case["kind"]
    pair, span = _PAIR[case["system"]], 1 << case["levels"]
    rows = n * (span + 1) * 24
    if kind == "single":
        evals = case["active"] * n * _reach(case) * (span >> case["level"])
        return dict(bytes=rows + _table_bytes(case, 1, evals), flops=evals * pair)
    if kind == "stages":
        evals = 2 * n * _reach(case) * (2 * span - 1)
        w = dict(bytes=rows + _table_bytes(case, case["levels"], evals), flops=evals * pair)
        if case["system"] == "coulomb":
            w["bytes"] += (span + 1) * _num_k(case) * 32
            w["flops"] += (span + 1) * _num_k(case) * 30
        return w
    pairs = n * (n - 1) // 2
    if kind == "gofr":
        return dict(bytes=n * m * 24 + 8 * case["points"], flops=pairs * m * 24)
    if kind == "energy":
        evals = pairs * m * _reach(case)
        w = dict(bytes=n * (m + 1) * 24 + _table_bytes(case, 1, evals), flops=evals * (pair + 36) + n * m * 30)
        if case["system"] == "coulomb":
            w["flops"] += n * (m + 1) * _num_k(case) * 14
        return w
    # moves: every move evaluates its top stage, and about half of all lower stages are reached
    per = max(1, m >> case["levels"]) if case["schedule"] != "sequential" else 1
    if case["schedule"] == "proposals":
        per *= case["cluster"]
    moves = case["steps"] * case["blocks"] * per
    evals = moves * 2 * n * _reach(case) * span
    w = dict(bytes=2 * n * (m + 1) * 24 + moves * 208 + _table_bytes(case, case["levels"], evals), flops=evals * pair)
    if case["system"] == "coulomb":
        w["flops"] += moves * span * _num_k(case) * 15
    return w


# ---------------------------------------------------------------------------
# the same in 64 bits, by plain numpy and torch
# ---------------------------------------------------------------------------
def exact(case, seed):
    """None for the chains of moves and batch: a Markov chain has to be replayed move by move, which takes minutes
    in Python.  None in the place of what depends on the optimized breakup's own fit (jellium, but kinetic)."""
    if case["kind"] in ("moves", "batch"):
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    rng = np.random.default_rng(seed)
    path = _case_path(case, rng)
    x = torch.from_numpy(path).to(dev)
    if case["kind"] == "gofr":
        return _exact_gofr(case, x)
    pa = None if case["system"] == "coulomb" else (_ExactDavid if case["system"] == "lj" else _ExactTricubic)(case, dev)
    if case["kind"] == "energy":
        return _exact_energy(case, x, pa)
    act, s1, s2, new = _moved(case, path, rng)
    y = torch.from_numpy(new).to(dev)
    if case["kind"] == "single":
        return None if pa is None else np.float64(_exact_short(case, y, pa, act, s1, s2, case["level"]))
    kin, short = [], []
    for level in range(case["levels"] - 1, -1, -1):
        for z in (y, x):
            kin.append(_exact_kinetic(case, z, act, s1, s2, level))
            if pa is not None:
                short.append(_exact_short(case, z, pa, act, s1, s2, level))
    return dict(kinetic=np.array(kin), short=np.array(short) if pa is not None else None,
                long=None if pa is None else np.zeros(0))


def _exact_link(box, a, b):
    """(q, z, s^2, r, r') of pair displacements a, b at a link's two slices, b in the image that follows a."""
    n = -torch.round(a / box)
    a = a + n * box
    b = b + torch.round((a - b) / box) * box
    r, rp = a.square().sum(-1).sqrt(), b.square().sum(-1).sqrt()
    return 0.5 * (r + rp), r - rp, (a - b).square().sum(-1)


def _exact_short(case, x, pa, act, s1, s2, level):
    box, skip, total, seen = _box(case), 1 << level, 0.0, []
    for p in act:
        seen.append(p)
        rest = [j for j in range(case["n"]) if j not in seen]
        for s in range(s1, s2, skip):
            a, b = x[s, rest] - x[s, p], x[s + skip, rest] - x[s + skip, p]
            total += float(pa.value(*_exact_link(box, a, b), level, False).sum())
    return total


def _exact_kinetic(case, x, act, s1, s2, level):
    box, skip = _box(case), 1 << level
    v = x[s1 + skip:s2 + 1:skip, act] - x[s1:s2:skip, act]
    v = v - torch.floor(v / box + 0.5) * box
    return float(v.square().sum()) / (4.0 * _lambda(case) * _tau(case) * skip)


def _exact_energy(case, x, pa):
    n, m, box, tau = case["n"], case["m"], _box(case), _tau(case)
    v = x[1:] - x[:-1]
    v = v - torch.floor(v / box + 0.5) * box
    kinetic = n * m * 1.5 / tau - float(v.square().sum()) / (4.0 * _lambda(case) * tau * tau)
    out = dict(kinetic=np.float64(kinetic), du_short=None, du_long=None, v_short=None, total=None)
    if pa is None:
        return out
    i, j = torch.tril_indices(n, n, -1, device=x.device)
    du = vs = 0.0
    step = max(1, (1 << 24) // i.numel())  # links at a time
    for s in range(0, m + 1, step):
        e = min(m + 1, s + step)
        a = x[s:e, j] - x[s:e, i]
        if s < m:
            b = x[s + 1:e + 1, j] - x[s + 1:e + 1, i]
            du += float(pa.value(*_exact_link(box, a[:b.shape[0]], b), 0, True).sum())
        a = a - torch.round(a / box) * box
        f = torch.ones(e - s, dtype=x.dtype, device=x.device)
        f[torch.arange(s, e, device=x.device) % m == 0] = 0.5
        vs += float((f[:, None] * pa.potential(a.square().sum(-1).sqrt())).sum())
    out.update(du_short=du, du_long=0.0, v_short=vs, total=(out["kinetic"] + du) / m)
    return {k: np.float64(v) for k, v in out.items()}


def _exact_gofr(case, x):
    n, m, box = case["n"], case["m"], _box(case)
    end, bins = (case["end"] or 1.0) * box, case["points"] - 1
    i, j = torch.tril_indices(n, n, -1, device=x.device)
    hist = torch.zeros(bins, dtype=torch.int64, device=x.device)
    delta = end / bins
    step = max(1, (1 << 24) // i.numel())
    for s in range(0, m, step):
        a = x[s:min(m, s + step), j] - x[s:min(m, s + step), i]
        a = a - torch.round(a / box) * box
        r = a.square().sum(-1).sqrt().reshape(-1)
        r = r[r < end]
        at = torch.round(r * (1.0 / delta) - 0.5).to(torch.int64)
        hist += torch.bincount(at[(at >= 0) & (at < bins)], minlength=bins)
    edge = delta * np.arange(bins + 1)
    vol = 4.0 * math.pi / 3.0 * (edge[1:] ** 3 - edge[:-1] ** 3)
    return dict(hist=None, g=hist.cpu().numpy() / (vol * (0.5 * m * n * (n - 1.0) / box ** 3)), samples=None)


def _second_derivatives(x, y, natural_end):
    """Cubic-spline second derivatives along axis 0: natural start; natural or zero-slope end."""
    n, h = len(x), x[1] - x[0]
    c, u = np.zeros(n), np.zeros_like(y)
    for k in range(1, n - 1):
        p = 0.5 * c[k - 1] + 2.0
        c[k] = -0.5 / p
        u[k] = (3.0 * (y[k + 1] - 2.0 * y[k] + y[k - 1]) / h ** 2 - 0.5 * u[k - 1]) / p
    d = np.zeros_like(y)
    if not natural_end:
        d[-1] = (-3.0 / h * (y[-1] - y[-2]) / h - 0.5 * u[-2]) / (0.5 * c[-2] + 1.0)
    for k in range(n - 2, -1, -1):
        d[k] = c[k] * d[k + 1] + u[k]
    return d


class _Cubic:
    """A cubic spline of many columns on a uniform grid."""

    def __init__(self, start, end, y, natural_end, dev):
        x = np.linspace(start, end, len(y))
        self.start, self.h, self.n = start, (end - start) / (len(y) - 1), len(y)
        self.y = torch.from_numpy(np.ascontiguousarray(y)).to(dev)
        self.d = torch.from_numpy(_second_derivatives(x, y, natural_end)).to(dev)

    def __call__(self, r, col):
        i = torch.clamp(torch.round((r - self.start) / self.h - 0.5), 0, self.n - 2).to(torch.int64)
        b = (r - (self.start + i.to(r.dtype) * self.h)) / self.h
        a = 1.0 - b
        y, d = self.y[:, col], self.d[:, col]
        return a * y[i] + b * y[i + 1] + ((a ** 3 - a) * d[i] + (b ** 3 - b) * d[i + 1]) * self.h ** 2 / 6.0


class _ExactDavid:
    def __init__(self, case, dev):
        self.start, self.end, u, du = _david(case)
        self.u = [_Cubic(self.start, self.end, t, False, dev) for t in u]
        self.du = [_Cubic(self.start, self.end, t, False, dev) for t in du]
        self.terms = case["offdiag"]

    def value(self, q, z, s2, level, deriv):
        r, rp = (q + 0.5 * z).clamp(max=self.end), (q - 0.5 * z).clamp(max=self.end)
        t = (self.du if deriv else self.u)[level]
        low = (r < self.start) | (rp < self.start)
        r, rp = r.clamp(min=self.start), rp.clamp(min=self.start)
        v = 0.5 * (t(r, 1) + t(rp, 1))
        if deriv:
            v = v + 0.5 * (self.u[level](r, 0) + self.u[level](rp, 0))
        if self.terms:
            off = torch.zeros_like(v)
            for k in range(1, self.terms + 1):
                for j in range(k + 1):
                    off = off + t(q, k * (k + 1) // 2 + j + 1) * (z * z) ** j * s2 ** (k - j)
            v = torch.where((s2 > 0) & (q < self.end), v + off, v)
        # U (not dU) of a pair below the grid's start is the diagonal there
        return v if deriv else torch.where(low, t(torch.full_like(q, self.start), 1), v)

    def potential(self, r):
        return self.u[0](r.clamp(self.start, self.end), 0)


def _slopes(f, axis, h):
    """First derivatives along `axis`: a tridiagonal solve of the spline's continuity, end slopes from 3/2 of the
    first and the last difference (the last one through the same elimination)."""
    f = np.moveaxis(f, axis, 0)
    n, g, mu = len(f), np.zeros_like(f), np.zeros(len(f))
    g[0] = 1.5 * (f[1] - f[0]) / h
    mu[0] = 0.5
    for k in range(1, n):
        last = k == n - 1
        lam = 0.5 if last else 0.25
        g[k] = 3.0 * lam * (f[k] - f[k - 1]) / h + (0.0 if last else 3.0 * 0.25 * (f[k + 1] - f[k]) / h)
        c = 1.0 - lam * mu[k - 1]
        g[k] = (g[k] - lam * g[k - 1]) / c
        mu[k] = (0.5 - lam) / c
    for k in range(n - 2, -1, -1):
        g[k] -= mu[k] * g[k + 1]
    return np.moveaxis(g, 0, axis)


class _ExactTricubic:
    def __init__(self, case, dev):
        q, y, t, umat, dumat, pot, v = _nodes(case)
        self.tau, self.end, self.pot_end = _tau(case), q[1], pot[1]
        self.h = [g[1] / (g[2] - 1) for g in (q, y, t)]
        self.shape = (q[2], y[2], t[2])
        need = range(case["levels"]) if case["kind"] != "energy" else [0]
        if case["kind"] == "single":
            need = [case["level"]]
        self.nodes = {lev: self._fill((dumat if case["kind"] == "energy" else umat)[lev], dev) for lev in need}
        self.pot = _Cubic(pot[0], pot[1], v[:, None], True, dev)

    def _fill(self, f, dev):
        fx, fy, fz = (_slopes(f, a, self.h[a]) for a in range(3))
        fxy, fxz, fyz = _slopes(fx, 1, self.h[1]), _slopes(fx, 2, self.h[2]), _slopes(fy, 2, self.h[2])
        parts = [f, fz, fy, fyz, fx, fxz, fxy, _slopes(fxy, 2, self.h[2])]  # index 4 [d/dx] + 2 [d/dy] + [d/dz]
        return torch.from_numpy(np.stack([p.reshape(-1) for p in parts], axis=1)).to(dev)

    def value(self, q, z, s2, level, deriv):
        z, s, top = z.abs(), s2.sqrt(), 2.0 * q
        inside = (q <= self.end) & (z < top) & (s < top)
        ok = inside & (q != 0)
        one = torch.ones_like(q)
        c = [torch.where(ok, q, 0 * q), torch.where(ok, z / torch.where(ok, top, one), 0 * q),
             torch.where(ok, (s - z) / torch.where(ok, top - z, one), 0 * q)]
        idx, basis = [], []
        for x, h, n in zip(c, self.h, self.shape):
            i = torch.clamp(torch.round(x / h - 0.5), 0, n - 2).to(torch.int64)
            u = (x - i.to(x.dtype) * h) / h
            idx.append(i)
            basis.append([[(u - 1) ** 2 * (1 + 2 * u), h * u * (u - 1) ** 2], [u * u * (3 - 2 * u), h * u * u * (u - 1)]])
        tri = torch.zeros_like(q)
        nodes = self.nodes[level]
        for k in range(8):
            dx, dy, dz = k >> 2, (k >> 1) & 1, k & 1
            f = nodes[((idx[0] + dx) * self.shape[1] + idx[1] + dy) * self.shape[2] + idx[2] + dz]
            for e in range(8):
                tri = tri + f[..., e] * (basis[0][dx][e >> 2] * basis[1][dy][(e >> 1) & 1] * basis[2][dz][e & 1])
        prim = 0.5 * (self.potential(q + 0.5 * z) + self.potential(q - 0.5 * z))
        return torch.where(inside, tri, prim if deriv else prim * self.tau * 2.0 ** level)

    def potential(self, r):
        return torch.where(r <= self.pot_end, self.pot(r.clamp(max=self.pot_end), 0), torch.zeros_like(r))
