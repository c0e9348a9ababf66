"""The work a user of this engine has it do, as cases that can be timed.

Every case is one call of a public entry point of `chaoslibrary_gb300`, with
results in device arrays the caller keeps (`out=`), on the systems, ranges and
horizons of the repository's own workloads (`bench.py`). The inputs -- initial
conditions and the ends of the swept ranges, or the points to cluster -- are
made from a seed.

A case is a dict: `kind` (the entry point), `system`, `precision` ("fp32",
"ff32", "fp64"), `nPts` (points per axis; points of a 1-D sweep; points to
cluster), `tMax` and `transient` (time units, h = 0.01 unless stated).
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import chaoslibrary_gb300 as C

H = 0.01
# flops of one step of the map (FMA = 2); Chameleon's cosine counted as one
STEP_FLOPS = {"lorenz": 71, "rossler": 63, "chen": 79, "chameleon": 42}
VALUES = {"lorenz": [10.0, 28.0, 8.0 / 3.0], "rossler": [0.2, 0.2, 5.7], "chen": [35.0, 3.0, 28.0],
          "chameleon": [0.5, 3.0, 0.0, 2.0, 1.0, 18.0, 1.0]}
START = {"lorenz": [0.1, 0.1, 0.1], "rossler": [1.0, 1.0, 1.0], "chen": [-10.0, 0.0, 37.0],
         "chameleon": [3.0, 3.0, 0.0]}
# swept parameters: 1-D sweeps and 2-D maps
SWEEP1 = {"lorenz": ([1], [20.0, 200.0]), "rossler": ([2], [2.0, 10.0]), "chen": ([2], [20.0, 30.0])}
SWEEP2 = {"lorenz": ([1, 0], [20.0, 200.0, 5.0, 15.0]), "rossler": ([0, 2], [0.1, 0.4, 2.0, 10.0]),
          "chen": ([2, 0], [20.0, 30.0, 30.0, 40.0]), "chameleon": ([3, 5], [0.0, 5.0, 0.0, 20.0])}
BASIN_VALUES = {"lorenz": [10.0, 24.0, 8.0 / 3.0], "rossler": [0.2, 0.2, 5.7], "chen": [35.0, 3.0, 28.0]}
BASIN_START = {"lorenz": [0.0, 0.0, 27.0], "rossler": [0.0, 0.0, 0.5], "chen": [0.0, 0.0, 20.0]}
RK4 = ("lorenz", "rossler", "chen")
NT, EPS = 0.1, 1e-8  # Benettin block and twin distance of the LLE and spectrum workloads


def listed():
    return [
        # The first look at a system: a 1-D bifurcation diagram one screen wide, waited for at the prompt.
        # 1,000 points leave most of the GPU idle; the length of one trajectory's chain decides.
        dict(name="bif1d_screen", kind="bif1d", system="lorenz", precision="fp32", nPts=1000, tMax=100.0,
             transient=100.0),
        # The same diagram in the library's default precision, which reproduces the original library's numbers.
        dict(name="bif1d_fp64", kind="bif1d", system="lorenz", precision="fp64", nPts=999, tMax=100.0,
             transient=100.0),
        # A diagram fine enough to zoom into: hundreds of thousands of points, the throughput of the 1-D sweep.
        dict(name="bif1d_fine", kind="bif1d", system="rossler", precision="fp32", nPts=700001, tMax=100.0,
             transient=100.0),
        # The original library's own 2-D timing sweep (its default system, long transient, per-point clustering
        # of the intervals between peaks).
        dict(name="bif2d_chameleon", kind="bif2d", system="chameleon", precision="fp32", nPts=300, tMax=400.0,
             transient=2000.0),
        # The Lyapunov map that is published: the precision-matched arithmetic at a full horizon.
        dict(name="lle_ff32", kind="lle", system="rossler", precision="ff32", nPts=512, tMax=500.0, transient=50.0),
        # A quick look at such a map in plain FP32: a coarse, odd-sized grid.
        dict(name="lle_quick", kind="lle", system="lorenz", precision="fp32", nPts=257, tMax=500.0, transient=50.0),
        # A small map in the default precision, as a check of the others.
        dict(name="lle_fp64", kind="lle", system="rossler", precision="fp64", nPts=100, tMax=250.0, transient=50.0),
        # Basins of attraction of a two-attractor flow, a megapixel, clustered into labels.
        dict(name="basins_map", kind="basins_dbscan", system="lorenz", precision="fp32", nPts=1024, tMax=50.0,
             transient=200.0),
        # The original library's basins call (its features and its clustering) in the default precision.
        dict(name="basins_fp64", kind="basins", system="lorenz", precision="fp64", nPts=150, tMax=50.0,
             transient=200.0),
        # All Lyapunov exponents over a parameter plane.
        dict(name="spectrum_map", kind="spectrum", system="lorenz", precision="fp32", nPts=384, tMax=100.0,
             transient=20.0),
        # Clustering of features that are already on the device (a map's, or those of several maps).
        dict(name="cluster", kind="dbscan", system="", precision="fp64", nPts=1000000, dims=3),
        # An uneven mix of jobs prepared once and replayed: the parameter study that is run again and again.
        dict(name="batch_mixed", kind="batch", system="", precision="fp32", nPts=100000, jobs=15),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng: random.Random):
    kind = rng.choice(["bif1d", "bif1d", "bif2d", "lle", "lle", "basins_dbscan", "basins", "spectrum", "dbscan",
                       "batch"])
    tMax = round(rng.uniform(30.0, 100.0), 1)
    transient = round(rng.uniform(20.0, 100.0), 1)
    system = rng.choice(RK4)
    if kind == "bif1d":
        precision = rng.choice(["fp32", "fp32", "fp64"])
        n = _log(rng, 300, 20000 if precision == "fp64" else 700000)
    elif kind == "bif2d":
        precision, system = rng.choice(["fp32", "fp32", "fp64"]), "chameleon"
        n = _log(rng, 24, 64 if precision == "fp64" else 300)
        tMax, transient = round(rng.uniform(100.0, 400.0), 1), round(rng.uniform(200.0, 2000.0), 1)
    elif kind == "lle":
        precision = rng.choice(["ff32", "fp32", "fp64"])
        n = _log(rng, 20, {"ff32": 512, "fp32": 700, "fp64": 100}[precision])
        tMax = round(rng.uniform(100.0, 500.0 if precision != "fp64" else 250.0), 1)
    elif kind in ("basins_dbscan", "basins"):
        precision = rng.choice(["fp32", "fp32", "fp64"])
        n = _log(rng, 40, 150 if precision == "fp64" else 1024)
        tMax, transient = round(rng.uniform(20.0, 50.0), 1), round(rng.uniform(50.0, 200.0), 1)
    elif kind == "spectrum":
        precision = rng.choice(["fp32", "fp32", "fp64"])
        n = _log(rng, 20, 64 if precision == "fp64" else 384)
    elif kind == "dbscan":
        return dict(kind=kind, system="", precision="fp64", nPts=int(_log(rng, 2000, 4000000)),
                    dims=rng.choice([2, 3]))
    else:
        return dict(kind=kind, system="", precision="fp32", nPts=int(_log(rng, 5000, 100000)),
                    jobs=rng.choice([6, 9, 12, 15]))
    return dict(kind=kind, system=system, precision=precision, nPts=int(n), tMax=tMax, transient=transient)


def _steps(t):
    return int(t / H)


def _cap(case):
    return max(1, min(64, _steps(case["tMax"]) // 2))


def _blocks(tMax):
    """Benettin blocks and steps per block of an LLE horizon."""
    ntp = int(NT / H)
    return _steps(tMax) // ntp + 2, ntp


def _jittered(rng, start, ranges):
    """Starting point and range ends as another user of the same workload would choose them."""
    ic = [x + rng.uniform(-0.05, 0.05) for x in start]
    width = [ranges[2 * (i // 2) + 1] - ranges[2 * (i // 2)] for i in range(len(ranges))]
    # ends move inwards only: every parameter stays in the workload's range
    rg = [r + (1 if i % 2 == 0 else -1) * rng.uniform(0.0, 0.02) * w for i, (r, w) in enumerate(zip(ranges, width))]
    return ic, rg


def _zeros(n, dtype):
    return torch.zeros(n, dtype=dtype, device="cuda")


def _points(n, dims, seed):
    """Normalised features as a basin map has them: points that settled on a few attractors (tight), a chaotic
    attractor's finite-time means (an elongated cloud), stragglers."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = dict(generator=g, device="cuda", dtype=torch.float64)
    centres = 0.1 + 0.8 * torch.rand(4, dims, **r)
    which = torch.rand(n, **r)
    pts = torch.randn(n, dims, **r)
    scale = torch.tensor([0.05, 0.02, 0.03], device="cuda", dtype=torch.float64)[:dims]
    pick = (which > 0.35).long() + (which > 0.6).long() + (which > 0.8).long()
    spread = torch.where((pick == 3)[:, None], scale, torch.full_like(scale, 2e-4))
    pts = centres[pick] + pts * spread
    stray = which > 0.997
    pts[stray] = torch.rand(int(stray.sum()), dims, **r)
    return pts.clamp_(0.0, 1.0).contiguous()


def _batch(case, rng):
    """Jobs of every kind and RK4 system, sizes over two decades below the largest."""
    b = C.Batch(device=True)
    work = 0.0
    for k in range(case["jobs"]):
        kind = ("bif1d", "lle", "basins")[k % 3]
        system = RK4[(k // 3) % 3]
        n = max(100, int(case["nPts"] * 10 ** (-2.0 * k / max(1, case["jobs"] - 1))))
        m = max(8, int(n ** 0.5))
        transient = round(20.0 + 80.0 * ((k * 7) % 10) / 10.0, 2)
        if kind == "bif1d":
            ic, rg = _jittered(rng, START[system], SWEEP1[system][1])
            b.add_bifurcation1d(system, 100.0, n, H, ic, rg, SWEEP1[system][0], 0, 1e4, transient, VALUES[system])
            work += n * (_steps(transient) + _steps(100.0)) * STEP_FLOPS[system]
        elif kind == "lle":
            ic, rg = _jittered(rng, START[system], SWEEP2[system][1])
            b.add_lle2d(system, 100.0, NT, m, H, EPS, ic, rg, SWEEP2[system][0], transient, VALUES[system])
            nb, ntp = _blocks(100.0)
            work += m * m * (_steps(transient) + 2 * nb * ntp) * STEP_FLOPS[system]
        else:
            ic, rg = _jittered(rng, BASIN_START[system], [-30.0, 30.0, -30.0, 30.0])
            b.add_basins(system, 50.0, m, H, ic, rg, [0, 1], 0, 1e8, transient, BASIN_VALUES[system])
            work += m * m * (_steps(transient) + _steps(50.0)) * STEP_FLOPS[system]
    return b, work


def _inputs(case, seed):
    rng = random.Random(seed)
    system = case["system"]
    if case["kind"] in ("basins", "basins_dbscan"):
        ic, rg = _jittered(rng, BASIN_START[system], [-30.0, 30.0, -30.0, 30.0])
        return ic, rg, [0, 1], BASIN_VALUES[system]
    mut, base = (SWEEP1 if case["kind"] == "bif1d" else SWEEP2)[system]
    ic, rg = _jittered(rng, START[system], base)
    return ic, rg, mut, VALUES[system]


def prepare(case, seed):
    kind, n = case["kind"], case["nPts"]
    if kind == "dbscan":
        return dict(case=case, points=_points(n, case["dims"], seed), out=_zeros(n, torch.int32))
    if kind == "batch":
        b, _ = _batch(case, random.Random(seed))
        return dict(case=case, batch=b.prepare())
    ic, rg, mut, values = _inputs(case, seed)
    st = dict(case=case, ic=np.array(ic), ranges=np.array(rg), mut=np.array(mut, np.int32), values=np.array(values))
    i32, f64 = torch.int32, torch.float64
    if kind == "bif1d":
        cap = _cap(case)
        st["out"] = dict(counts=_zeros(n, i32), flags=_zeros(n, i32), first=_zeros(n, f64),
                         peaks=_zeros((n, cap), f64), intervals=_zeros((n, cap), f64))
    elif kind == "bif2d":
        st["out"] = dict(labels=_zeros(n * n, i32), counts=_zeros(n * n, i32))
    elif kind == "lle":
        st["out"] = _zeros(n * n, f64)
    elif kind == "spectrum":
        st["out"] = _zeros((n * n, 3), f64)
    elif kind == "basins_dbscan":
        st["out"] = dict(labels=_zeros(n * n, i32), flags=_zeros(n * n, i32), features=_zeros((n * n, 3), f64))
    else:
        st["out"] = dict(labels=_zeros(n * n, i32), avg_peaks=_zeros(n * n, f64), avg_intervals=_zeros(n * n, f64),
                         flags=_zeros(n * n, i32))
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "dbscan":
        return C.dbscan(st["points"], 0.05, 8, out=st["out"])
    if kind == "batch":
        return st["batch"].replay()
    system, n, tMax, tr, prec = case["system"], case["nPts"], case["tMax"], case["transient"], case["precision"]
    ic, rg, mut, values, out = st["ic"], st["ranges"], st["mut"], st["values"], st["out"]
    if kind == "bif1d":
        return C.bifurcation1d(system, tMax, n, H, ic, rg, mut, 0, 1e4, tr, values, peakCapacity=_cap(case),
                               precision=prec, out=out)
    if kind == "bif2d":
        return C.bifurcation2d(system, tMax, n, H, ic, rg, mut, 0, 1e4, tr, values, eps=0.001, precision=prec,
                               out=out)
    if kind == "lle":
        return C.lle2d(system, tMax, NT, n, H, EPS, ic, rg, mut, tr, values, precision=prec, out=out)
    if kind == "spectrum":
        return C.lyapunov_spectrum(system, 2, tMax, NT, n, H, EPS, ic, rg, mut, tr, values, precision=prec, out=out)
    if kind == "basins_dbscan":
        return C.basins_dbscan(system, tMax, n, H, ic, rg, mut, 0, 1e8, tr, values, eps=0.05, minPts=8,
                               precision=prec, out=out)
    return C.basins(system, tMax, n, H, ic, rg, mut, 0, 1e8, tr, values, eps=0.05, precision=prec, out=out)


def work(case):
    kind, n = case["kind"], case["nPts"]
    if kind == "dbscan":
        # the features read, the labels written; a distance test per point and dimension at least
        return {"bytes": n * (8 * case["dims"] + 4), "flops": 3 * n * case["dims"]}
    if kind == "batch":
        total = 0.0
        for k in range(case["jobs"]):
            sort, system = ("bif1d", "lle", "basins")[k % 3], RK4[(k // 3) % 3]
            p = max(100, int(case["nPts"] * 10 ** (-2.0 * k / max(1, case["jobs"] - 1))))
            m = max(8, int(p ** 0.5))
            tr = _steps(round(20.0 + 80.0 * ((k * 7) % 10) / 10.0, 2))
            nb, ntp = _blocks(100.0)
            steps = {"bif1d": p * (tr + _steps(100.0)), "lle": m * m * (tr + 2 * nb * ntp),
                     "basins": m * m * (tr + _steps(50.0))}[sort]
            total += steps * STEP_FLOPS[system]
        return {"bytes": 24 * case["nPts"], "flops": total}
    f = STEP_FLOPS[case["system"]]
    s, b = _steps(case["transient"]), _steps(case["tMax"])
    nb, ntp = _blocks(case["tMax"])
    if kind == "bif1d":  # counts, flags, first sample; the kept peaks and intervals are fewer than the rows hold
        return {"bytes": n * 16, "flops": n * (s + b) * f}
    if kind == "bif2d":
        return {"bytes": n * n * 8, "flops": n * n * (s + b) * f}
    if kind == "lle":
        return {"bytes": n * n * 8, "flops": n * n * (s + 2 * nb * ntp) * f}
    if kind == "spectrum":
        return {"bytes": n * n * 24, "flops": n * n * (s + 4 * nb * ntp) * f}
    return {"bytes": n * n * (32 if kind == "basins_dbscan" else 24), "flops": n * n * (s + b) * f}


# ---- plain FP64 ---------------------------------------------------------------
def _field(system, x, a):
    if system == "lorenz":
        return torch.stack([a[0] * (x[1] - x[0]), x[0] * (a[1] - x[2]) - x[1], x[0] * x[1] - a[2] * x[2]])
    if system == "rossler":
        return torch.stack([-x[1] - x[2], x[0] + a[0] * x[1], a[1] + x[2] * (x[0] - a[2])])
    return torch.stack([a[0] * (x[1] - x[0]), (a[2] - a[0]) * x[0] - x[0] * x[2] + a[2] * x[1],
                        x[0] * x[1] - a[1] * x[2]])


def _rk4(system, x, a):
    k1 = _field(system, x, a)
    k2 = _field(system, x + 0.5 * H * k1, a)
    k3 = _field(system, x + 0.5 * H * k2, a)
    k4 = _field(system, x + H * k3, a)
    x.add_((H / 6.0) * (k1 + 2.0 * (k2 + k3) + k4))


def _graph(f):
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        f()
    torch.cuda.current_stream().wait_stream(s)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        f()
    return g


def _grid(case, seed):
    """State [3, n*n] and parameters (each [n*n]) of a 2-D parameter map: point j*n + i."""
    n = case["nPts"]
    ic, rg, mut, values = _inputs(case, seed)
    d = dict(device="cuda", dtype=torch.float64)
    k = torch.arange(n, **d)
    axis = [rg[2 * q] + k * ((rg[2 * q + 1] - rg[2 * q]) / (n - 1)) for q in (0, 1)]
    a = [torch.full((n * n,), v, **d) for v in values]
    a[mut[0]] = axis[0].repeat(n)
    a[mut[1]] = axis[1].repeat_interleave(n)
    return torch.tensor(ic, **d)[:, None].repeat(1, n * n).contiguous(), a


def _settle(case, x, a):
    keep = x.clone()
    g = _graph(lambda: [_rk4(case["system"], x, a) for _ in range(10)])
    x.copy_(keep)
    n = _steps(case["transient"])
    for _ in range(n // 10):
        g.replay()
    for _ in range(n % 10):
        _rk4(case["system"], x, a)


def exact(case, seed):
    """Lyapunov maps and spectra in FP64. A sweep's peaks, a basin's means and the labels made of them belong to
    single chaotic orbits, which no other arithmetic follows to the end: they have no such value. Maps too large
    for plain FP64 in about 20 seconds are left out."""
    kind, n = case["kind"], case["nPts"]
    if kind == "lle" and n <= 260 and case["system"] != "rossler":
        # not the Rossler map, whose small exponents (0 to 0.1) move by a tenth of themselves with the rounding
        # of the orbit
        return _exact_lle(case, seed)
    if kind == "spectrum" and n <= 400:
        return _exact_spectrum(case, seed)
    return None


def _exact_lle(case, seed):
    system = case["system"]
    x, a = _grid(case, seed)
    _settle(case, x, a)
    n = x.shape[1]
    both = torch.stack([x, x], 1).reshape(3, 2 * n)  # the orbit and its twin
    both[0, n:] += EPS
    a2 = [v.repeat(2) for v in a]
    nb, ntp = _blocks(case["tMax"])
    total = torch.zeros(n, device="cuda", dtype=torch.float64)

    def block():
        for _ in range(ntp):
            _rk4(system, both, a2)
        d = both[:, n:] - both[:, :n]
        r = d.square().sum(0).sqrt() / EPS
        total.add_(r.log())
        both[:, n:] = both[:, :n] + d / r

    keep = both.clone()
    g = _graph(block)
    both.copy_(keep)
    total.zero_()
    for _ in range(nb):
        g.replay()
    return total / case["tMax"]


def _exact_spectrum(case, seed):
    system = case["system"]
    x, a = _grid(case, seed)
    _settle(case, x, a)
    n = x.shape[1]
    every = x.repeat(1, 4)  # the orbit and a twin along each axis
    for j in range(3):
        every[j, (j + 1) * n:(j + 2) * n] += EPS
    a4 = [v.repeat(4) for v in a]
    nb, ntp = _blocks(case["tMax"])
    total = torch.zeros(n, 3, device="cuda", dtype=torch.float64)

    def block():
        for _ in range(ntp):
            _rk4(system, every, a4)
        x0 = every[:, :n]
        made = []
        for j in range(3):
            d = every[:, (j + 1) * n:(j + 2) * n] - x0
            w = d.clone()
            for b in made:
                w = w - ((d * b).sum(0) / (b * b).sum(0)) * b
            made.append(w)
        for j, w in enumerate(made):
            r = w.square().sum(0).sqrt()
            total[:, j] += (r / EPS).log()
            every[:, (j + 1) * n:(j + 2) * n] = x0 + w / r * EPS

    keep = every.clone()
    g = _graph(block)
    every.copy_(keep)
    total.zero_()
    for _ in range(nb):
        g.replay()
    return total / case["tMax"]
