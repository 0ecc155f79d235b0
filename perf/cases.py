"""Timed cases of the counting engine: the calls its users make, over the sizes they make them at.

A process keeps one engine, as a user's program does, and every case counts catalogs of its own in it, so
that each pass plans and counts what the engine has not just counted.  All outputs are histograms of counts:
whole numbers, the same whatever path computes them.

listed() are the cases, draw(rng) makes more of the same ranges, prepare/run/work/exact serve both.
"""
import ctypes
import importlib
import math
import platform

import numpy as np
import torch

synth = importlib.import_module("3pcf_gb300.synth")
tpcf = importlib.import_module("3pcf_gb300.tpcf")
voxels = importlib.import_module("3pcf_gb300.voxels")

# binnings: the benchmark's triangle binning, the reference's own default triangle binning, JBJ, three-side
# (compat and clean) and pair binnings
AXES = {
    "tp": [(8, 2.0, 10.0), (8, 1.0, 3.0), (16, 0.0, 1.0)],
    "tp_default": [(50, 2.0, 12.0), (16, 0.9, 4.1), (25, 0.0, 1.0)],
    "jbj": [(8, 2.0, 10.0), (8, 0.2, 1.0), (10, 0.0, 1.0)],
    "three": [(16, 0.0, 40.0)],
    "lattice": [(32, 0.0, 32.0)],
    "pair": [(700, 0.0, 70.0)],
}
# longest side (separation) that can be counted
REACH = {"tp": 40.0, "tp_default": 61.2, "jbj": 60.0, "three": 40.0, "lattice": 32.0, "pair": 70.0}
# arithmetic per triangle within reach (per pair): side bins, ratios, angles, bins
OPS = {"tp": 58, "tp_default": 58, "jbj": 40, "three": 10, "lattice": 10, "pair": 8}
LOOPS = {"same": tpcf.LOOP_SAME, "one": tpcf.LOOP_ONE, "all": tpcf.LOOP_ALL}
# the estimator's four histograms: roles of the data (D) and random (R) catalog and the loop nest
FOUR = [("DDD", "same"), ("DDR", "one"), ("DRR", "one"), ("RRR", "same")]
PAIRS = [("DD", "same"), ("DR", "one"), ("RR", "same")]
NATIVE_NAN = tpcf.NAN_ZERO if platform.machine() == "aarch64" else tpcf.NAN_INT_MIN

_engine = None


def engine():
    global _engine
    if _engine is None:
        _engine = tpcf.Engine(0)
    return _engine


def listed():
    return [
        # the smallest estimator: four triangle histograms of a small field, where launches, planning and the
        # tail of a launch count
        {"name": "tp_1k", "op": "tp", "nd": 1000, "nr": 1000},
        # the headline workload as a program calls it: catalogs from host arrays, four histograms, release
        {"name": "tp_10k_call", "op": "tp_call", "nd": 10000, "nr": 10000},
        # the reference's own default binning (50 x 16 x 25 bins, ratios up to 4.1) on a narrow survey field
        {"name": "tp_default_bins", "op": "tp_default", "nd": 5013, "nr": 4999},
        # a survey light cone: the four histograms and every neighbour-voxel job, summed per kind
        {"name": "voxel_cone", "op": "voxel", "nd": 20000, "nr": 20000, "grid": 4},
        # a burst of jobs of many sizes on resident catalogs, submitted and waited for
        {"name": "serving_burst", "op": "serving", "jobs": 40, "nmax": 6000},
        # the JBJ shape parametrization
        {"name": "jbj_5k", "op": "jbj", "nd": 5000, "nr": 5000},
        # the double-precision geometry that the correlation function's error is quoted against
        {"name": "geometry_1k", "op": "geometry", "nd": 1000, "nr": 1000},
        # the three-side histogram in the reference's own mode, DDD and RRR of the reference's sample size
        {"name": "three_side_1k", "op": "three", "nd": 1000, "nr": 1000, "mixed": False},
        # ... and with the cross terms D-D-R and D-R-R of larger, odd-sized catalogs
        {"name": "three_side_cross_3k", "op": "three", "nd": 3001, "nr": 2777, "mixed": True},
        # the three-side histogram restricted to its range, 32 bins, points on bin edges
        {"name": "lattice_150k", "op": "lattice", "nd": 150000},
        # the two-point function: DD, DR, RR in 700 bins
        {"name": "pairs_50k", "op": "pair", "nd": 50000, "nr": 50000},
        # pair counts of device arrays without allocation: the smallest and latency-bound call
        {"name": "pairs_device_5k", "op": "noalloc", "nd": 5000, "nr": 4801},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["tp", "tp_call", "tp_default", "voxel", "serving", "jbj", "geometry", "three", "lattice", "pair",
                     "noalloc"])
    if op == "voxel":
        n = size(2000, 20000)
        return {"op": op, "nd": n, "nr": n + rng.randrange(500), "grid": rng.choice([3, 4])}
    if op == "serving":
        return {"op": op, "jobs": rng.randrange(8, 41), "nmax": size(1500, 6000)}
    if op == "lattice":
        return {"op": op, "nd": size(2000, 150000)}
    if op == "three":
        mixed = rng.random() < 0.5
        top = 3000 if mixed else 4000
        return {"op": op, "nd": size(300, top), "nr": size(300, top), "mixed": mixed}
    lo, hi = {"tp": (500, 10000), "tp_call": (500, 10000), "tp_default": (500, 5000), "jbj": (500, 5000),
              "geometry": (300, 1000), "pair": (1000, 50000), "noalloc": (1000, 40000)}[op]
    return {"op": op, "nd": size(lo, hi), "nr": size(lo, hi)}


# ---------------------------------------------------------------------------------------------------------
# inputs

def catalogs(case, seed):
    """The host arrays of a case: {"D": points, "R": points}."""
    op, nd, nr = case["op"], case.get("nd", 0), case.get("nr", 0)
    if op == "lattice":  # four points in a thousand units of volume, three of ten on the integer lattice
        return {"D": synth.lattice_mix(nd, box=500.0 * (nd / 500000.0) ** (1.0 / 3.0), frac=0.3, seed=seed)}
    if op == "voxel":
        return {"D": synth.lightcone(nd, clustered=True, n_blobs=max(1, nd // 50), seed=seed),
                "R": synth.lightcone(nr, seed=seed + 500009)}
    if op == "tp_default":
        return {"D": synth.lightcone(nd, clustered=True, n_blobs=max(1, nd // 25), half_angle_deg=2.5, seed=seed),
                "R": synth.lightcone(nr, half_angle_deg=2.5, seed=seed + 500009)}
    box = 200.0 if op == "tp_call" else 100.0
    return {"D": synth.blobs(nd, n_blobs=max(2, nd // 500), sigma=5.0, box=100.0, seed=seed),
            "R": synth.uniform(nr, box=box, seed=seed + 500009)}


class State:
    """What a program holds before the call; its catalogs are released with it."""

    def __init__(self):
        self.handles = []

    def add(self, points):
        h = engine().catalog(points)
        self.handles.append(h)
        return h

    def __del__(self):
        for h in self.handles:
            try:
                engine().release(h)
            except Exception:  # the engine may be gone at the process's end
                pass


def _spec(name, loop, **more):
    kind = {"tp": tpcf.TRIANGLE, "tp_default": tpcf.TRIANGLE, "jbj": tpcf.TRIANGLE_JBJ, "three": tpcf.THREE_SIDE,
            "lattice": tpcf.THREE_SIDE, "pair": tpcf.PAIR}[name]
    return tpcf.make_spec(kind, LOOPS[loop], AXES[name], nan_policy=NATIVE_NAN, **more)


def _set_of(case):
    """(binning, jobs as (roles, loop), spec options) of the cases that count one batch."""
    op = case["op"]
    if op == "geometry":
        return "tp", FOUR, {"precision": tpcf.GEOMETRY_FP64}
    if op == "three":
        return "three", [(r, "all") for r in (("DDD", "DDR", "DRR", "RRR") if case["mixed"] else ("DDD", "RRR"))], {}
    if op == "lattice":
        return "lattice", [("DDD", "all")], {"overflow": tpcf.OVERFLOW_CLEAN}
    if op in ("pair", "noalloc"):
        return "pair", PAIRS, {}
    return {"tp_call": "tp", "voxel": "tp"}.get(op, op), FOUR, {}


def prepare(case, seed):
    s = State()
    s.case = case
    op = case["op"]
    if op == "serving":
        return _prepare_serving(s, case, seed)
    cats = catalogs(case, 10 * seed + 1)
    name, jobs, more = _set_of(case)
    if op == "noalloc":
        s.dev = {k: [torch.from_numpy(np.ascontiguousarray(v[:, a])).cuda() for a in range(3)] for k, v in cats.items()}
        s.hist = [torch.empty(AXES["pair"][0][0], dtype=torch.int64, device="cuda") for _ in jobs]
        s.jobs = jobs
        return s
    s.specs = [_spec(name, loop, **more) for _, loop in jobs]
    if op == "tp_call":
        s.cats, s.roles = cats, [r for r, _ in jobs]
        return s
    if op == "voxel":
        return _prepare_voxel(s, case, cats)
    h = {k: s.add(v) for k, v in cats.items()}
    s.jobs = [engine().job([h[x] for x in roles]) for roles, _ in jobs]
    return s


def _prepare_voxel(s, case, cats):
    """Voxel-ordered catalogs, the four full counts (outputs 0-3) and the voxel jobs (outputs 4-7)."""
    grid = (case["grid"],) * 3
    pts = np.concatenate([cats["D"], cats["R"]]).astype(np.float64)
    lo, hi = pts.min(0), pts.max(0) + 1e-6
    h, ranges = {}, {}
    for k, v in cats.items():
        order, start, end = voxels.voxel_order(v, lo, hi, grid)
        h[k], ranges[k] = s.add(v[order]), (start, end)
    specs, jobs, outs = [], [], []
    spec = {loop: _spec("tp", loop) for loop in LOOPS}
    for o, (roles, loop) in enumerate(FOUR):
        specs.append(spec[loop])
        jobs.append(engine().job([h[x] for x in roles]))
        outs.append(o)
    for o, (kind, _) in enumerate(FOUR):
        for roles, rng, loop, glob in voxels.spatial_jobs(kind, ranges["D"], ranges["R"], grid):
            specs.append(spec[loop])
            jobs.append(engine().job([h[x] for x in roles], rng, global_index=glob))
            outs.append(4 + o)
    s.batch = engine().prepare(specs, jobs, outs, 8)
    return s


def _serving_mix(case):
    """Catalog sizes, and the jobs (binning, roles, loop, data catalog, random catalog): the same for every seed."""
    rng = np.random.Generator(np.random.PCG64(case["jobs"] + case["nmax"]))
    sizes = np.exp(rng.uniform(np.log(500), np.log(case["nmax"]), size=6)).astype(int)
    jobs = []
    for _ in range(case["jobs"]):
        a = int(rng.integers(6))
        b = (a + 2 * int(rng.integers(3))) % 6  # of the same family
        if rng.random() < 0.7:
            jobs.append(("tp",) + FOUR[int(rng.integers(4))] + (a, b))
        else:
            jobs.append(("pair",) + PAIRS[int(rng.integers(3))] + (a, b))
    return [int(n) for n in sizes], jobs


def _prepare_serving(s, case, seed):
    sizes, jobs = _serving_mix(case)
    h = []
    for i, n in enumerate(sizes):
        if i % 2 == 0:
            d, r = synth.blobs(n, n_blobs=max(1, n // 500), seed=1000 * seed + i), synth.uniform(n, seed=2000 * seed + i)
        else:
            d = synth.lightcone(n, clustered=True, n_blobs=max(1, n // 50), half_angle_deg=2.5, seed=1000 * seed + i)
            r = synth.lightcone(n, half_angle_deg=2.5, seed=2000 * seed + i)
        h.append((s.add(d), s.add(r)))
    s.specs, s.jobs = [], []
    for name, roles, loop, a, b in jobs:
        s.specs.append(_spec(name, loop))
        s.jobs.append(engine().job([h[a][0] if x == "D" else h[b][1] for x in roles]))
    return s


# ---------------------------------------------------------------------------------------------------------
# one pass

def run(s):
    op, e = s.case["op"], engine()
    if op == "tp_call":
        h = {k: e.catalog(v) for k, v in s.cats.items()}
        out = e.count_batch(s.specs, [e.job([h[x] for x in roles]) for roles in s.roles])
        for v in h.values():
            e.release(v)
    elif op == "voxel":
        out = e.count_prepared(s.batch)
    elif op == "serving":
        tickets = [e.submit(sp, jb) for sp, jb in zip(s.specs, s.jobs)]
        out = [e.wait(t, sp) for t, sp in zip(tickets, s.specs)]
    elif op == "noalloc":
        n, lo, hi = AXES["pair"][0]
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        for (roles, loop), hist in zip(s.jobs, s.hist):
            a, b = s.dev[roles[0]], s.dev[roles[1]]
            st = tpcf.lib().tpcf_pair_count_noalloc(
                a[0].data_ptr(), a[1].data_ptr(), a[2].data_ptr(), a[0].numel(),
                b[0].data_ptr(), b[1].data_ptr(), b[2].data_ptr(), b[0].numel(),
                LOOPS[loop], lo, hi, n, hist.data_ptr(), stream)
            if st != 0:
                raise RuntimeError(tpcf.status_string(st))
        return list(s.hist)
    else:
        out = e.count_batch(s.specs, s.jobs)
    return [h.view(np.int64) for h in out]


# ---------------------------------------------------------------------------------------------------------
# the work of a pass

def _within(a, b, reach):
    d2 = ((a[:, None, :].astype(np.float64) - b[None, :, :]) ** 2).sum(-1)
    return d2 < reach * reach


def _tuples(cats, reach, sample=64):
    """Distinct triples (pairs, for two roles) of points that are all within reach of one another: every point of a
    sample of the first role with the neighbours among a subset of the others, scaled up."""
    a = cats[0]
    a = a[:: max(1, len(a) // sample)]
    rest, scale = [], len(cats[0]) / len(a)
    for c in cats[1:]:
        step = max(1, len(c) // 2000)
        rest.append(c[::step])
        scale *= len(c) / len(rest[-1])
    near = [_within(a, c, reach) for c in rest]
    if len(rest) == 1:
        return float(near[0].sum()) * scale
    got = 0.0
    for i in range(len(a)):
        b, c = rest[0][near[0][i]], rest[1][near[1][i]]
        pb, pc = max(1, len(b) // 200), max(1, len(c) // 200)
        if len(b) and len(c):
            got += float(_within(b[::pb], c[::pc], reach).mean()) * len(b) * len(c)
    return got * scale


def work(case):
    """Bytes: the coordinates once and the histograms once; operations: the arithmetic of each distinct triple (pair)
    within reach, counted on a sample of the inputs."""
    if case["op"] == "serving":
        sizes, jobs = _serving_mix(case)
        total, flops = sum(24 * n for n in sizes), 0.0
        for name, roles, _, a, b in jobs:
            kind = "tp" if a % 2 == 0 else "tp_default"
            cats = catalogs({"op": kind, "nd": sizes[a], "nr": sizes[b]}, 1)
            flops += OPS[name] * _tuples([cats[x] for x in roles], REACH[name], 16) / _repeats(roles)
            total += 8 * _bins(name)
        return {"bytes": total, "flops": flops}
    cats = catalogs(case, 1)
    name, jobs, _ = _set_of(case)
    copies = 2 if case["op"] == "voxel" else 1  # the full counts and the voxel sums
    flops = sum(OPS[name] * _tuples([cats[x] for x in roles], REACH[name]) / _repeats(roles) for roles, _ in jobs)
    return {"bytes": sum(12 * len(v) for v in cats.values()) + copies * 8 * _bins(name) * len(jobs),
            "flops": copies * flops}


def _bins(name):
    n = 1
    for axis in AXES[name]:
        n *= axis[0]
    return n ** 3 if name in ("three", "lattice") else n


def _repeats(roles):
    """Orders in which one set of points of these roles comes up."""
    return math.prod(math.factorial(roles.count(x)) for x in set(roles))


def exact(case, seed):
    """Counts are whole numbers, defined by the reference's single-precision arithmetic: they have to be equal, and no
    64-bit value stands in for them."""
    return None
