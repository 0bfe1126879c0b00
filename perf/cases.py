"""The calls whose speed this repository tracks, with their inputs and sizes.

Each case is one pass through the package's public entry points at a size
that its users run: the whole host-buffer call, its layers (start points,
PSO seeding, the BFGS of each kernel layout, bit-reproducible exact mode with
recorded trajectories) and the persistent batches.  Sizes and objectives are
those of bench.py's workloads and of the tests, or plain round numbers with
ragged ones between them.  Stop-early is off throughout (which runs it stops
depends on timing), so a pass has one answer.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import zeus_b200 as zb
from zeus_b200 import device as zd

BOUNDS = {"rosenbrock": (-5.0, 5.0), "rastrigin": (-5.12, 5.12),
          "ackley": (-32.768, 32.768), "gaussian": (-5.0, 5.0)}
# the dimensions each objective is built for
DIMS = {"rosenbrock": (2, 4, 8, 10, 16, 32, 64, 128), "rastrigin": (2, 10, 16),
        "ackley": (2, 10, 30), "gaussian": (2, 8, 32, 150)}
NBINS = 100          # dijet spectrum bins
RUNS_PER_TOY = 256   # starts per dijet toy
NEVER = 1 << 30      # a required-convergence count that is not reached

# The mixed batch's classes: objective, dimension, and the layout and tile
# that zeus_b200.autotune picks for each on a B200.  They are given here
# instead of tuned on the spot: a pick by timing may differ from process to
# process, and the layouts do not round alike.
MIXED = (("rosenbrock", 128, zb.LAYOUT_ROWS, 0), ("rosenbrock", 64, zb.LAYOUT_ROWS, 0),
         ("ackley", 30, zb.LAYOUT_TILE, 32), ("rosenbrock", 32, zb.LAYOUT_ROWS, 0),
         ("rosenbrock", 8, zb.LAYOUT_TILE, 32), ("rosenbrock", 2, zb.LAYOUT_THREAD, 0))


def listed():
    return [
        # the smallest whole call: a small correlated fit, a short swarm;
        # launches and host work are most of it
        dict(name="call_gaussian8", what="call", obj="gaussian", dim=8, n=200, pso=5),
        # the reference's first example: 2-D Rosenbrock from a swarm of 1024
        dict(name="call_rosenbrock2", what="call", obj="rosenbrock", dim=2, n=1024, pso=10),
        # start points for a large multi-start search
        dict(name="starts_10", what="starts", dim=10, n=1000003, prng="philox"),
        # swarm seeding of a multimodal search
        dict(name="pso_rastrigin10", what="pso", obj="rastrigin", dim=10, n=16384, iters=20,
             prng="philox"),
        # swarm seeding of the 150-D Gaussian, the largest example of the reference
        dict(name="pso_gaussian150", what="pso", obj="gaussian", dim=150, n=1024, iters=10,
             prng="philox"),
        # small-dimension BFGS, a ragged number of starts
        dict(name="bfgs_rosenbrock8", what="bfgs", obj="rosenbrock", dim=8, n=4099,
             gradient="adjoint", max_iter=10000),
        # mid-dimension BFGS of a multimodal search
        dict(name="bfgs_rastrigin10", what="bfgs", obj="rastrigin", dim=10, n=16384,
             gradient="adjoint", max_iter=10000),
        # large-dimension BFGS, one block a run
        dict(name="bfgs_rosenbrock64", what="bfgs", obj="rosenbrock", dim=64, n=1024,
             gradient="adjoint", max_iter=10000),
        # the 150-D Gaussian's BFGS: a dense matrix shared by every run
        dict(name="bfgs_gaussian150", what="bfgs", obj="gaussian", dim=150, n=1024,
             gradient="adjoint", max_iter=10000),
        # the default benchmark: six classes of uneven dimension in one batch
        dict(name="batch_mixed", what="mixed", per_class=1365),
        # toy fits of a binned spectrum, then d(fit)/d(counts) of each best fit
        dict(name="batch_dijet", what="dijet", toys=128),
        # bit-reproducible runs with dual-number gradients and every iterate
        # recorded
        dict(name="exact_rosenbrock10", what="exact", obj="rosenbrock", dim=10, n=512,
             max_iter=300),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(("call", "starts", "pso", "pso", "bfgs", "bfgs", "bfgs", "mixed",
                       "dijet", "exact"))
    if what == "starts":
        return dict(what=what, dim=rng.choice((2, 3, 10, 32, 100, 150)),
                    n=_log_int(rng, 500, 1 << 20), prng=rng.choice(("philox", "sobol")))
    if what == "mixed":
        return dict(what=what, per_class=_log_int(rng, 100, 1365))
    if what == "dijet":
        return dict(what=what, toys=_log_int(rng, 2, 127))
    obj = rng.choice(("rosenbrock", "rastrigin", "ackley", "gaussian"))
    if what == "call":
        return dict(what=what, obj=obj, dim=rng.choice([d for d in DIMS[obj] if d <= 32]),
                    n=_log_int(rng, 64, 8192), pso=rng.choice((-1, 5, 10, 20)))
    if what == "pso":
        dim = rng.choice(DIMS[obj])
        return dict(what=what, obj=obj, dim=dim, n=_log_int(rng, 64, 32768 if dim <= 32 else 4096),
                    iters=rng.choice((5, 10, 20)), prng=rng.choice(("philox", "philox", "sobol")))
    if what == "bfgs":
        dim = rng.choice(DIMS[obj])
        grads = ("adjoint", "adjoint", "dual") if dim <= 32 else ("adjoint",)
        return dict(what=what, obj=obj, dim=dim, n=_log_int(rng, 64, 16384 if dim <= 32 else 1024),
                    gradient=rng.choice(grads), max_iter=rng.choice((500, 10000)))
    return dict(what=what, obj=obj, dim=rng.choice([d for d in DIMS[obj] if d <= 32]),
                n=_log_int(rng, 32, 512), max_iter=rng.choice((100, 300)))


def _objective(obj, dim):
    if obj == "gaussian":
        return zb.Gaussian(zb.gaussian_matrix(dim))
    return {"rosenbrock": zb.Rosenbrock, "rastrigin": zb.Rastrigin, "ackley": zb.Ackley}[obj](dim)


def _uniform(gen, n, dim, lo, hi):
    u = torch.rand((n, dim), dtype=torch.float64, device="cuda", generator=gen)
    return lo + (hi - lo) * u


def _dijet(toys, seed):
    """Poisson toys of a falling dijet spectrum, one after another: log-spaced
    bins in x = m/13000 over [0.085, 0.54], 1e6 events."""
    edges = np.geomspace(0.085, 0.54, NBINS + 1)
    x = 0.5 * (edges[1:] + edges[:-1])
    lam = (1 - x) ** 10.0 / x ** (5.0 + 0.1 * np.log(x))
    lam *= 1e6 / lam.sum()
    k = np.random.default_rng(seed).poisson(np.tile(lam, (toys, 1))).astype(np.int32)
    return zb.PoissonNLL(k.reshape(-1), np.tile(x, toys))


def prepare(case, seed):
    what = case["what"]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    s = {"case": case, "seed": 42 + 7919 * seed}
    if what == "starts":
        return s
    if what == "mixed":
        jobs = []
        for obj, dim, layout, tile in MIXED:
            x0 = _uniform(gen, case["per_class"], dim, *BOUNDS[obj])
            jobs.append(zb.BatchJob(zd.DeviceProblem(_objective(obj, dim)), x0, layout=layout,
                                    tile=tile))
        s["batch"] = zd.Batch(jobs)
        return s
    if what == "dijet":
        n = case["toys"] * RUNS_PER_TOY
        # one warp per run, what autotune picks for this fit
        job = zb.BatchJob(zd.DeviceProblem(_dijet(case["toys"], seed)),
                          _uniform(gen, n, 4, 0.0, 10.0), layout=zb.LAYOUT_TILE, tile=32,
                          runs_per_instance=RUNS_PER_TOY)
        s["batch"] = zd.Batch([job])
        return s
    obj = _objective(case["obj"], case["dim"])
    if what == "call":
        s["obj"] = obj
        return s
    s["problem"] = zd.DeviceProblem(obj)
    if what in ("bfgs", "exact"):
        s["x0"] = _uniform(gen, case["n"], case["dim"], *BOUNDS[case["obj"]])
    return s


def _runs(r):
    return {"fval": r.fval, "status": r.status, "iter": r.iter, "gnorm": r.gnorm, "x": r.x,
            "counters": r.counters}


def run(s):
    c, what = s["case"], s["case"]["what"]
    if what == "call":
        r = zb.Zeus(s["obj"], *BOUNDS[c["obj"]], c["n"], 10000, c["pso"], c["n"] + 1, c["obj"],
                    1e-8, s["seed"], per_run=True)
        return {"idx": r.idx, "status": r.status, "fval": r.fval, "gnorm": r.gradientNorm,
                "x": r.coordinates, "iter": r.iter, "actual": r.c.actual,
                "claimed": r.c.claimed, "surrendered": r.c.surrendered,
                "per_run_fval": r.per_run_fval, "per_run_status": r.per_run_status}
    if what == "starts":
        return zb.starts(s["seed"], c["n"], c["dim"], -5.0, 5.0, prng=c["prng"])
    if what == "pso":
        lo, hi = BOUNDS[c["obj"]]
        x, f, g = zb.pso_device(s["problem"], s["seed"], c["n"], lo, hi, c["iters"],
                                prng=c["prng"])
        return {"pbest_x": x, "pbest_f": f, "gbest": g}
    if what == "bfgs":
        return _runs(zb.bfgs_device(s["problem"], s["x0"], max_iter=c["max_iter"],
                                    gradient=c["gradient"]))
    if what == "exact":
        r = zb.bfgs_device(s["problem"], s["x0"], max_iter=c["max_iter"], mode="exact",
                           gradient="dual", traj=True)
        return {"runs": _runs(r), "traj": r.traj}
    b = s["batch"].launch()
    out = {"%d" % i: _runs(j) for i, j in enumerate(b.jobs)}
    if what == "dijet":
        out["best"], out["sens"] = zd.nll_sensitivity(b.jobs[0])
    return out


# ---------------------------------------------------------------- work
# Mean iterations and function evaluations of a run from uniform starts,
# as the counters of bfgs_device report them (10000-iteration limit).
MEAN = {"rosenbrock": {2: (870, 17700), 4: (360, 6700), 8: (175, 2300), 10: (163, 1850),
                       16: (140, 720), 32: (205, 690), 64: (315, 900), 128: (514, 1620)},
        "rastrigin": {2: (26, 400), 10: (31, 264), 16: (36, 229)},
        "ackley": {2: (264, 5380), 10: (20, 58), 30: (20, 56)},
        "gaussian": {2: (4, 7), 8: (5, 11), 32: (4, 16), 150: (10, 24)}}
FN = 20  # flops counted for a transcendental function


def _eval_flops(obj, d):
    """One f(x + a p)."""
    return {"rosenbrock": 10 * d, "rastrigin": (FN + 6) * d, "ackley": (FN + 5) * d + 3 * FN,
            "gaussian": 2 * d * d + 4 * d}[obj]


def _run_flops(obj, d, max_iter=10000, gradient="adjoint"):
    it, ev = MEAN[obj][d]
    cut = min(1.0, max_iter / 10000) if it > 100 else 1.0
    grad = _eval_flops(obj, d) * (1.5 if gradient == "adjoint" else 3 * d)
    return cut * (it * (6 * d * d + 15 * d + grad) + ev * _eval_flops(obj, d))


def _run_bytes(n, d):
    """Starts read; fval, status, iter, gnorm, x and counters written."""
    return n * (16 * d + 48)


def work(case):
    what = case["what"]
    if what == "mixed":
        n = case["per_class"]
        return {"bytes": sum(_run_bytes(n, d) for _, d, _, _ in MIXED),
                "flops": n * sum(_run_flops(o, d) for o, d, _, _ in MIXED)}
    if what == "dijet":
        n, toys = case["toys"] * RUNS_PER_TOY, case["toys"]
        it, ev = 400, 3050
        return {"bytes": _run_bytes(n, 4) + toys * (NBINS * (12 + 32) + 48),
                "flops": n * NBINS * (ev * (FN + 10) + it * (FN + 18))
                + toys * NBINS * (3 * FN + 60)}
    d, n = case["dim"], case["n"]
    if what == "starts":
        return {"bytes": 8 * n * d, "flops": 2 * n * d}
    f = _eval_flops(case["obj"], d)
    if what == "pso":
        # the swarm's own state stays on the chip; bests come out
        return {"bytes": 8 * (n * (d + 1) + d + 1), "flops": n * (case["iters"] + 1) * (f + 9 * d)}
    if what == "call":
        swarm = n * (max(case["pso"], -1) + 1) * (f + 9 * d)
        return {"bytes": 12 * n + 8 * d, "flops": n * _run_flops(case["obj"], d) + swarm}
    if what == "exact":
        t, (it, ev) = case["max_iter"], MEAN[case["obj"]][d]
        it, ev = min(it, 0.4 * t), min(ev, 4 * t)
        # recorded: x, f and |g| and a status byte for each iterate
        return {"bytes": _run_bytes(n, d) + n * t * (8 * d + 17),
                "flops": n * (it * (4 * d ** 3 + 4 * d * d + 3 * d * f) + ev * f)}
    return {"bytes": _run_bytes(n, d),
            "flops": n * _run_flops(case["obj"], d, case["max_iter"], case["gradient"])}


# ---------------------------------------------------------------- exact values
def _philox(c0, c1, c2, c3, seed):
    """Philox4x32-10 (Salmon et al., SC'11) on arrays of counter words."""
    m32 = np.uint64(0xFFFFFFFF)
    c = [np.asarray(v, np.uint64) for v in np.broadcast_arrays(c0, c1, c2, c3)]
    k0, k1 = seed & 0xFFFFFFFF, (seed >> 32) & 0xFFFFFFFF
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        s32 = np.uint64(32)
        c = [(p1 >> s32) ^ c[1] ^ np.uint64(k0), p1 & m32, (p0 >> s32) ^ c[3] ^ np.uint64(k1),
             p0 & m32]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def _pairs(seed, tag, n, blocks):
    """(n, blocks, 2) uniforms in [0, 1): one Philox block holds two."""
    o = _philox(np.arange(n)[:, None], np.arange(blocks)[None, :], tag, 0, seed)
    u = [((o[2 * i] << np.uint64(32)) | o[2 * i + 1]) >> np.uint64(11) for i in (0, 1)]
    return np.stack(u, -1).astype(np.float64) * 2.0 ** -53


def _uniforms(seed, tag, n, dim):
    return _pairs(seed, tag, n, (dim + 1) // 2).reshape(n, -1)[:, :dim]


def _value(obj, x):
    d = x.shape[1]
    if obj == "rosenbrock":
        return ((1 - x[:, :-1]) ** 2 + 100 * (x[:, 1:] - x[:, :-1] ** 2) ** 2).sum(1)
    if obj == "rastrigin":
        return 10.0 * d + (x * x - 10 * np.cos(2 * np.pi * x)).sum(1)
    if obj == "ackley":
        return (-20 * np.exp(-0.2 * np.sqrt((x * x).sum(1) / d))
                - np.exp(np.cos(2 * np.pi * x).sum(1) / d) + 20 + np.e)
    return 0.5 * ((x @ zb.gaussian_matrix(d)) * x).sum(1)


def exact(case, seed):
    what, seed = case["what"], 42 + 7919 * seed
    # the iterates of an optimiser are what its own rounding makes them, and
    # the Sobol' directions are this package's own
    if what not in ("starts", "pso") or case["prng"] != "philox":
        return None
    n, d = case["n"], case["dim"]
    if what == "starts":
        return -5.0 + 10.0 * _uniforms(seed, 1, n, d)
    lo, hi = BOUNDS[case["obj"]]
    x = lo + (hi - lo) * _uniforms(seed, 2, n, d)
    vr = 0.1 * (hi - lo)
    v = -vr + 2 * vr * _uniforms(seed, 3, n, d)
    f = _value(case["obj"], x)
    px, pf = x.copy(), f.copy()
    i = int(np.argmin(f))
    gf, gx = f[i], x[i].copy()
    for t in range(1, case["iters"] + 1):
        r = _pairs(seed, 16 + t, n, d)
        v = 0.5 * v + 1.2 * r[:, :, 0] * (px - x) + 1.5 * r[:, :, 1] * (gx - x)
        x = x + v
        f = _value(case["obj"], x)
        better = f < pf
        pf[better], px[better] = f[better], x[better]
        i = int(np.argmin(f))
        if f[i] < gf:
            gf, gx = f[i], x[i].copy()
    return {"pbest_x": px, "pbest_f": pf, "gbest": np.concatenate([[gf], gx])}
