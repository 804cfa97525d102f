"""The work this library is timed on: Hausdorff solves through its public
Python API (Engine.solve, Engine.solve_f64, Engine.solve_batch and the
variant classes), from sets of two thousand points, where a call is all
latency, to LiDAR scans of fifty million.

The sets are the benchmark's distributions (hausdorffdistance_gb300/synth.py:
uniform2d, clusters3d, planes3d, unit64, polylines) drawn on the GPU from a
seed.  A program keeps one Engine and gives it one pair of sets after another,
so one Engine serves every case here too.

A case names a distribution ("data"), the sizes, the entry point ("call") and
its options:
  call      solve     Engine.solve, the selector's choice of algorithm
            solve_f64 Engine.solve_f64 on float64 sets
            batch     Engine.solve_batch, n_a problems
            eb        HausdorffDistanceEarlyBreak.CalculateDistance
  undirected  max(h(A,B), h(B,A)) in one call, else h(A,B)
  host      the sets are pinned host arrays, copied inside the call
"""
import math

import numpy as np
import torch

import hausdorffdistance_gb300 as hd

_KEPT = {}


def _kept(name, make):
    if name not in _KEPT:
        _KEPT[name] = make()
    return _KEPT[name]


def _case(call, data, dims, n_a, n_b, undirected, host=False, **name):
    return dict(name, call=call, data=data, dims=dims, n_a=n_a, n_b=n_b, undirected=undirected,
                host=host)


def listed():
    return [
        # Two contours or outlines of an interactive program: all latency.
        _case("solve", "uniform2d", 2, 2000, 2000, True, name="contours2d_2k"),
        # Two decimated CAD meshes' vertices, handed over as host arrays.
        _case("solve", "clusters3d", 3, 20011, 17989, False, host=True, name="mesh3d_20k_host"),
        # The benchmark's 2-D workload: map points against their noisy copy.
        _case("solve", "uniform2d", 2, 200000, 200000, True, name="uniform2d_200k"),
        # One scan against a reference model, ragged sizes, one direction.
        _case("solve", "clusters3d", 3, 1000003, 700001, False, name="clusters3d_1m_directed"),
        # The benchmark's headline workload.
        _case("solve", "clusters3d", 3, 10000000, 10000000, True, name="clusters3d_10m"),
        # The same from pinned host memory, as a program that reads its sets
        # from files calls it (the benchmark's end-to-end figure).
        _case("solve", "clusters3d", 3, 10000000, 10000000, True, host=True,
              name="clusters3d_10m_host"),
        # The benchmark's largest workload: two LiDAR scans.
        _case("solve", "planes3d", 3, 50000000, 50000000, True, name="planes3d_50m"),
        # Double coordinates, exact in FP64 (the benchmark's FP64 workload).
        _case("solve_f64", "clusters3d", 3, 10000000, 10000000, True, name="clusters3d_10m_f64"),
        # Embedding vectors: the benchmark's 64-D workload.
        _case("solve", "unit", 64, 1000000, 1000000, True, name="unit64_1m"),
        # Feature vectors whose length no tensor-core tile fits.
        _case("solve", "unit", 10, 60000, 50000, False, name="unit10_60k"),
        # Many small problems in one call: the benchmark's polyline workload.
        _case("batch", "polylines", 2, 100000, 100000, True, name="polylines_100k"),
        # The plain early-break algorithm, asked for by its class.
        _case("eb", "clusters3d", 3, 1000000, 1000000, False, name="early_break3d_1m"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _pair(rng, lo, hi):
    """Two set sizes of [lo, hi], within a factor of two of each other."""
    n = _log(rng, lo, hi)
    return n, min(hi, max(lo, int(n * math.exp(rng.uniform(-0.7, 0.7)))))


def draw(rng):
    kind = rng.choice(["uniform2d", "uniform2d", "clusters3d", "clusters3d", "clusters3d",
                       "planes3d", "f64", "unit", "nd", "batch", "eb"])
    undirected = rng.random() < 0.7
    host = rng.random() < 0.25
    if kind == "uniform2d":
        return _case("solve", "uniform2d", 2, *_pair(rng, 1000, 4000000), undirected, host=host)
    if kind == "clusters3d":
        return _case("solve", "clusters3d", 3, *_pair(rng, 1000, 10000000), undirected, host=host)
    if kind == "planes3d":
        return _case("solve", "planes3d", 3, *_pair(rng, 100000, 50000000), undirected)
    if kind == "f64":
        data, dims = rng.choice([("uniform2d", 2), ("clusters3d", 3)])
        return _case("solve_f64", data, dims, *_pair(rng, 2000, 10000000), undirected, host=host)
    if kind == "unit":
        return _case("solve", "unit", rng.choice([16, 32, 48, 64]), *_pair(rng, 10000, 1000000),
                     undirected)
    if kind == "nd":
        return _case("solve", "unit", rng.choice([4, 6, 10, 24, 40]), *_pair(rng, 2000, 60000),
                     undirected)
    if kind == "batch":
        n = _log(rng, 200, 100000)
        return _case("batch", "polylines", rng.choice([2, 2, 3]), n, n, undirected, host=host)
    return _case("eb", rng.choice(["uniform2d", "clusters3d"]), 0, *_pair(rng, 2000, 1000000),
                 undirected)


# ---------------------------------------------------------------------------
# Inputs (the distributions of synth.py, drawn on the GPU)

def _uniform2d(g, n_a, n_b, t):
    """A uniform in the unit square; B points of A jittered by N(0, 1e-3), 5 %
    of them replaced by outliers of [0, 1.2]^2."""
    a = torch.rand(n_a, 2, generator=g, device="cuda", dtype=t)
    b = (a[torch.randint(n_a, (n_b,), generator=g, device="cuda")] if n_a != n_b
         else a[torch.randperm(n_a, generator=g, device="cuda")])
    b = b + 1e-3 * torch.randn(n_b, 2, generator=g, device="cuda", dtype=t)
    k = n_b // 20
    b[torch.randperm(n_b, generator=g, device="cuda")[:k]] = 1.2 * torch.rand(
        k, 2, generator=g, device="cuda", dtype=t)
    return a, b


def _clusters3d(g, n_a, n_b, t):
    """A mixture of 64 Gaussians of sigma 0.01 in the unit cube; B drawn from
    the same mixture shifted by 0.05 along x."""
    c = torch.rand(64, 3, generator=g, device="cuda", dtype=t)

    def some(n):
        k = torch.randint(64, (n,), generator=g, device="cuda")
        return c[k] + 0.01 * torch.randn(n, 3, generator=g, device="cuda", dtype=t)

    a, b = some(n_a), some(n_b)
    b[:, 0] += 0.05
    return a, b


def _planes3d(g, n_a, n_b, t):
    """500 planar patches of 10 x 10 in a 100^3 cube with noise 0.02 along the
    normal; B such points turned by one degree about z, 0.1 % of them replaced
    by points of the whole cube."""
    c = 100 * torch.rand(500, 3, generator=g, device="cuda", dtype=t)
    w, u = torch.nn.functional.normalize(
        torch.randn(2, 500, 3, generator=g, device="cuda", dtype=t), dim=2)
    u = torch.nn.functional.normalize(torch.linalg.cross(w, u))  # in the plane
    v = torch.linalg.cross(w, u)

    def some(n):
        p = torch.empty(n, 3, device="cuda", dtype=t)
        for s in range(0, n, 10000000):
            m = min(10000000, n - s)
            k = torch.randint(500, (m,), generator=g, device="cuda")
            x = 10 * torch.rand(m, 2, generator=g, device="cuda", dtype=t) - 5
            h = 0.02 * torch.randn(m, 1, generator=g, device="cuda", dtype=t)
            p[s:s + m] = c[k] + x[:, :1] * u[k] + x[:, 1:] * v[k] + h * w[k]
        return p

    a = some(n_a)
    b = a.clone() if n_a == n_b else some(n_b)
    mid = a[:1000000].mean(0)
    th = math.radians(1.0)
    x, y = b[:, 0] - mid[0], b[:, 1] - mid[1]
    b[:, 0], b[:, 1] = (math.cos(th) * x - math.sin(th) * y + mid[0],
                        math.sin(th) * x + math.cos(th) * y + mid[1])
    k = n_b // 1000
    b[torch.randint(n_b, (k,), generator=g, device="cuda")] = 100 * torch.rand(
        k, 3, generator=g, device="cuda", dtype=t)
    return a, b


def _unit(g, n_a, n_b, dims):
    """Rows of unit length; B rows of A, 1 % of them replaced by fresh ones."""
    def some(n):
        return torch.nn.functional.normalize(torch.randn(n, dims, generator=g, device="cuda"))

    a = some(n_a)
    b = a.clone() if n_a == n_b else a[torch.randint(n_a, (n_b,), generator=g, device="cuda")]
    k = max(1, n_b // 100)
    b[torch.randint(n_b, (k,), generator=g, device="cuda")] = some(k)
    return a, b


def _polylines(g, n, dims):
    """n random walks (steps of 0.01, lengths lognormal around 200, 8 to
    50,000 vertices) and the same walks' vertices re-noised by 0.002."""
    z = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    sizes = (200 * torch.exp(1.2 * z)).round().clamp(8, 50000).long()
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    off[1:] = sizes.cumsum(0)
    total = int(off[-1])
    step = 0.01 * torch.randn(total, dims, generator=g, device="cuda", dtype=torch.float64)
    step[off[:-1]] = 0.0
    walk = step.cumsum(0)
    start = 100 * torch.rand(n, dims, generator=g, device="cuda", dtype=torch.float64)
    owner = torch.repeat_interleave(torch.arange(n, device="cuda"), sizes)
    a = walk + (start - walk[off[:-1]])[owner]
    b = a + 0.002 * torch.randn(total, dims, generator=g, device="cuda", dtype=torch.float64)
    return a.float(), b.float(), off.cpu().numpy()


def _inputs(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    if case["data"] == "polylines":
        return _polylines(g, case["n_a"], case["dims"])
    if case["data"] == "unit":
        a, b = _unit(g, case["n_a"], case["n_b"], case["dims"])
    else:
        make = {"uniform2d": _uniform2d, "clusters3d": _clusters3d, "planes3d": _planes3d}
        t = torch.float64 if case["call"] == "solve_f64" else torch.float32
        a, b = make[case["data"]](g, case["n_a"], case["n_b"], t)
    return a.contiguous(), b.contiguous(), None


def prepare(case, seed):
    a, b, off = _inputs(case, seed)
    if case["host"]:
        a, b = (x.cpu().pin_memory().numpy() for x in (a, b))
    torch.cuda.synchronize()
    if case["call"] == "eb":
        handle = _kept("eb", hd.HausdorffDistanceEarlyBreak)
    else:
        handle = _kept("engine", hd.Engine)
    return {"call": case["call"], "undirected": case["undirected"], "handle": handle, "a": a,
            "b": b, "off": off}


# ---------------------------------------------------------------------------
# One pass

def run(state):
    h, a, b = state["handle"], state["a"], state["b"]
    if state["call"] == "batch":
        r = h.solve_batch(a, b, state["off"], state["off"], undirected=state["undirected"])
        return {k: r[k] for k in ("hd_f32", "ia", "ib", "direction")}
    if state["call"] == "eb":
        d = h.CalculateDistance(a, b, undirected=state["undirected"])
        s = h.get_stats()
        return {"hd_f32": d, "hd": s["HD64"], "ia": s["CertifyingPair"][0],
                "ib": s["CertifyingPair"][1], "direction": s["Direction"]}
    solve = h.solve_f64 if state["call"] == "solve_f64" else h.solve
    r = solve(a, b, undirected=state["undirected"])
    return {"hd": r.hd, "hd_f32": np.float32(r.hd_f32), "hd_ab": r.hd_ab, "hd_ba": r.hd_ba,
            "ia": r.ia, "ib": r.ib, "direction": r.direction}


def work(case):
    """Every coordinate is read once; every query point needs one distance at
    least.  How many more it needs depends on the data and the algorithm."""
    if case["call"] == "batch":
        mean = 200 * math.exp(0.5 * 1.2 ** 2)  # of the lognormal; the clipping changes little
        points, size, out = 2 * case["n_a"] * mean, 4, 16 * case["n_a"]
    else:
        points, size, out = case["n_a"] + case["n_b"], 8 if case["call"] == "solve_f64" else 4, 64
    dims = case["dims"] or (2 if case["data"] == "uniform2d" else 3)
    queries = points if case["undirected"] else points / 2
    return {"bytes": points * dims * size + out, "flops": queries * (3 * dims - 1)}


# ---------------------------------------------------------------------------
# The same in 64 bits

def _max_min(a, b, undirected):
    """(h(A,B)^2, h(B,A)^2 or -1) by all pairs in float64."""
    ab = torch.zeros((), device="cuda", dtype=torch.float64)
    col = torch.full((b.shape[0],), math.inf, device="cuda", dtype=torch.float64)
    chunk = max(1, int(2e8) // b.shape[0])
    for s in range(0, a.shape[0], chunk):
        x = a[s:s + chunk]
        d2 = (x[:, :1] - b[:, 0]).square_()
        for k in range(1, a.shape[1]):
            d2 += (x[:, k:k + 1] - b[:, k]).square_()
        ab = torch.maximum(ab, d2.amin(1).amax())
        if undirected:
            torch.minimum(col, d2.amin(0), out=col)
    return ab, (col.amax() if undirected else ab - ab - 1)


def exact(case, seed):
    if case["call"] == "batch":
        if case["n_a"] > 20000:
            return None
    elif case["n_a"] * case["n_b"] * (case["dims"] or 3) > 1e11:
        return None
    a, b, off = _inputs(case, seed)
    a, b = a.double(), b.double()
    if case["call"] == "batch":
        h = torch.stack([torch.maximum(*_max_min(a[s:e], b[s:e], case["undirected"]))
                         for s, e in zip(off[:-1].tolist(), off[1:].tolist())])
        return {"hd_f32": h.sqrt(), "ia": None, "ib": None, "direction": None}
    ab, ba = (float(x) for x in _max_min(a, b, case["undirected"]))
    h = math.sqrt(max(ab, ba))
    out = {"hd": h, "hd_f32": h, "ia": None, "ib": None, "direction": None}
    if case["call"] != "eb":
        out["hd_ab"] = math.sqrt(ab)
        out["hd_ba"] = math.sqrt(ba) if case["undirected"] else -1.0
    return out
