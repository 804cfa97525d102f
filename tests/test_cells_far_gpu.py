"""Cell filter, queries far from the target's box or from anything in it: sets apart
along each axis, one around the other, targets in opposite corners, single
outliers.  Values and pairs are the oracle's, and a call costs no multiple of the
index alone (which lbvh_budget, set by the caller, asks for)."""
import time

import numpy as np
import pytest

import hd_oracle

pytestmark = pytest.mark.gpu


def corners(x):
    x = 0.02 * x
    x[::2] += 0.98
    return x


KINDS = {
    "apart_up": lambda a, b, k: (a, b + 3.0 * np.eye(b.shape[1])[k]),
    "apart_down": lambda a, b, k: (a, b - 3.0 * np.eye(b.shape[1])[k]),
    "apart_all": lambda a, b, k: (a, b + (3.0, -3.0, 0.7)[k]),
    "small_target_beside": lambda a, b, k: (a, 0.1 * b + 0.45 + 2.0 * np.eye(b.shape[1])[k]),
    "small_target_inside": lambda a, b, k: (a, 0.01 * b + (0.1, 0.5, 0.95)[k]),
    "corners": lambda a, b, k: (a if k else 0.3 * a, corners(b)),
    "around": lambda a, b, k: (a + np.where(a > 0.5, 1.0, -1.0), (1.0, 0.5, 0.01)[k] * b),
    "outliers": lambda a, b, k: (np.where(np.arange(len(a))[:, None] % 97 == 5, a + 3.0 * (k + 1), a), b),
}


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("d", [2, 3])
@pytest.mark.parametrize("k", [0, 1, 2])
def test_far_queries(engine, kind, d, k):
    if k >= d:
        k = 0
    rng = np.random.default_rng(d * 10 + k)
    a, b = KINDS[kind](rng.random((30_011, d)), rng.random((28_007, d)), k)
    f = [np.ascontiguousarray(x, np.float32) for x in (a, b)]
    for x, y in (f, f[::-1]):
        for undirected, variant in ((False, "lbvh"), (True, "lbvh"), (False, "eb")):
            r = engine.solve(x, y, undirected=undirected, variant=variant)
            want = hd_oracle.hd_f32(x, y, undirected=undirected)
            assert np.float32(r.hd_f32) == want["hd_f32"], (undirected, variant)
            src, dst = (x, y) if r.direction == 0 else (y, x)
            assert hd_oracle.dist2_f32(src[int(r.ia)], dst[int(r.ib)]) == want["d2"]
    r = engine.solve_f64(a, b, undirected=True)
    ab, ba = hd_oracle.exact_f64(a, b), hd_oracle.exact_f64(b, a)
    assert (r.hd_ab, r.hd_ba) == (np.sqrt(ab[0]), np.sqrt(ba[0]))
    win = ba if ba[0] > ab[0] else ab
    assert (int(r.ia), int(r.ib)) == (win[1], win[2])


@pytest.mark.parametrize("kind", ["apart_all", "small_target_beside", "corners", "outliers"])
@pytest.mark.parametrize("d", [2, 3])
def test_far_queries_cost_no_multiple(kind, d):
    import torch
    import hausdorffdistance_gb300 as hd
    rng = np.random.default_rng(d)
    a, b = KINDS[kind](rng.random((1_000_003, d)), rng.random((1_000_000, d)), 0)
    sets = [torch.from_numpy(np.ascontiguousarray(x, np.float32)).cuda() for x in (a, b)]
    best = []
    # Both walk with the same budget; the caller's is not the table's by one visit.
    for budget in (0, 257):
        with hd.Engine(lbvh_budget=budget) as engine:
            ts = []
            for _ in range(8):
                torch.cuda.synchronize()
                t = time.perf_counter()
                r = engine.solve(*sets, undirected=True, variant="lbvh")
                ts.append(time.perf_counter() - t)
            best.append((min(ts), r.hd_ab, r.hd_ba))
    assert best[0][1:] == best[1][1:]
    assert best[0][0] < 4 * best[1][0]


def test_finer_grid_for_the_second_direction():
    """The sets' boxes lie in the call's order, also when the direction that is
    tried again is its second."""
    import torch
    import hausdorffdistance_gb300 as hd
    from hausdorffdistance_gb300 import synth
    a, b = synth.planes3d(22_000_003, seed=78)
    sets = [torch.from_numpy(x).cuda() for x in (b[:21_000_001], a)]
    got = []
    for budget in (0, 257):
        with hd.Engine(lbvh_budget=budget) as engine:
            r = engine.solve(*sets, undirected=True, variant="lbvh")
            got.append((r.hd_ab, r.hd_ba, r.hd_f32, r.direction, r.ia, r.ib))
    assert got[0] == got[1]
