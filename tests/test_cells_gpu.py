"""The cell filter before the indexes (hd_cells.cu): sets from 40,000 points
(|A| + |B|) of the shapes where a grid of cells can go wrong, against the oracle.
The filter decides how much of a set is searched, never what is found: value
and certifying distance are the oracle's bit for bit."""
import numpy as np
import pytest

import hd_oracle
from hausdorffdistance_gb300 import synth

pytestmark = pytest.mark.gpu


def uniform(rng, n, d):
    return rng.random((n, d))


def shapes(kind, d, rng):
    """(A, B) float64 arrays."""
    n, m = 30_011, 25_007
    a, b = uniform(rng, n, d), uniform(rng, m, d)
    if kind == "apart":  # disjoint: every query's nearest target is far away
        b = b * 0.1 + 3.0
    elif kind == "one_outlier":
        b = a[:m] + rng.normal(0, 1e-4, (m, d))
        a[17] = 5.0
    elif kind == "outliers_both_sides":
        a[:40] = rng.normal(0, 3, (40, d))
        b[:40] = rng.normal(0, 3, (40, d))
    elif kind == "flat":  # one axis without extent
        a[:, -1] = b[:, -1] = 0.25
    elif kind == "line":
        a = np.repeat(a[:, :1], d, 1)
        b = np.repeat(b[:, :1] * 1.1, d, 1)
    elif kind == "on_cell_borders":  # coordinates on multiples of the extent / 255
        a = rng.integers(0, 256, (n, d)).astype(np.float64)
        b = rng.integers(0, 200, (m, d)).astype(np.float64)
    elif kind == "lattice_and_translate":  # every row ties
        k = 200 if d == 2 else 34
        g = np.stack(np.meshgrid(*[np.arange(k)] * d, indexing="ij"), -1).reshape(-1, d)
        a, b = g * 1.0, g + 0.25
    elif kind == "duplicates":
        a = np.repeat(a[:300], 100, 0)
        b = np.repeat(b[:200], 120, 0)
    elif kind == "identical":
        b = a.copy()
    elif kind == "offset":  # float spacing of 1/16 in an extent of 100
        a, b = 1e6 + 100 * a, 1e6 + 110 * b
    elif kind == "huge":
        a, b = 1e14 * a, 1.1e14 * b
    elif kind == "beyond_the_grid":  # past the extents the grid takes
        a, b = 1e16 * a, 1.1e16 * b
    elif kind == "tiny":
        a, b = 1e-9 * a, 1.2e-9 * b
    elif kind == "below_the_grid":
        a, b = 1e-14 * a, 1.2e-14 * b
    elif kind == "one_target":
        b = b[:1]
        a = uniform(rng, 50_000, d)
    elif kind == "one_query":
        a = a[:1] + 0.3
        b = uniform(rng, 50_000, d)
    elif kind == "shells":  # dense surfaces: many open queries, wide target lists
        for x in (a, b):
            x -= 0.5
            x /= np.linalg.norm(x, axis=1, keepdims=True)
        b *= 1.05
    return a, b


KINDS = ["uniform", "apart", "one_outlier", "outliers_both_sides", "flat", "line", "on_cell_borders",
         "lattice_and_translate", "duplicates", "identical", "offset", "huge", "beyond_the_grid",
         "tiny", "below_the_grid", "one_target", "one_query", "shells"]


def check(a, b, r, undirected):
    want = hd_oracle.hd_f32(a, b, undirected=undirected)
    assert np.float32(r.hd_f32) == want["hd_f32"]
    src, dst = (a, b) if r.direction == 0 else (b, a)
    assert hd_oracle.dist2_f32(src[int(r.ia)], dst[int(r.ib)]) == want["d2"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("d", [2, 3])
def test_shapes(engine, kind, d):
    rng = np.random.default_rng(d * 100 + KINDS.index(kind))
    a, b = (np.ascontiguousarray(x, np.float32) for x in shapes(kind, d, rng))
    for undirected in (False, True):
        check(a, b, engine.solve(a, b, undirected=undirected, variant="lbvh"), undirected)
    check(b, a, engine.solve(b, a, variant="lbvh", count_pairs=True, timing=True), False)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("d", [2, 3])
def test_early_break_starts_from_the_cells(engine, kind, d):
    # The scan's running maximum starts at the filter's bound, which no row has;
    # the third identical solve replays a graph.
    rng = np.random.default_rng(d * 300 + KINDS.index(kind))
    a, b = (np.ascontiguousarray(x, np.float32) for x in shapes(kind, d, rng))
    for _ in range(3):
        check(a, b, engine.solve(a, b, undirected=True, variant="eb"), True)
    a, b = np.tile(a, (2, 1)), np.tile(b, (2, 1))
    check(a, b, engine.solve(a, b, variant="eb", count_pairs=True), False)


@pytest.mark.parametrize("kind", [k for k in KINDS if k not in ("huge", "beyond_the_grid")])
@pytest.mark.parametrize("d", [2, 3])
def test_shapes_f64(engine, kind, d):
    rng = np.random.default_rng(d * 200 + KINDS.index(kind))
    a, b = shapes(kind, d, rng)
    r = engine.solve_f64(a, b, undirected=True)
    ab, ba = hd_oracle.exact_f64(a, b), hd_oracle.exact_f64(b, a)
    assert r.hd_ab == np.sqrt(ab[0]) and r.hd_ba == np.sqrt(ba[0])
    win = ba if ba[0] > ab[0] else ab
    assert (int(r.ia), int(r.ib)) == (win[1], win[2])


@pytest.mark.parametrize("rows,cols", [(1, 1), (255, 64), (300, 20), (129, 127), (129, 128),
                                       (3000, 2)])
@pytest.mark.parametrize("d", [2, 3])
def test_f64_rows_that_floats_cannot_order(engine, d, rows, cols):
    # rows x cols pairs at the maximum to within float precision: finished pair
    # by pair up to 16,384 of them, by the index beyond; half are exact copies.
    rng = np.random.default_rng(d * 1000 + rows + cols)
    a, b = rng.random((30_011, d)), rng.random((25_007, d)) * 1.05
    a[rng.permutation(len(a))[:rows]] = 3.0 + 1e-10 * (np.arange(rows) // 2)[:, None]
    b[rng.permutation(len(b))[:cols]] = 1.2 + 1e-10 * (np.arange(cols) // 2)[:, None]
    for x, y in ((a, b), (b, a)):
        r = engine.solve_f64(x, y, undirected=x is a)
        want = [hd_oracle.exact_f64(x, y)] + ([hd_oracle.exact_f64(y, x)] if x is a else [])
        assert r.hd_ab == np.sqrt(want[0][0])
        win = max(want, key=lambda w: w[0])
        assert (r.hd, int(r.ia), int(r.ib)) == (np.sqrt(win[0]), win[1], win[2])


def test_nan_points_leave_their_direction_to_the_index(engine):
    # Targets with NaN coordinates are nobody's nearest neighbour, as before.
    rng = np.random.default_rng(4)
    a = rng.random((30_000, 3)).astype(np.float32)
    b = rng.random((30_000, 3)).astype(np.float32)
    bad = b.copy()
    bad[::1000, 1] = np.nan
    keep = ~np.isnan(bad).any(1)
    r = engine.solve(a, bad, variant="lbvh")
    assert np.float32(r.hd_f32) == hd_oracle.hd_f32(a, b[keep])["hd_f32"]


@pytest.mark.parametrize("maker,na,nb", [
    ("uniform2d", 900_001, 700_003),      # the finer 2-D grid
    ("clusters3d", 700_000, 500_001),     # occupied cells set in two launches
    ("planes3d", 22_000_003, 19_000_001)  # a direction that only the finest grid settles
])
def test_grids_by_size(engine, maker, na, nb):
    a, b = getattr(synth, maker)(max(na, nb), seed=77)
    a, b = a[:na], b[:nb]
    check(a, b, engine.solve(a, b, variant="lbvh"), False)
