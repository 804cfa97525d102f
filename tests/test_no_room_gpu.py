"""Solves that find no device memory for a buffer they can do without: the same
answers by the way that is left.  hd_debug_no_room refuses the growths; nothing is
exhausted on the device."""
import numpy as np
import pytest

import hd_oracle

pytestmark = pytest.mark.gpu

ALWAYS = 0xFFFFFFFF


def no_room(engine, buffer, times):
    from hausdorffdistance_gb300 import _lib
    assert engine.lib.hd_debug_no_room(engine._h, buffer, times) == 0


def sets(kind, d, n, m, seed):
    rng = np.random.default_rng(seed)
    a = rng.random((n, d))
    if kind == "copy":  # the filter gives both directions up
        b = a[rng.permutation(n)[:m]] + rng.normal(0, 1e-6, (m, d))
    else:               # it settles them
        b = rng.random((m, d)) * 1.2
    return np.ascontiguousarray(a, np.float32), np.ascontiguousarray(b, np.float32)


def check(a, b, r, undirected):
    want = hd_oracle.hd_f32(a, b, undirected=undirected)
    assert np.float32(r.hd_f32) == want["hd_f32"]
    src, dst = (a, b) if r.direction == 0 else (b, a)
    assert hd_oracle.dist2_f32(src[int(r.ia)], dst[int(r.ib)]) == want["d2"]


@pytest.mark.parametrize("kind", ["copy", "wider"])
@pytest.mark.parametrize("d", [2, 3])
@pytest.mark.parametrize("known", [False, True])
def test_no_room_for_the_filter(kind, d, known):
    """The index alone, behind the call's own copies and resets, on a context
    whose filter never ran and on one where it ran before (on smaller sets)."""
    import torch
    import hausdorffdistance_gb300 as hd
    from hausdorffdistance_gb300 import _lib
    with hd.Engine() as engine:
        if known:
            a, b = sets(kind, d, 30_000, 20_000, 1)
            check(a, b, engine.solve(a, b, variant="lbvh"), False)
        no_room(engine, _lib.DEBUG_FILTER, ALWAYS)
        a, b = sets(kind, d, 210_011, 190_007, 2)
        ta, tb = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
        for undirected in (False, True):
            for variant in ("lbvh", "auto"):
                r = engine.solve(a, b, undirected=undirected, variant=variant, count_pairs=True)
                check(a, b, r, undirected)
                if variant == "lbvh":  # the index found it
                    assert r.visited_nodes > 0
                check(a, b, engine.solve(ta, tb, undirected=undirected, variant=variant), undirected)
        check(a, b, engine.solve(a, b, variant="eb"), False)
        r = engine.solve_f64(a.astype(np.float64), b.astype(np.float64), undirected=True)
        assert r.hd_ab == np.sqrt(hd_oracle.exact_f64(a.astype(np.float64), b.astype(np.float64))[0])
        no_room(engine, _lib.DEBUG_FILTER, 0)
        check(a, b, engine.solve(a, b, undirected=True, variant="lbvh"), True)


def one_given_up_one_narrowed(rng, d, n=400_000, m=40_000):
    """A on a unit square of the plane; B its jittered copy and m points of a part
    of the square 0.1 above it, all equally far from A.  A -> B is too near for the
    cells; of B -> A every raised point stays open, too many for the pair scan."""
    a = np.zeros((n, 3))
    a[:, :2] = rng.random((n, 2))
    b = a + rng.normal(0, 1e-6, (n, 3))
    up = np.full((m, 3), 0.1)
    up[:, :2] = 0.45 * rng.random((m, 2))
    b = np.concatenate([b, up])[rng.permutation(n + m)]
    return (a, b) if d == 0 else (b, a)


@pytest.mark.parametrize("d", [0, 1])
def test_no_room_for_the_index_beside_the_filter(d):
    """The given-up direction's index finds no room while the filter runs and is
    tried again once the filter's lists have been through the index."""
    import hausdorffdistance_gb300 as hd
    from hausdorffdistance_gb300 import _lib
    a, b = one_given_up_one_narrowed(np.random.default_rng(5), d)
    f = [np.ascontiguousarray(x, np.float32) for x in (a, b)]
    want = hd_oracle.exact(f[0], f[1]), hd_oracle.exact(f[1], f[0])
    want64 = hd_oracle.exact_f64(a, b), hd_oracle.exact_f64(b, a)
    for refused in (0, 1):
        for variant in ("lbvh", "auto"):
            with hd.Engine() as engine:
                no_room(engine, _lib.DEBUG_TREE, refused)
                for _ in range(2):
                    r = engine.solve(f[0], f[1], undirected=True, variant=variant)
                    win = r.direction
                    assert win == 1 - d
                    assert r.hd_ab == pytest.approx(np.sqrt(want[0][0]), rel=1e-6)
                    assert r.hd_ba == pytest.approx(np.sqrt(want[1][0]), rel=1e-6)
                    assert np.float32(r.hd_f32) == np.sqrt(np.float32(want[win][0]))
                    assert (int(r.ia), int(r.ib)) == want[win][1:]
        with hd.Engine() as engine:
            no_room(engine, _lib.DEBUG_TREE, refused)
            for _ in range(2):
                r = engine.solve_f64(a, b, undirected=True)
                assert (r.hd_ab, r.hd_ba) == tuple(np.sqrt(w[0]) for w in want64)
                assert (int(r.ia), int(r.ib)) == want64[r.direction][1:]


@pytest.mark.parametrize("undirected", [False, True])
def test_no_room_for_the_index_of_sets_given_up(undirected):
    import hausdorffdistance_gb300 as hd
    from hausdorffdistance_gb300 import _lib
    a, b = sets("copy", 3, 210_011, 210_011, 3)
    with hd.Engine() as engine:
        no_room(engine, _lib.DEBUG_TREE, 1)
        for _ in range(2):
            check(a, b, engine.solve(a, b, undirected=undirected, variant="lbvh"), undirected)
    with hd.Engine() as engine:  # no room afterwards either: an error, then an answer
        no_room(engine, _lib.DEBUG_TREE, 2)
        with pytest.raises(hd.HDError) as e:
            engine.solve(a, b, undirected=undirected, variant="lbvh")
        assert e.value.status == 2
        check(a, b, engine.solve(a, b, undirected=undirected, variant="lbvh"), undirected)


@pytest.mark.parametrize("refused", [1, 2])
@pytest.mark.parametrize("undirected", [False, True])
def test_no_room_for_the_tiles(refused, undirected):
    """AUTO scans where the packed sets don't fit; by name the variant says so."""
    import hausdorffdistance_gb300 as hd
    from hausdorffdistance_gb300 import _lib
    rng = np.random.default_rng(6)
    a = rng.random((2105, 16)).astype(np.float32)
    b = (rng.random((1999, 16)) * 1.05).astype(np.float32)
    with hd.Engine() as engine:
        no_room(engine, _lib.DEBUG_TILES, refused)
        for _ in range(2):
            check(a, b, engine.solve(a, b, undirected=undirected), undirected)
    with hd.Engine() as engine:
        no_room(engine, _lib.DEBUG_TILES, 1)
        with pytest.raises(hd.HDError) as e:
            engine.solve(a, b, undirected=undirected, variant="bf16")
        assert e.value.status == 2
        check(a, b, engine.solve(a, b, undirected=undirected, variant="bf16"), undirected)
