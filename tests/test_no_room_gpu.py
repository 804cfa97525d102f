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
