"""Early-break scans that start at the cell filter's bound: where that bound is
poor (L a cell or two; targets so far that the seeds stop short) the scan takes
seed rows of its own, so that it visits no more pairs than the plain scan
(hd_solve_eb_noalloc) by more than the few that vary from run to run."""
import ctypes

import numpy as np
import pytest

import hd_oracle
from hausdorffdistance_gb300 import synth

pytestmark = pytest.mark.gpu


def corners(n, seed):
    rng = np.random.default_rng(seed)
    a, b = rng.random((n, 3)), 0.02 * rng.random((n, 3))
    b[::2] += 0.98
    return a.astype(np.float32), b.astype(np.float32)


@pytest.mark.parametrize("make,n,most", [
    (synth.planes3d, 300_000, 1.04), (synth.planes3d, 1_000_000, 1.04), (corners, 100_000, 1.04),
    (synth.clusters3d, 300_000, 0.8)])  # near the maximum from the start
def test_pairs_against_the_plain_scan(engine, make, n, most):
    import torch
    from hausdorffdistance_gb300 import _lib
    a, b = make(n, seed=5)
    ta, tb = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    plain = _lib.Result()
    st = _lib.load().hd_solve_eb_noalloc(ta.data_ptr(), n, tb.data_ptr(), n, 3,
                                         _lib.HD_DEVICE_PTRS, None, ctypes.byref(plain))
    assert st == 0
    for _ in range(3):  # the third replays a graph
        r = engine.solve(ta, tb, variant="eb", count_pairs=True)
        assert (r.hd, r.hd_f32, r.ia) == (plain.hd, plain.hd_f32, plain.ia)
        assert r.visited_pairs <= most * plain.visited_pairs


def test_bound_in_a_query_set_of_fewer_points_than_seeds(engine):
    rng = np.random.default_rng(6)
    for n in (1, 7, 151, 152, 153, 256, 257):
        a = rng.random((n, 3)).astype(np.float32)
        b = np.concatenate([a + np.float32(1e-6), rng.random((50_000, 3)).astype(np.float32)])
        for undirected in (False, True):
            want = hd_oracle.hd_f32(a, b, undirected=undirected)
            for _ in range(2):
                r = engine.solve(a, b, variant="eb", undirected=undirected)
                assert np.float32(r.hd_f32) == want["hd_f32"], (n, undirected)
                src, dst = (a, b) if r.direction == 0 else (b, a)
                assert hd_oracle.dist2_f32(src[int(r.ia)], dst[int(r.ib)]) == want["d2"]
