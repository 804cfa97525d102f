"""Batches of a few long problems: each direction gets an SM of its own, whichever
SM asks first."""
import time

import numpy as np
import pytest

import hd_oracle

pytestmark = pytest.mark.gpu


def batch(rng, sizes, d):
    total = sum(sizes)
    a, b = (rng.random((total, d)).astype(np.float32) for _ in range(2))
    return a, b, np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)


def seconds(engine, a, b, off):
    import torch
    ts = []
    for _ in range(6):
        torch.cuda.synchronize()
        t = time.perf_counter()
        engine.solve_batch(a, b, off, off, undirected=True)
        ts.append(time.perf_counter() - t)
    return min(ts[2:])


@pytest.mark.parametrize("rows,many", [(4096, 60), (5000, 60)])  # a warp, a block per direction
def test_long_problems_run_side_by_side(rows, many):
    import torch
    import hausdorffdistance_gb300 as hd
    rng = np.random.default_rng(rows)
    with hd.Engine() as engine:
        a, b, off = batch(rng, [rows] * many, 3)
        ta, tb = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
        one = max(seconds(engine, ta[s:s + rows].contiguous(), tb[s:s + rows].contiguous(), off[:2])
                  for s in off[:6])
        assert seconds(engine, ta, tb, off) < 1.7 * one


@pytest.mark.parametrize("sizes", [[4096] * 3, [4097] * 2 + [30] * 40, [9] * 700, [70_000, 4097, 4096, 1],
                                   [300] * 2000])
def test_queue_places(engine, sizes):
    rng = np.random.default_rng(len(sizes))
    a, b, off = batch(rng, sizes, 2)
    for undirected in (False, True):
        out = engine.solve_batch(a, b, off, off, undirected=undirected)
        for p in range(0, len(sizes), max(1, len(sizes) // 50)):
            x, y = a[off[p]:off[p + 1]], b[off[p]:off[p + 1]]
            want = hd_oracle.hd_f32(x, y, undirected=undirected)
            assert out["hd_f32"][p] == want["hd_f32"], (p, undirected)
            src, dst = (x, y) if out["direction"][p] == 0 else (y, x)
            assert hd_oracle.dist2_f32(src[out["ia"][p]], dst[out["ib"][p]]) == want["d2"]
