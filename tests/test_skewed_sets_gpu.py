"""Sets of very different sizes: the cell filter stays out where hardly a cell of the
queries can be near one of the few targets, and out of scans that are over before
it; values and pairs are the oracle's."""
import numpy as np
import pytest

import hd_oracle

pytestmark = pytest.mark.gpu


def launches(engine, a, b, **kw):
    n = engine.kernel_launches
    r = engine.solve(a, b, **kw)
    return r, engine.kernel_launches - n


@pytest.mark.parametrize("d", [2, 3])
@pytest.mark.parametrize("na,nb", [(300_000, 2000), (300_000, 2400), (60_000, 20), (1, 100_000),
                                   (100_000, 1), (7999, 200_000), (200_000, 7999), (20, 60_000)])
def test_skewed(na, nb, d):
    import hausdorffdistance_gb300 as hd
    rng = np.random.default_rng(d + nb)
    a, b = rng.random((na, d)).astype(np.float32), rng.random((nb, d)).astype(np.float32)
    with hd.Engine() as engine, hd.Engine(lbvh_budget=257) as index:  # the table's and a visit
        for undirected in (False, True):
            want = hd_oracle.hd_f32(a, b, undirected=undirected)
            for variant in ("auto", "lbvh", "eb"):
                r, n = launches(engine, a, b, undirected=undirected, variant=variant)
                assert np.float32(r.hd_f32) == want["hd_f32"], (variant, undirected)
                src, dst = (a, b) if r.direction == 0 else (b, a)
                assert hd_oracle.dist2_f32(src[int(r.ia)], dst[int(r.ib)]) == want["d2"]
                if variant == "lbvh" and not undirected and na > 128 * nb + 127:
                    assert n == launches(index, a, b, variant=variant)[1]
                if variant == "eb" and min(na, nb) < 8000:  # pack, seeds, scan, certification
                    assert n <= 9 * (1 + undirected)
        r = engine.solve_f64(a.astype(np.float64), b.astype(np.float64))
        assert r.hd == np.sqrt(hd_oracle.exact_f64(a.astype(np.float64), b.astype(np.float64))[0])
