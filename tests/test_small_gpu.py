"""Small sets solved in one kernel (hd_small.cu): the sizes at its edges (query
tiles of 256 and 512, target chunks of 32 to 256, odd counts, the largest sets
and pair counts it takes and the first it leaves), against the oracle, one
after the other through the same context, whose minima each solve has to leave
as it found them."""
import numpy as np
import pytest

import hd_oracle

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (1, 2), (2, 1), (3, 255), (255, 257), (256, 256), (257, 31), (511, 513),
         (1, 32768), (32768, 1), (32768, 4882), (4883, 32768), (32769, 100), (8191, 8193),
         (8192, 8192), (12_649, 12_649), (12_651, 12_649)]


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("undirected", [False, True])
def test_sizes(engine, dims, undirected):
    rng = np.random.default_rng(dims)
    for i, (na, nb) in enumerate(SIZES):
        a = rng.random((na, dims)).astype(np.float32)
        b = (rng.random((nb, dims)) * 1.1).astype(np.float32)
        if i % 3 == 2:
            b = np.round(b * 8) / 8  # ties
        want = hd_oracle.hd_f32(a, b, undirected=undirected)
        for variant in ("eb", "auto"):
            r = engine.solve(a, b, undirected=undirected, variant=variant, count_pairs=True)
            assert np.float32(r.hd_f32) == want["hd_f32"], (na, nb, variant)
            src, dst = (a, b) if r.direction == 0 else (b, a)
            assert hd_oracle.dist2_f32(src[int(r.ia)], dst[int(r.ib)]) == want["d2"]
            assert r.visited_pairs > 0


def test_ready_again_after_an_error(engine):
    import hausdorffdistance_gb300 as hd
    rng = np.random.default_rng(9)
    a, b = rng.random((700, 3)).astype(np.float32), rng.random((900, 3)).astype(np.float32)
    bad = a.copy()
    bad[5] = np.nan  # a row without a nearest neighbour
    want = hd_oracle.hd_f32(a, b)["hd_f32"]
    assert np.float32(engine.solve(a, b).hd_f32) == want
    with pytest.raises(hd.HDError):
        engine.solve(bad, b)
    assert np.float32(engine.solve(a, b).hd_f32) == want
