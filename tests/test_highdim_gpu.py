"""High-dimensional inputs: the FP32 scans (EB, brute) for any n_dims up to
128 and the split-BF16 tcgen05 tiles, against the oracle.  The BF16 kernel's
raw approximate row minima are also checked against FP64 minima within the
error bound the certification relies on."""
import ctypes

import numpy as np
import pytest

import hd_oracle
from hausdorffdistance_gb300 import synth

pytestmark = pytest.mark.gpu
REL_TOL_F64 = 1e-6


def row_bound(a, b, K):
    """Python copy of the kernel's per-row bound (hd_bf16.cu, row_bound)."""
    c = 4.0 * 2.0 ** -18 + (3.0 * K + 16.0) * 2.0 ** -23
    s = (a + b) ** 2
    e = 2.0 * c * a * b + 2.0 ** -21 * s + (K + 2.0) * 2.0 ** -24 * s
    return 2.0 * e + 1e-30


def exact_rowmin(a, b):
    a64 = a.astype(np.float64)
    b64 = b.astype(np.float64)
    out = np.empty(len(a))
    for s in range(0, len(a), 256):
        d = ((a64[s:s + 256, None, :] - b64[None, :, :]) ** 2).sum(-1)
        out[s:s + 256] = d.min(1)
    return out


@pytest.mark.parametrize("dims", [16, 32, 48, 64])
def test_bf16_rowmin_within_certified_bound(engine, dims):
    from hausdorffdistance_gb300 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(dims)
    a = (rng.standard_normal((700, dims)) * rng.uniform(0.2, 3.0, (700, 1))).astype(np.float32)
    b = (rng.standard_normal((900, dims)) * rng.uniform(0.2, 3.0, (900, 1))).astype(np.float32)
    b[:50] = a[:50]  # exact duplicates: minima of 0
    rowmin = np.zeros(len(a), np.float32)
    st = lib.hd_debug_bf16_rowmin(engine._h, a.ctypes.data, len(a), b.ctypes.data, len(b), dims,
                                  rowmin.ctypes.data)
    assert st == 0, lib.hd_last_error(engine._h)
    want = exact_rowmin(a, b)
    bmax = np.linalg.norm(b.astype(np.float64), axis=1).max()
    an = np.linalg.norm(a.astype(np.float64), axis=1)
    err = np.abs(rowmin.astype(np.float64) - want)
    assert np.all(err <= row_bound(an, bmax, dims)), err.max()
    # The bound is loose; the split products are far more accurate than it.
    assert err.max() < 1e-3 * (an.max() * bmax)


@pytest.mark.parametrize("variant", ["bf16", "eb", "brute", "auto"])
@pytest.mark.parametrize("dims", [16, 64])
def test_highdim_matches_oracle(engine, variant, dims):
    a, b = synth.unit64(3000, seed=30 + dims, dims=dims, replace_frac=0.02)
    b = b[:2500]
    r = engine.solve(a, b, undirected=True, variant=variant)
    want = hd_oracle.hd_f32(a, b, undirected=True)
    assert np.float32(r.hd_f32) == want["hd_f32"]
    assert r.hd == pytest.approx(hd_oracle.hd_f64(a, b, True), rel=REL_TOL_F64)
    src, dst = (a, b) if r.direction == 0 else (b, a)
    assert hd_oracle.dist2_f32(src[r.ia], dst[r.ib]) == want["d2"]
    if variant == "bf16":
        assert r.rechecked >= 1 and r.err_bound > 0


@pytest.mark.parametrize("dims", [1, 4, 5, 7, 24, 100, 128])
@pytest.mark.parametrize("variant", ["eb", "brute"])
def test_fp32_scans_any_dims(engine, dims, variant):
    rng = np.random.default_rng(dims * 3)
    a = rng.random((1500, dims)).astype(np.float32)
    b = rng.random((1300, dims)).astype(np.float32) * 1.05
    r = engine.solve(a, b, undirected=True, variant=variant)
    want = hd_oracle.hd_f32(a, b, undirected=True)
    assert np.float32(r.hd_f32) == want["hd_f32"]


def test_bf16_rejects_unsupported_dims(engine):
    import hausdorffdistance_gb300 as hd
    a = np.ones((10, 20), np.float32)
    with pytest.raises(hd.HDError) as ei:
        engine.solve(a, a, variant="bf16")
    assert ei.value.status == 5


# Runs of tiles with rows dropped between them (|A| * |B| >= 2e9): fewer rows
# than one seed block, a ragged last row block and tile, B far from A (no row
# drops out early), exact copies (every early seed may be one), one repeated
# point (every row ties, none can be dropped).
@pytest.mark.parametrize("na,nb,dims,kind", [
    (200, 10_000_019, 16, "gauss"), (45_000, 44_501, 64, "copies"), (50_001, 40_003, 48, "far"),
    (70_000, 30_000, 32, "repeated"), (2_000_003, 1025, 16, "gauss")])
def test_bf16_runs_of_tiles(engine, na, nb, dims, kind):
    rng = np.random.default_rng(na + dims)
    a = rng.standard_normal((na, dims), dtype=np.float32)
    if kind == "copies":
        b = a[rng.permutation(na)[:nb]].copy()
        b[::100] = rng.standard_normal(b[::100].shape, dtype=np.float32)
    elif kind == "repeated":
        a[:] = a[0]
        b = np.repeat(a[:1] + np.float32(0.5), nb, axis=0)
    else:
        b = rng.standard_normal((nb, dims), dtype=np.float32)
        if kind == "far":
            b += np.float32(10.0)
    r = engine.solve(a, b, variant="bf16")
    if kind == "repeated":
        d2 = hd_oracle.dist2_f32(a[0], b[0])
    else:
        d2 = hd_oracle.exact(a, b, 32)[0]
    assert np.float32(r.hd_f32) == np.sqrt(np.float32(d2))
    assert hd_oracle.dist2_f32(a[r.ia], b[r.ib]) == np.float32(d2)


# AUTO pads rows to a multiple of 16 for the tiles; rows far from the origin,
# whose bound exceeds their distances, and rows that all tie go back to the scan.
@pytest.mark.parametrize("dims", [1, 4, 5, 10, 24, 31, 33, 63])
@pytest.mark.parametrize("kind", ["plain", "far_from_origin", "all_tie"])
def test_auto_pads_to_tiles(engine, dims, kind):
    rng = np.random.default_rng(dims)
    a = rng.random((2105, dims)).astype(np.float32)
    b = (rng.random((1999, dims)) * 1.05).astype(np.float32)
    if kind == "far_from_origin":
        a, b = a + np.float32(300.0), b + np.float32(300.0)
    elif kind == "all_tie":
        a[:] = a[0]
        b[:] = a[0] + np.float32(0.25)
    r = engine.solve(a, b, undirected=True)
    want = hd_oracle.hd_f32(a, b, undirected=True)
    assert np.float32(r.hd_f32) == want["hd_f32"]
    src, dst = (a, b) if r.direction == 0 else (b, a)
    assert hd_oracle.dist2_f32(src[r.ia], dst[r.ib]) == want["d2"]
    assert r.variant_used == 4


# No tiles are built past 64 dimensions: AUTO scans there at any size.
@pytest.mark.parametrize("dims", [65, 80, 96, 100, 112, 127, 128])
@pytest.mark.parametrize("na,nb", [(2011, 1501), (300, 7001)])
def test_auto_scans_beyond_the_tiles(engine, dims, na, nb):
    rng = np.random.default_rng(dims + na)
    a = rng.standard_normal((na, dims)).astype(np.float32)
    b = rng.standard_normal((nb, dims)).astype(np.float32)
    r = engine.solve(a, b, undirected=True)
    want = hd_oracle.hd_f32(a, b, undirected=True)
    assert np.float32(r.hd_f32) == want["hd_f32"]
    src, dst = (a, b) if r.direction == 0 else (b, a)
    assert hd_oracle.dist2_f32(src[r.ia], dst[r.ib]) == want["d2"]
    assert r.variant_used == 1 and r.variant_used_ba == 1


# Inputs that leave the tiles' bounds without a value: AUTO answers what the scan
# by name answers, or fails as it does (a row with a NaN has no nearest point).
# The sizes are below and above those of runs of tiles.
@pytest.mark.parametrize("kind", ["nan_targets", "huge_targets", "all_huge", "nan_row",
                                  "huge_row", "huge_row_and_products"])
@pytest.mark.parametrize("dims,na,nb", [(10, 2105, 1999), (16, 2105, 1999), (64, 200, 15_001),
                                        (16, 50_001, 40_003)])
def test_auto_where_bounds_have_no_value(engine, kind, dims, na, nb):
    import hausdorffdistance_gb300 as hd
    rng = np.random.default_rng(dims + na)
    a = rng.random((na, dims)).astype(np.float32)
    b = (rng.random((nb, dims)) * 1.05).astype(np.float32)
    keep = np.ones(nb, bool)
    if kind == "all_huge":  # FP32 values near 2e19 lie 2e12 apart
        a = (2e19 + 1e16 * a.astype(np.float64)).astype(np.float32)
        b = (2e19 + 1e16 * b.astype(np.float64)).astype(np.float32)
    elif kind in ("nan_targets", "huge_targets"):
        keep[::700] = False
        b[~keep, dims // 2] = 1e25 if kind == "huge_targets" else np.nan
        a[7] = 0.0
    else:
        if kind == "huge_row_and_products":
            b += np.float32(4.0)
        a[7, 1] = np.nan if kind == "nan_row" else 1e38
    got = []
    for variant in ("auto", "eb"):
        try:
            r = engine.solve(a, b, variant=variant)
            got.append((np.float32(r.hd_f32), r.hd, int(r.ia), int(r.ib)))
        except hd.HDError as e:
            got.append(e.status)
    assert got[0] == got[1]
    if keep.sum() < nb or kind == "all_huge":
        d2 = hd_oracle.exact(a, b[keep], 32)[0]
        assert got[0][0] == np.sqrt(np.float32(d2)) and keep[got[0][3]]
        assert hd_oracle.dist2_f32(a[got[0][2]], b[got[0][3]]) == np.float32(d2)


# Few targets don't repay packing A: there AUTO scans, in either direction by its
# own sizes.
@pytest.mark.parametrize("dims,na,nb,tiles", [
    (4, 200_000, 599, False), (4, 20_000, 600, True), (4, 151_000, 1000, False),
    (10, 100_000, 299, False), (16, 20_000, 300, True), (16, 600_000, 320, False),
    (32, 100_000, 99, False), (32, 100_000, 100, True), (64, 100_000, 20, True)])
def test_auto_scans_for_few_targets(engine, dims, na, nb, tiles):
    rng = np.random.default_rng(dims + nb)
    a = rng.standard_normal((na, dims)).astype(np.float32)
    b = rng.standard_normal((nb, dims)).astype(np.float32)
    r = engine.solve(a, b)
    d2 = hd_oracle.exact(a, b, 32)[0]
    assert np.float32(r.hd_f32) == np.sqrt(np.float32(d2))
    assert hd_oracle.dist2_f32(a[r.ia], b[r.ib]) == np.float32(d2)
    assert r.variant_used == (4 if tiles else 1)
