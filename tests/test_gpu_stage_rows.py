"""Pass 1 of the staged split search (csrc/stage.cu) against the fused search, whose bins come from feature_bin:
threshold counts on either side of the padded rows, candidates in any order with extreme parameters, feature
counts that leave partial units, ragged frames, and depths with and without a checked reciprocal."""
import numpy as np
import pytest

import curfil_b200 as cf
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from curfil_b200 import _build
    _build.build()
    c = cf.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("T", [1, 31, 32, 33, 63, 64])
@pytest.mark.parametrize("F,w,h", [(1, 33, 27), (77, 97, 71), (264, 128, 96)])
def test_bins_equal_the_fused_search(ctx, T, F, w, h):
    n, C = 4, 17
    rgb, depth, labels = H.frames(seed=T + F, n=n, w=w, h=h, cells=9, classes=C)
    ds = cf.Dataset.from_raw(ctx, rgb, depth)
    rng = np.random.default_rng(1000 * T + F)
    sizes = [1, 65, 700, 31, 64, 1500, 2]
    offsets = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    s = H.random_samples(rng, n, w, h, C, int(offsets[-1]), depth=depth, flips=True)
    # depths in whole millimetres without a checked reciprocal, invalid ones, and far outside the usual range
    odd = np.array([0.3, 0.36, 0.6, 0.72, 1.2, 2.4, 0.0, -1.0, np.nan, np.inf, 1e-4, 1e-3, 1e6, 3e7, 1.2345678],
                   np.float32)
    pick = rng.random(len(s)) < 0.3
    s["depth"][pick] = rng.choice(odd, int(pick.sum()))
    fe = H.random_features(rng, F)                     # depth and colour candidates in random order
    fe[1:5, : F // 4] = rng.choice(np.array([-128, -127, 0, 127], np.int8), (4, F // 4))
    fe[5:9, : F // 5] = rng.choice(np.array([-5, 0, 1, 127], np.int8), (4, F // 5))
    r = cf.feature_responses(ds, s, fe)
    th = np.empty((T, F), np.float32)
    for t in range(T):
        th[t] = np.nan_to_num(r[np.arange(F), rng.integers(0, len(s), F)], nan=0.0)
    out = {}
    try:
        for stage in (0, 2):
            ctx.set_tuning(stage_bins=stage, stage_max_mb=1)
            out[stage] = cf.level_left_counts(ds, offsets, s, C, fe, th)
    finally:
        ctx.set_tuning()
        ds.close()
    np.testing.assert_array_equal(out[2][1], out[0][1])
    for k in ("score", "feature", "threshold_index", "threshold"):
        np.testing.assert_array_equal(out[2][0][k], out[0][0][k], err_msg=k)


@pytest.mark.parametrize("T", [64, 200])
@pytest.mark.parametrize("rows", [4000, 90000])
def test_general_bins_of_small_and_large_levels(ctx, T, rows):
    """Thresholds that the gather kernel does not serve, in levels on both sides of the item count from which the
    general kernel takes wider tiles (2664 items of 256 rows x 32 features on 148 SMs)."""
    n, C, F, w, h = 3, 11, 250, 97, 71
    rgb, depth, labels = H.frames(seed=T, n=n, w=w, h=h, cells=9, classes=C)
    ds = cf.Dataset.from_raw(ctx, rgb, depth)
    rng = np.random.default_rng(T + rows)
    offsets = np.array([0, rows // 7, rows // 7 + 1, rows], np.int64)
    s = H.random_samples(rng, n, w, h, C, rows, depth=depth)
    fe = H.random_features(rng, F)
    r = cf.feature_responses(ds, s[:500], fe)
    th = np.nan_to_num(r[np.arange(F), rng.integers(0, 500, (T, F))], nan=0.0).astype(np.float32)
    out = {}
    try:
        for stage in (0, 2):
            ctx.set_tuning(stage_bins=stage)
            ctx.set_timing(True)
            ctx.reset_timing()
            out[stage] = cf.level_left_counts(ds, offsets, s, C, fe, th)
            assert (ctx.kernel_time("stage_bins")[1] > 0) == (stage == 2)
            ctx.set_timing(False)
    finally:
        ctx.set_timing(False)
        ctx.set_tuning()
        ds.close()
    np.testing.assert_array_equal(out[2][1], out[0][1])
    for k in ("score", "feature", "threshold_index", "threshold"):
        np.testing.assert_array_equal(out[2][0][k], out[0][0][k], err_msg=k)


@pytest.mark.parametrize("rows,F,T,staged", [(84000, 100, 20, False), (168000, 100, 20, True), (66000, 128, 20, True),
                                             (65000, 128, 20, False), (66000, 128, 64, False)])
def test_levels_within_l2_are_staged_by_their_size(ctx, rows, F, T, staged):
    n, C, w, h = 3, 5, 97, 71
    rgb, depth, labels = H.frames(seed=F, n=n, w=w, h=h, cells=9, classes=C)
    ds = cf.Dataset.from_raw(ctx, rgb, depth)
    rng = np.random.default_rng(rows + T)
    offsets = np.array([0, rows // 3, rows], np.int64)
    s = H.random_samples(rng, n, w, h, C, rows, depth=depth)
    fe = H.random_features(rng, F)
    r = cf.feature_responses(ds, s[:500], fe)
    th = np.nan_to_num(r[np.arange(F), rng.integers(0, 500, (T, F))], nan=0.0).astype(np.float32)
    out = {}
    try:
        for stage in (0, 1):
            ctx.set_tuning(stage_bins=stage)
            ctx.set_timing(True)
            ctx.reset_timing()
            out[stage] = cf.evaluate_best_splits(ds, offsets, s, C, fe, th)
            assert (ctx.kernel_time("stage_bins")[1] > 0) == (staged and stage == 1)
            ctx.set_timing(False)
    finally:
        ctx.set_timing(False)
        ctx.set_tuning()
        ds.close()
    for k in ("score", "feature", "threshold_index", "threshold"):
        np.testing.assert_array_equal(out[1][k], out[0][k], err_msg=k)


def assert_staged_equals_fused(ctx, ds, offsets, s, C, fe, th):
    out = {}
    try:
        for stage in (0, 2):
            ctx.set_tuning(stage_bins=stage)
            ctx.set_timing(True)
            ctx.reset_timing()
            out[stage] = cf.level_left_counts(ds, offsets, s, C, fe, th)
            assert (ctx.kernel_time("stage_bins")[1] > 0) == (stage == 2)
            ctx.set_timing(False)
    finally:
        ctx.set_timing(False)
        ctx.set_tuning()
    np.testing.assert_array_equal(out[2][1], out[0][1])
    for k in ("score", "feature", "threshold_index", "threshold"):
        np.testing.assert_array_equal(out[2][0][k], out[0][0][k], err_msg=k)


@pytest.mark.parametrize("T", [20, 32, 45, 64])
def test_bins_on_padded_frames_equal_the_fused_search(ctx, T):
    """Corners in the padding hold NaN colours and zero depth integrals: counts of boxes come out zero or negative."""
    n, C, w, h, F = 4, 13, 70, 50, 160
    rgb, depth, labels = H.frames(seed=T, n=n, w=w, h=h, cells=9, classes=C)
    ds = cf.Dataset(ctx, n, 96, 72)
    ds.upload_raw_padded(rgb, depth)
    rng = np.random.default_rng(T)
    offsets = np.array([0, 1, 900, 901, 3000], np.int64)
    s = H.random_samples(rng, n, w, h, C, 3000, depth=depth, flips=True)
    fe = H.random_features(rng, F)
    r = cf.feature_responses(ds, s[:500], fe)
    th = np.nan_to_num(r[np.arange(F), rng.integers(0, 500, (T, F))], nan=0.0).astype(np.float32)
    assert_staged_equals_fused(ctx, ds, offsets, s, C, fe, th)
    ds.close()


@pytest.mark.parametrize("w,h", [(1399, 999), (1400, 1000)])
def test_bins_on_large_frames_equal_the_fused_search(ctx, w, h):
    """Frames on either side of the largest one whose byte offsets the gather kernel holds in floats."""
    n, C, F, T = 1, 7, 96, 20
    rng = np.random.default_rng(w)
    rgb = rng.integers(0, 256, (n, h, w, 3), dtype=np.uint8)
    depth = rng.integers(500, 5001, (n, h, w)).astype(np.uint16)
    depth[rng.random(depth.shape) < 0.1] = 0
    ds = cf.Dataset.from_raw(ctx, rgb, depth)
    offsets = np.array([0, 700, 2500], np.int64)
    s = H.random_samples(rng, n, w, h, C, 2500, depth=depth, flips=True)
    s["x"][:200], s["y"][:200] = w - 1 - rng.integers(0, 60, 200), h - 1 - rng.integers(0, 60, 200)
    s["depth"][:200] = np.float32(2.5)
    fe = H.random_features(rng, F)
    r = cf.feature_responses(ds, s[:500], fe)
    th = np.nan_to_num(r[np.arange(F), rng.integers(0, 500, (T, F))], nan=0.0).astype(np.float32)
    assert_staged_equals_fused(ctx, ds, offsets, s, C, fe, th)
    ds.close()
