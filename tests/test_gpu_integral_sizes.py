"""Integral images, depth filling and plane integration at the sizes their kernels distinguish: rows on either side
of a 128-pixel step, widths that are no multiple of 4 (pixel-wise reads), columns on either side of a 128-row
step, single rows and columns, empty rows; exact against numpy (the sums are integers, or doubles added in the
same order)."""
import numpy as np
import pytest

import curfil_b200 as cf

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (3, 130), (4, 127), (33, 128), (127, 9), (128, 7), (129, 257), (132, 300), (260, 40), (257, 33)]


@pytest.fixture(scope="module")
def ctx():
    from curfil_b200 import _build
    _build.build()
    c = cf.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("w,h", SIZES)
def test_integral_images_equal_numpy(ctx, w, h):
    rng = np.random.default_rng(w * 1000 + h)
    rgb = rng.integers(0, 256, (3, h, w, 3), dtype=np.uint8)
    depth = rng.integers(0, 65536, (3, h, w)).astype(np.uint16)
    depth[rng.random(depth.shape) < 0.2] = 0
    rgb[1], depth[1] = 255, 65535
    ds = cf.Dataset.from_raw(ctx, rgb, depth)
    color, d = ds.download_integral()
    ds.close()
    want = rgb.transpose(0, 3, 1, 2).astype(np.uint64).cumsum(3).cumsum(2)
    np.testing.assert_array_equal(color, want.astype(np.float32))
    sums = depth.astype(np.uint64).cumsum(2).cumsum(1).astype(np.uint32).view(np.int32)
    np.testing.assert_array_equal(d[:, 0], sums)
    np.testing.assert_array_equal(d[:, 1], (depth > 0).astype(np.int64).cumsum(2).cumsum(1))


def fill(d):
    d = d.copy()
    h, w = d.shape
    for x in range(w - 2, -1, -1):
        d[:, x] = np.where(d[:, x] == 0, d[:, x + 1], d[:, x])
    for x in range(1, w):
        d[:, x] = np.where(d[:, x] == 0, d[:, x - 1], d[:, x])
    for y in range(1, h):
        d[y] = np.where(d[y] == 0, d[y - 1], d[y])
    for y in range(h - 2, -1, -1):
        d[y] = np.where(d[y] == 0, d[y + 1], d[y])
    return d


@pytest.mark.parametrize("w,h", SIZES)
def test_fill_depth_equals_the_four_passes(ctx, w, h):
    rng = np.random.default_rng(w + h)
    d = rng.integers(1, 5000, (6, h, w)).astype(np.uint16)
    for i, missing in enumerate((0.0, 0.1, 0.9, 0.99, 1.0, 0.5)):
        d[i][rng.random((h, w)) < missing] = 0
    d[5, : h // 3] = 0           # empty rows at the top, in the middle and at the bottom
    d[5, h // 2] = 0
    d[5, -1] = 0
    np.testing.assert_array_equal(cf.fill_depth(ctx, d), np.stack([fill(x) for x in d]))


@pytest.mark.parametrize("w,h", SIZES)
def test_plane_integrals_equal_sums_in_order(ctx, w, h):
    rng = np.random.default_rng(w * 7 + h)
    color = rng.normal(0, 50, (2, 3, h, w)).astype(np.float32)
    depth = rng.integers(0, 5000, (2, 2, h, w)).astype(np.int32)
    c, d = cf.integrate_planes(ctx, color, depth)
    np.testing.assert_array_equal(c, color.astype(np.float64).cumsum(3).cumsum(2).astype(np.float32))
    np.testing.assert_array_equal(d, depth.astype(np.int64).cumsum(3).cumsum(2).astype(np.int32))
