"""The forms of the prediction kernel (csrc/classify.cu) against the plain form, bit for bit: one, two and four threads
a pixel over the class counts of every instance and over more trees than are walked at a time; frames whose byte
offsets pass 2^24 (element indices in integers), up to sides that take the general responses; padded frames."""
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


def random_tree(rng, ds, samples, C, levels=8, along_rows=False):
    """A tree of uneven depth whose thresholds are responses of the frames' own pixels, so that some pixels meet
    their threshold exactly; parameters up to the ends of their range."""
    left, depth = [-1], [0]
    for i in range(1 << (levels + 1)):
        if i >= len(left):
            break
        if depth[i] < levels and (depth[i] < 2 or rng.random() < 0.8):
            left[i] = len(left)
            left += [-1, -1]
            depth += [depth[i] + 1] * 2
    n = len(left)
    f = H.random_features(rng, n, box_radius=90, region_size=12)
    odd = rng.random(n) < 0.1
    f[1:5, odd] = rng.choice(np.array([-128, -127, -1, 0, 1, 127], np.int8), (4, int(odd.sum())))
    f[5:9, odd] = rng.choice(np.array([-3, 0, 1, 127], np.int8), (4, int(odd.sum())))
    if along_rows:
        f[[2, 4]] = 0
    r = cf.feature_responses(ds, samples, f)
    thr = np.nan_to_num(r[np.arange(n), rng.integers(0, len(samples), n)], nan=0.0).astype(np.float32)
    hist = rng.integers(0, 50, (n, C)) * (rng.random((n, C)) < 0.4)
    hist[:, 0] += 1
    return cf.Tree.from_arrays(0, np.array(left, np.int32), np.ascontiguousarray(f.T), thr, hist.astype(np.uint32))


def noisy_frames(rng, n, w, h):
    rgb = rng.integers(0, 256, (n, h, w, 3), dtype=np.uint8)
    blocks = rng.integers(300, 6000, (n, -(-h // 16), -(-w // 16)))
    depth = (np.kron(blocks, np.ones((1, 16, 16), np.int64))[:, :h, :w] + rng.integers(0, 40, (n, h, w))).astype(np.uint16)
    depth[rng.random(depth.shape) < 0.1] = 0
    return rgb, depth


def assert_equals_plain(ctx, ds, depth, n, w, h, trees, C, seed):
    import torch
    rng = np.random.default_rng(seed)
    s = H.random_samples(rng, n, w, h, C, 400, depth=depth)
    grown = [random_tree(rng, ds, s, C) for _ in range(trees)]
    forest = cf.Forest(ctx, grown, prior=rng.integers(1, 100, C).astype(np.uint32))
    out = []
    for predict in (forest.predict_dataset, forest.predict_dataset_plain):
        probs = torch.zeros((n, C, h, w), dtype=torch.float32, device="cuda:0")
        labels = torch.zeros((n, h, w), dtype=torch.uint8, device="cuda:0")
        torch.cuda.synchronize()
        predict(ds, 0, n, probs.data_ptr(), labels.data_ptr())
        ctx.synchronize()
        out.append((probs.view(torch.int32), labels))
    assert torch.equal(out[0][0], out[1][0])
    assert torch.equal(out[0][1], out[1][1])
    assert len(torch.unique(out[0][1])) > 1
    forest.close()
    for t in grown:
        t.close()


@pytest.mark.parametrize("w,h,trees,C", [(1400, 999, 2, 13), (1400, 1000, 1, 13), (1920, 1080, 5, 40), (1399, 1001, 3, 100),
                                         (65535, 24, 2, 5)])
def test_large_frames_equal_the_plain_form(ctx, w, h, trees, C):
    rng = np.random.default_rng(w + h)
    rgb, depth = noisy_frames(rng, 1, w, h)
    ds = cf.Dataset.from_raw(ctx, rgb, depth)
    assert_equals_plain(ctx, ds, depth, 1, w, h, trees, C, seed=trees * 1000 + C)
    ds.close()


@pytest.mark.parametrize("w", [1500000, 2097152, 2097153])
def test_long_host_frames_equal_the_plain_form(ctx, w):
    h, C = 3, 5
    rng = np.random.default_rng(w)
    rgb, depth = noisy_frames(rng, 1, w, h)
    depth[depth > 0] += 59000   # boxes of three rows and columns, offsets of up to two columns
    piece = np.ascontiguousarray(rgb[:, :, -5000:]), np.ascontiguousarray(depth[:, :, -5000:])
    ds = cf.Dataset.from_raw(ctx, *piece)
    s = H.random_samples(rng, 1, 5000, h, C, 400, depth=piece[1])
    s["y"] = 1
    grown = [random_tree(rng, ds, s, C, along_rows=True) for _ in range(2)]
    ds.close()
    forest = cf.Forest(ctx, grown, prior=np.full(C, 7, np.uint32))
    p1, l1 = forest.predict(rgb, depth)
    p2, l2 = forest.predict_plain(rgb, depth)
    np.testing.assert_array_equal(p1.view(np.uint32), p2.view(np.uint32))
    np.testing.assert_array_equal(l1, l2)
    assert len(np.unique(l1[0, 1])) > 1
    forest.close()


# 595 tiles of 16 x 16 pixels take the forms of large launches, 35 the four threads of small ones
@pytest.mark.parametrize("n", [17, 1])
@pytest.mark.parametrize("trees,C", [(1, 5), (3, 16), (4, 8), (2, 17), (3, 32), (4, 31), (1, 40), (2, 33), (5, 40), (1, 41),
                                     (3, 64), (1, 65), (3, 128), (2, 129), (1, 256), (32, 7), (33, 13), (33, 40), (65, 3),
                                     (65, 64), (34, 70)])
def test_threads_per_pixel_equal_the_plain_form(ctx, n, trees, C):
    w, h = 97, 71
    rng = np.random.default_rng(trees * 300 + C)
    rgb, depth = noisy_frames(rng, n, w, h)
    ds = cf.Dataset.from_raw(ctx, rgb, depth)
    assert_equals_plain(ctx, ds, depth, n, w, h, trees, C, seed=trees + C)
    ds.close()


@pytest.mark.parametrize("n", [18, 1])
def test_padded_frames_equal_the_plain_form(ctx, n):
    """Corners in the padding hold NaN colours and zero depth integrals: box counts come out zero or negative."""
    w, h = 96, 72
    rng = np.random.default_rng(n)
    rgb, depth = noisy_frames(rng, n, 70, 50)
    ds = cf.Dataset(ctx, n, w, h)
    ds.upload_raw_padded(rgb, depth)
    padded = np.zeros((n, h, w), np.uint16)
    padded[:, :50, :70] = depth
    assert_equals_plain(ctx, ds, padded, n, w, h, 5, 13, seed=n)
    ds.close()


def test_depths_past_the_table_equal_the_plain_form(ctx):
    """Depths above 65.535 m have no checked reciprocal in the forest's table."""
    n, w, h, C = 17, 97, 71, 13
    rng = np.random.default_rng(9)
    rgb, depth = noisy_frames(rng, n, w, h)
    far = depth.astype(np.int64) * np.where(rng.random(depth.shape) < 0.5, 37, 1)
    color = np.cumsum(np.cumsum(rgb.transpose(0, 3, 1, 2).astype(np.int64), 3), 2).astype(np.float32)
    planes = np.stack([np.cumsum(np.cumsum(v, 2), 1) for v in (far, (far > 0).astype(np.int64))], 1).astype(np.int32)
    ds = cf.Dataset.from_integral(ctx, color, np.ascontiguousarray(planes))
    assert (far > 65535).mean() > 0.2
    assert_equals_plain(ctx, ds, depth, n, w, h, 5, C, seed=3)
    ds.close()
