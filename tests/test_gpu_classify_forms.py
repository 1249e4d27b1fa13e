"""The forms of the prediction kernel (csrc/classify.cu) against the plain form, bit for bit: frames whose byte
offsets pass 2^24 (element indices in integers), up to sides that take the general responses."""
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
