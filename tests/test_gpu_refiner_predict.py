"""Refined prediction over the widths and radii that its kernels distinguish (hidden units of 32, 64 and 128 lanes,
box radii on either side of a run of eight outputs and of the tiled kernel's limit) and over frames that leave
partial tiles, against numpy in 64 bits.

Tolerances: a box mean is two float sums of at most 35 terms each and a division, within 72 x 2^-24 < 5e-6
relative. A logit is two chains of at most 130 fused multiply-adds; with the parameters below the absolute terms
of a chain sum to less than 16, so a logit is within 260 x 16 x 2^-24 < 2.5e-4 and a probability within twice that.
"""
import numpy as np
import pytest
import torch

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


def box_mean(p, r):
    C, h, w = p.shape
    cs = np.zeros((C, h + 1, w + 1))
    cs[:, 1:, 1:] = p.astype(np.float64).cumsum(1).cumsum(2)
    y, x = np.arange(h), np.arange(w)
    y0, y1 = np.maximum(0, y - r), np.minimum(h, y + r + 1)
    x0, x1 = np.maximum(0, x - r), np.minimum(w, x + r + 1)
    s = cs[:, y1][:, :, x1] - cs[:, y0][:, :, x1] - cs[:, y1][:, :, x0] + cs[:, y0][:, :, x0]
    return s / ((y1 - y0)[:, None] * (x1 - x0)[None])


@pytest.mark.parametrize("hidden,radii,w,h,C", [(5, (0, 1), 67, 65, 6), (32, (3, 4), 64, 64, 9), (33, (4, 16), 96, 72, 6),
                                                (64, (16, 3), 130, 37, 13), (65, (2, 17), 70, 66, 2),
                                                (128, (4, 16), 33, 129, 17)])
def test_refined_prediction_matches_numpy(ctx, hidden, radii, w, h, C):
    rgb, depth, labels = H.frames(seed=hidden, n=2, w=w, h=h, cells=8, classes=C)
    ds = cf.Dataset.from_raw(ctx, rgb, depth)
    samples, _ = H.class_uniform_samples(labels, depth, C, 40)
    cfg = cf.TrainConfig(feature_count=40, thresholds=8, max_depth=5, min_sample_count=10, box_radius=20, region_size=6)
    tree, _ = cf.train_tree(ds, samples, C, cfg, seed_counter=3)
    forest = cf.Forest(ctx, [tree], prior=np.ones(C, np.uint32))
    r = cf.Refiner(ctx, C, hidden=hidden, radius1=radii[0], radius2=radii[1])
    D = 3 * C + 2
    rng = np.random.default_rng(hidden)
    prm = (rng.uniform(-1, 1, hidden * D + hidden + C * hidden + C) * 0.25).astype(np.float32)
    r.params(new=prm)
    probs = torch.empty(2, C, h, w, device="cuda")
    lab = torch.empty(2, h, w, dtype=torch.uint8, device="cuda")
    r.predict(forest, ds, 0, 2, probs.data_ptr(), lab.data_ptr())
    probs, lab = probs.cpu().numpy(), lab.cpu().numpy()
    p0, _ = forest.predict_dataset_host(ds, 0, 2)
    W1, b1, W2, b2 = np.split(prm.astype(np.float64), np.cumsum([hidden * D, hidden, C * hidden]))
    for i in range(2):
        means = [box_mean(p0[i], k) for k in radii]
        xy = np.stack(np.meshgrid(np.arange(w), np.arange(h)), -1).reshape(-1, 2).astype(np.int32)
        rows = r.features(forest, ds, i, xy).reshape(h, w, D).transpose(2, 0, 1)
        np.testing.assert_array_equal(rows[:C], p0[i])
        for k in range(2):
            np.testing.assert_allclose(rows[(k + 1) * C:(k + 2) * C], means[k], rtol=5e-6, atol=1e-12)
        m = depth[i].astype(np.float64) / 1000
        X = np.concatenate([p0[i].astype(np.float64), *means, m[None] / 5, (m > 0)[None]]).reshape(D, -1)
        hid = np.maximum(W1.reshape(hidden, D) @ X + b1[:, None], 0)
        z = W2.reshape(C, hidden) @ hid + b2[:, None]
        e = np.exp(z - z.max(0))
        e /= e.sum(0)
        np.testing.assert_allclose(probs[i].reshape(C, -1), e, atol=5e-4)
        top = np.sort(e, 0)
        sure = top[-1] - top[-2] > 2e-3
        assert sure.mean() > 0.5
        np.testing.assert_array_equal(lab[i].reshape(-1)[sure], e.argmax(0)[sure])
    r.close()
    forest.close()
    ds.close()
