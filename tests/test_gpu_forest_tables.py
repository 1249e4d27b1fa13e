"""The table of checked reciprocals that predictions read depends on nothing in a forest: it is made once per context,
also where several threads make its first forests at a time, and outlives the forest that made it."""
import threading

import numpy as np
import pytest

import curfil_b200 as cf
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [1, 4])
def test_reciprocals_are_made_once_per_context(threads):
    from curfil_b200 import _build
    _build.build()
    ctx = cf.Context(0)
    rgb, depth, labels = H.frames(seed=4, n=2, w=61, h=43, cells=5, classes=4)
    cfg = cf.TrainConfig(feature_count=32, thresholds=5, max_depth=5, min_sample_count=5, box_radius=9, region_size=3,
                         samples_per_image=80, sampler=1)
    trees = cf.train_forest(ctx, rgb, depth, labels, 4, cfg, 2)
    want = None
    ctx.set_timing(True)
    ctx.reset_timing()
    results, errors = [], []

    def work():
        try:
            for _ in range(3):
                forest = cf.Forest(ctx, trees)
                with lock:   # predictions of one context are made one at a time
                    results.append(forest.predict(rgb, depth))
                forest.close()
        except Exception as e:   # noqa: BLE001
            errors.append(e)
    lock = threading.Lock()
    pool = [threading.Thread(target=work) for _ in range(threads)]
    for t in pool:
        t.start()
    for t in pool:
        t.join()
    assert not errors
    launches = ctx.kernel_time("reciprocals")[1]
    ctx.set_timing(False)
    forest = cf.Forest(ctx, trees)
    want = forest.predict_plain(rgb, depth)
    for probs, lab in results:
        np.testing.assert_array_equal(probs.view(np.uint32), want[0].view(np.uint32))
        np.testing.assert_array_equal(lab, want[1])
    forest.close()
    for t in trees:
        t.close()
    ctx.close()
    assert launches == 1
