"""The views of a prediction graph's pinned buffers hold the graph: a result outlives the last name of the graph."""
import gc
import weakref

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


@pytest.mark.parametrize("probabilities", [False, True])
def test_a_view_keeps_the_graph(ctx, probabilities):
    rgb, depth, labels = H.frames(seed=3, n=2, w=33, h=17, cells=4, classes=3)
    cfg = cf.TrainConfig(feature_count=32, thresholds=5, max_depth=4, min_sample_count=5, box_radius=8, region_size=3,
                         samples_per_image=60, sampler=1)
    forest = cf.Forest(ctx, cf.train_forest(ctx, rgb, depth, labels, 3, cfg, 1))
    graph = cf.PredictGraph(forest, 2, 33, 17, probabilities=probabilities)
    graph.rgb[...] = rgb
    graph.depth[...] = depth
    graph.run()
    held = weakref.ref(graph)
    view = graph.probabilities if probabilities else graph.labels
    want = view.copy()
    assert (graph.probabilities is None) == (not probabilities)
    del graph
    gc.collect()
    assert held() is not None
    part = view[1:]
    del view
    gc.collect()
    assert held() is not None
    np.testing.assert_array_equal(part, want[1:])
    del part
    gc.collect()
    assert held() is None
