"""The buffers of a prediction graph as a program sees them (host logic; the library's graph calls are replaced by
ones that hand out numpy memory)."""
import ctypes

import numpy as np
import pytest

import curfil_b200 as cf


class FakeLibrary:
    """The cf_predict_graph_* entry points over host memory."""
    kept = []

    def __init__(self, n, w, h, C):
        self.memory = [np.zeros(n * h * w * 3, np.uint8), np.zeros(n * h * w, np.uint16),
                       np.zeros(n * C * h * w, np.float32), np.zeros(n * h * w, np.uint8)]
        self.destroyed = 0
        self.kept.append(self.memory)   # for the views in the report of a failed test

    def cf_predict_graph_create(self, forest, count, width, height, probabilities, out):
        out._obj.value = 1
        return 0

    def cf_predict_graph_buffers(self, handle, *places):
        for place, m in zip(places, self.memory):
            place._obj.value = m.ctypes.data
        return 0

    def cf_predict_graph_destroy(self, handle):
        self.destroyed += 1
        return 0


class FakeForest:
    handle = ctypes.c_void_p(1)
    num_classes = 4


@pytest.fixture
def library(monkeypatch):
    fake = FakeLibrary(2, 6, 5, 4)
    monkeypatch.setattr(cf, "lib", lambda: fake)
    return fake


@pytest.fixture
def graph(library):
    g = cf.PredictGraph(FakeForest(), 2, 6, 5, probabilities=True)
    yield g
    g.close()   # while the calls are still replaced


@pytest.mark.parametrize("name", ["rgb", "depth", "labels", "probabilities"])
def test_a_closed_graph_gives_no_views(library, graph, name):
    assert getattr(graph, name).size > 0
    graph.close()
    assert library.destroyed == 1
    with pytest.raises(cf.CurfilError):
        getattr(graph, name)
    graph.close()
    assert library.destroyed == 1


@pytest.mark.parametrize("name", ["rgb", "depth", "labels", "probabilities"])
def test_assignments_write_the_buffer(library, graph, name):
    buffer = library.memory[["rgb", "depth", "probabilities", "labels"].index(name)]
    view = getattr(graph, name)
    new = np.arange(view.size).reshape(view.shape) % 50
    setattr(graph, name, new)
    np.testing.assert_array_equal(buffer, new.ravel())
    if name == "rgb":
        graph.rgb += 3
    elif name == "depth":
        graph.depth += 3
    elif name == "labels":
        graph.labels += 3
    else:
        graph.probabilities += 3
    np.testing.assert_array_equal(buffer, new.ravel() + 3)
    np.testing.assert_array_equal(getattr(graph, name), new + 3)
    getattr(graph, name)[...] = 0
    assert not buffer.any()


def test_a_graph_without_probabilities_has_no_buffer_for_them(library):
    graph = cf.PredictGraph(FakeForest(), 2, 6, 5)
    assert graph.probabilities is None
    with pytest.raises(AttributeError):
        graph.probabilities = 0
    graph.close()
