"""The split-search time of the benchmark's roofline counts every kernel that evaluates candidates."""
import bench


def test_split_search_time_counts_all_its_kernels():
    ms = {"level_eval": (2.0, 4), "stage_bins": (5.0, 3), "stage_general": (1.0, 3), "route_flags": (9.0, 1)}
    total, kernels = bench.split_search_times(lambda name: ms.get(name, (0.0, 0)))
    assert total == 8.0
    assert {k: (v["ms"], v["launches"]) for k, v in kernels.items()} == {k: ms[k] for k in bench.SEARCH_KERNELS}
    assert abs(sum(v["share"] for v in kernels.values()) - 1.0) < 1e-12
    assert bench.split_search_times(lambda name: (0.0, 0))[0] == 0
