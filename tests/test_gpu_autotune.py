"""The autotuner leaves alone what its timing does not see: a whole graph's solve does not read the work list, so the
list's shape, which the integer, push and feature forms run on, is the caller's, with and without a cache file."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_work_list_is_left_alone(gpu, oracle, tmp_path, monkeypatch):
    ag = gpu
    monkeypatch.setenv("AG_TUNE_CACHE", str(tmp_path / "tune.txt"))
    g = ag.Graph.rmat(13, 16, seed=4)
    ref = oracle.pagerank_pull(g.in_edges_idx(), g.in_degree(), g.in_neighbours(), g.out_degree(), 30, 1e-6)
    hot = []
    for shape in ((64, 512), (32, 96)):  # the second handle is served from the cache file
        dg = ag.DeviceGraph(g)
        dg.set_tiles(*shape, 8192, 65536)
        tasks = dg.tasks()
        best, us = dg.autotune(passes=4)
        assert us > 0 and (best.task_edges, best.hub_chunk) == shape
        assert np.array_equal(dg.tasks(), tasks)
        hot.append((best.hot_entries, best.warm_entries, us))
        r, res, _ = dg.pagerank(30, 1e-6, order=ag.AG_ORDER_EXACT)
        assert res.iterations == ref["iterations"] and np.array_equal(r, ref["ranks"])
        dg.release()
    assert hot[0][:2] == hot[1][:2] and abs(hot[0][2] - hot[1][2]) <= 5e-4
