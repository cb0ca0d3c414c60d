"""What a fetch does to the caller's memory when its bounded wait runs out, and that it stays bounded."""
import ctypes as C
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned", [True, False])
def test_timeout_leaves_the_buffer_alone(gpu, oracle, monkeypatch, pinned):
    """ag_pagerank_fetch that timed out writes nothing into `ranks`, neither then nor when the solve ends; a second
    fetch delivers."""
    import torch

    ag = gpu
    g = ag.Graph.rmat(18, 16, seed=5)
    ref = oracle.pagerank_pull(g.in_edges_idx(), g.in_degree(), g.in_neighbours(), g.out_degree(), 400, 0.0)
    dg = ag.DeviceGraph(g)
    dg.pagerank(2, 1e-6, order=ag.AG_ORDER_EXACT)
    ranks = torch.full((g.num_vertices,), -7.0, pin_memory=pinned)
    ptr, res = C.cast(ranks.data_ptr(), ag.f32p), ag.PRResult()

    def fetch():
        return ag.lib.ag_pagerank_fetch(dg.h, ptr, C.byref(res), None, None, None, 0)

    dg.launch(400, 0.0, order=ag.AG_ORDER_EXACT)
    monkeypatch.setenv("AG_WAIT_TIMEOUT_S", "1e-7")
    assert fetch() == ag.AG_ERR_TIMEOUT
    monkeypatch.delenv("AG_WAIT_TIMEOUT_S")
    assert ag.lib.ag_synchronize(C.c_double(120.0)) == ag.AG_OK
    assert (ranks.numpy() == -7.0).all()
    assert fetch() == ag.AG_OK and res.passes == ref["passes"]
    assert np.array_equal(ranks.numpy(), ref["ranks"])
    dg.release()


def test_fetch_beside_another_is_bounded(gpu, oracle, monkeypatch):
    """While another thread's fetch holds the staging, a fetch copies directly; its wait for the solve still has the
    limit that the caller set."""
    ag = gpu
    ga, gb = ag.Graph.rmat(20, 16, seed=6), ag.Graph.rmat(12, 16, seed=7)
    ref = oracle.pagerank_pull(gb.in_edges_idx(), gb.in_degree(), gb.in_neighbours(), gb.out_degree(), 20, 1e-6)
    da, db = ag.DeviceGraph(ga), ag.DeviceGraph(gb)
    got = []
    da.launch(4000, 0.0, order=ag.AG_ORDER_EXACT)  # some 0.3 s
    thread = threading.Thread(target=lambda: got.append(da.fetch()[1].passes))
    thread.start()
    time.sleep(0.05)
    db.launch(20, 1e-6, order=ag.AG_ORDER_EXACT)
    monkeypatch.setenv("AG_WAIT_TIMEOUT_S", "1e-7")
    with pytest.raises(ag.AGError) as err:
        db.fetch()
    assert err.value.status == ag.AG_ERR_TIMEOUT
    monkeypatch.delenv("AG_WAIT_TIMEOUT_S")
    thread.join()
    assert got == [4000]
    r, res, _ = db.fetch()
    assert res.iterations == ref["iterations"] and np.array_equal(r, ref["ranks"])
    da.release()
    db.release()


def test_device_memory_as_the_host_destination_is_refused(gpu, oracle):
    """The host reads and writes staged destinations itself: a device pointer is an error, not a crash."""
    import torch

    ag = gpu
    g = ag.Graph.rmat(10, 8)
    dg = ag.DeviceGraph(g)
    buf = torch.zeros(g.num_vertices, device="cuda")
    ptr = C.cast(buf.data_ptr(), ag.f32p)
    dg.launch(5, 1e-6)
    assert ag.lib.ag_pagerank_fetch(dg.h, ptr, None, None, None, None, 0) == ag.AG_ERR_INVALID_ARG
    x = np.ones(g.num_vertices, np.float32)
    assert ag.lib.ag_spmv_pull(dg.h, x.ctypes.data_as(ag.f32p), ptr, 0) == ag.AG_ERR_INVALID_ARG
    assert ag.lib.ag_synchronize(C.c_double(60.0)) == ag.AG_OK and not buf.any()
    want = oracle.spmv_pull(g.in_edges_idx(), g.in_degree(), g.in_neighbours(), np.ones(g.num_edges, np.float32), x)
    assert np.array_equal(dg.spmv(x, ag.AG_SPMV_UNIT | ag.AG_SPMV_EXACT), want)
    dg.release()
