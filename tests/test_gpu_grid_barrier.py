"""The solve kernel's bounded grid barrier.  With AG_GRID_SPINS=0 the first CTA to wait gives up at once; every other
CTA then stops too, the call reports AG_ERR_DEVICE_WAIT, and the same graph is usable again (nothing hangs or faults).
With a few polls a barrier may open or not: the call gives the right bits or reports, and the next one is right."""
import numpy as np
import pytest

from test_gpu_solve import LENGTHS, UNITS, _graph

pytestmark = pytest.mark.gpu


def _lengths(plan):
    rows = LENGTHS["hub_rounds"] + LENGTHS["hub_chunks"] + LENGTHS["around_32"]
    if plan == "units":
        rows = UNITS + [36] * ((17_200_000 - sum(UNITS)) // 36)
    return rows


@pytest.mark.parametrize("launch", ["one", "stream"])
@pytest.mark.parametrize("plan", ["bins", "units"])
def test_solve_gives_up_and_recovers(gpu, oracle, monkeypatch, plan, launch):
    ag = gpu
    if launch == "stream":
        monkeypatch.setenv("AG_LAUNCH_MODE", "stream")
    g = _graph(ag, _lengths(plan), 41)
    ref = oracle.pagerank_pull(g.in_edges_idx(), g.in_degree(), g.in_neighbours(), g.out_degree(), 6, 1e-6)
    dg = ag.DeviceGraph(g)
    for spins in ("0", "0", "20", "200", "2000"):
        monkeypatch.setenv("AG_GRID_SPINS", spins)
        dg.launch(6, 1e-6, order=ag.AG_ORDER_EXACT)
        try:
            r, _, _ = dg.fetch()
            assert spins != "0" and np.array_equal(r, ref["ranks"])
        except ag.AGError as err:
            assert err.status == ag.AG_ERR_DEVICE_WAIT
            with pytest.raises(ag.AGError) as again:  # there is no result left to fetch
                dg.fetch()
            assert again.value.status == ag.AG_ERR_INVALID_ARG
        monkeypatch.delenv("AG_GRID_SPINS")
        r, res, _ = dg.pagerank(6, 1e-6, order=ag.AG_ORDER_EXACT)
        assert res.iterations == ref["iterations"] and np.array_equal(r, ref["ranks"])
    dg.release()


def test_two_launches_before_a_fetch(gpu, oracle, monkeypatch):
    ag = gpu
    g = _graph(ag, _lengths("bins"), 42)
    ref = oracle.pagerank_pull(g.in_edges_idx(), g.in_degree(), g.in_neighbours(), g.out_degree(), 6, 1e-6)
    dg = ag.DeviceGraph(g)
    monkeypatch.setenv("AG_GRID_SPINS", "0")
    dg.launch(6, 1e-6, order=ag.AG_ORDER_EXACT)
    monkeypatch.delenv("AG_GRID_SPINS")
    with pytest.raises(ag.AGError) as err:  # the launch reports it, or (still running then) the fetch
        dg.launch(6, 1e-6, order=ag.AG_ORDER_EXACT)
        dg.fetch()
    assert err.value.status == ag.AG_ERR_DEVICE_WAIT
    r, _, _ = dg.pagerank(6, 1e-6, order=ag.AG_ORDER_EXACT)
    assert np.array_equal(r, ref["ranks"])
    dg.release()


@pytest.mark.parametrize("plan", ["bins", "units"])
@pytest.mark.parametrize("exact", [0, 2])
def test_product_gives_up_and_recovers(gpu, monkeypatch, plan, exact):
    """A relabelled graph's product waits at a barrier: the host form reports it, the device form through
    ag_synchronize or the graph's next call."""
    import ctypes as C

    import torch

    ag = gpu
    g = _graph(ag, _lengths(plan), 43)
    n = g.num_vertices
    dg = ag.DeviceGraph(g)
    xh = np.random.default_rng(1).random(n, dtype=np.float32)
    want = dg.spmv(xh, exact).view(np.uint32)
    x, y = torch.from_numpy(xh).cuda(), torch.zeros(n, device="cuda")
    torch.cuda.synchronize()

    def product():
        return ag.lib.ag_spmv_pull_device(dg.h, x.data_ptr(), y.data_ptr(), exact)

    monkeypatch.setenv("AG_GRID_SPINS", "0")
    with pytest.raises(ag.AGError) as err:
        dg.spmv(xh, exact)
    assert err.value.status == ag.AG_ERR_DEVICE_WAIT
    assert product() == ag.AG_OK
    assert ag.lib.ag_synchronize(C.c_double(60.0)) == ag.AG_ERR_DEVICE_WAIT
    assert ag.lib.ag_synchronize(C.c_double(60.0)) == ag.AG_OK  # reported once
    monkeypatch.delenv("AG_GRID_SPINS")
    assert product() == ag.AG_OK and ag.lib.ag_synchronize(C.c_double(60.0)) == ag.AG_OK
    assert np.array_equal(y.cpu().numpy().view(np.uint32), want)
    monkeypatch.setenv("AG_GRID_SPINS", "0")
    assert product() == ag.AG_OK
    torch.cuda.synchronize()
    monkeypatch.delenv("AG_GRID_SPINS")
    assert product() == ag.AG_ERR_DEVICE_WAIT
    assert np.array_equal(dg.spmv(xh, exact).view(np.uint32), want)
    dg.release()


def test_csr_product_reports(gpu, monkeypatch):
    import ctypes as C

    ag = gpu
    g = _graph(ag, _lengths("bins"), 44)
    args = ag.default_arguments(2, 1e-4)
    out = C.POINTER(ag.SPMVStats)()
    monkeypatch.setenv("AG_GRID_SPINS", "0")
    assert ag.lib.ag_spmv_pull_ex(C.byref(args), g.ptr, 1, C.byref(out)) == ag.AG_ERR_DEVICE_WAIT
    monkeypatch.delenv("AG_GRID_SPINS")
    assert ag.lib.ag_spmv_pull_ex(C.byref(args), g.ptr, 1, C.byref(out)) == ag.AG_OK
    ag.lib.freeSPMVStats(out)


def test_product_behind_a_solve_that_gives_up(gpu, monkeypatch):
    """A product without a barrier of its own (caller's order, bins) does not run on a graph that was given up."""
    import ctypes as C

    import torch

    ag = gpu
    g = _graph(ag, _lengths("bins"), 45)
    n = g.num_vertices
    dg = ag.DeviceGraph(g, flags=ag.AG_UPLOAD_KEEP_ORDER)
    xh = np.random.default_rng(2).random(n, dtype=np.float32)
    x, y = torch.from_numpy(xh).cuda(), torch.zeros(n, device="cuda")
    torch.cuda.synchronize()
    monkeypatch.setenv("AG_GRID_SPINS", "0")
    dg.launch(6, 1e-6, order=ag.AG_ORDER_EXACT)
    monkeypatch.delenv("AG_GRID_SPINS")
    st = ag.lib.ag_spmv_pull_device(dg.h, x.data_ptr(), y.data_ptr(), ag.AG_SPMV_EXACT)
    if st == ag.AG_OK:  # queued before the host could see it
        st = ag.lib.ag_synchronize(C.c_double(60.0))
    assert st == ag.AG_ERR_DEVICE_WAIT and not y.any()
    want = ag.DeviceGraph(g, flags=ag.AG_UPLOAD_KEEP_ORDER).spmv(xh, ag.AG_SPMV_EXACT)
    assert np.array_equal(dg.spmv(xh, ag.AG_SPMV_EXACT), want)
    dg.release()


@pytest.mark.parametrize("order", [0, 1])
def test_union_gives_up_and_recovers(gpu, monkeypatch, order):
    ag = gpu
    mg = ag.MultiGraph([_graph(ag, LENGTHS["hub_rounds"], 46), ag.Graph.rmat(10, 8, seed=3), _graph(ag, [40] * 900, 47)])
    want, info = mg.pagerank(12, 1e-6, order)
    for spins in ("0", "0", "50", "500"):
        monkeypatch.setenv("AG_GRID_SPINS", spins)
        try:
            parts, _ = mg.pagerank(12, 1e-6, order)
            assert spins != "0" and all(np.array_equal(a, b) for a, b in zip(parts, want))
        except ag.AGError as err:
            assert err.status == ag.AG_ERR_DEVICE_WAIT
        monkeypatch.delenv("AG_GRID_SPINS")
        parts, again = mg.pagerank(12, 1e-6, order)
        assert all(np.array_equal(a, b) for a, b in zip(parts, want)) and np.array_equal(again["passes"], info["passes"])
    mg.release()
