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
