"""Both sides of the limits by which an upload chooses its plan, at sizes that tests can have (the limits are overridden
in the environment): unions on the solve kernel and on the pull kernel's loop, graphs of a few rows as units, and the
work lists' split rows in the forms that still run on them."""
import ctypes as C
import datetime
import socket

import numpy as np
import pytest

from test_gpu_solve import LENGTHS, _f64, _graph

pytestmark = pytest.mark.gpu


def _star(ag, leaves):
    """A row of `leaves` in-edges whose graph is done after a few passes."""
    return ag.Graph.from_edges(leaves + 1, np.arange(1, leaves + 1, dtype=np.uint32), np.zeros(leaves, np.uint32))


def _union(ag):
    return [_star(ag, 5000), _graph(ag, LENGTHS["hub_rounds"], 3), ag.Graph.from_edges(3, [], []),
            ag.Graph.rmat(11, 16, seed=4), _graph(ag, LENGTHS["hub_chunks"] + LENGTHS["around_32"], 5),
            ag.Graph.from_edges(5, [0, 1, 2], [1, 2, 3]), _star(ag, 2049)]


def _bytes(ag, mg):
    info = ag.GraphInfo()
    ag.check(ag.lib.ag_graph_get_info(mg.h, C.byref(info)), "ag_graph_get_info")
    return info.device_bytes


@pytest.mark.parametrize("order", [0, 1])
def test_union_on_either_side(gpu, oracle, monkeypatch, order):
    ag = gpu
    gs = _union(ag)
    refs = [oracle.pagerank_pull(g.in_edges_idx(), g.in_degree(), g.in_neighbours(), g.out_degree(), 60, 1e-5)
            for g in gs]
    x = np.random.default_rng(2).random(sum(g.num_vertices for g in gs), dtype=np.float32) - np.float32(0.5)
    at = np.cumsum([0] + [g.num_vertices for g in gs])
    ys = np.concatenate([oracle.gather(g.in_edges_idx(), g.in_degree(), g.in_neighbours(), x[at[i]:at[i + 1]])
                         for i, g in enumerate(gs)])
    # FAST sums are closer to 64 bits than the oracle's binary32 chain of 5000 adds is
    r64 = [_f64(g, 60) for g in gs]
    row = np.concatenate([at[i] + np.repeat(np.arange(g.num_vertices), g.in_degree()) for i, g in enumerate(gs)])
    xs = np.concatenate([x[at[i] + g.in_neighbours().astype(np.int64)] for i, g in enumerate(gs)]).astype(np.float64)
    y64 = np.bincount(row, weights=xs, minlength=x.size)
    sizes = []
    for limit in ("0", "4294967295"):
        monkeypatch.setenv("AG_UNION_MAX_EDGES", limit)
        mg = ag.MultiGraph(gs)
        sizes.append(_bytes(ag, mg))
        for _ in range(2):  # the second solve starts from what the first left
            parts, info = mg.pagerank(60, 1e-5, order)
            for i, ref in enumerate(refs):
                if order == ag.AG_ORDER_EXACT:
                    assert info["iterations"][i] == ref["iterations"] and info["passes"][i] == ref["passes"], i
                    assert np.array_equal(parts[i], ref["ranks"]), i
                else:
                    assert np.abs(parts[i] - r64[i]).sum() <= 1e-5 * r64[i].sum()
            y = np.empty_like(x)
            mode = ag.AG_SPMV_UNIT | (ag.AG_SPMV_EXACT if order == ag.AG_ORDER_EXACT else 0)
            ag.check(ag.lib.ag_spmv_pull(mg.h, x.ctypes.data_as(ag.f32p), y.ctypes.data_as(ag.f32p), mode), "spmv")
            if order == ag.AG_ORDER_EXACT:
                assert np.array_equal(y, ys)
            else:
                assert np.abs(y - y64).sum() <= 1e-5 * np.abs(xs).sum()
        mg.release()
    assert sizes[0] < sizes[1]  # without and with the solve kernel's plan


def _units_graph(ag, n):
    if isinstance(n, str):
        return _graph(ag, LENGTHS[n], len(n))
    rng = np.random.default_rng(n)
    m = 9 * n
    dst = np.minimum(rng.integers(0, n, m), rng.integers(0, n, m))  # longer rows first
    dst[: m // 4] = n // 2  # and one of a quarter of the edges
    return ag.Graph.from_edges(n, rng.integers(0, n, m).astype(np.uint32), dst.astype(np.uint32),
                               rng.random(m, dtype=np.float32))


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 257, 2047, 2048, 2049, 4100, "empty_and_one", "around_2048",
                               "hub_rounds", "hub_chunks", "short_only"])
@pytest.mark.parametrize("keep_order", [False, True])
def test_small_units(gpu, oracle, monkeypatch, n, keep_order):
    ag = gpu
    monkeypatch.setenv("AG_UNIT_MIN_EDGES", "0")
    g = _units_graph(ag, n)
    args = (g.in_edges_idx(), g.in_degree(), g.in_neighbours(), g.out_degree())
    flags = ag.AG_UPLOAD_KEEP_ORDER if keep_order else 0
    dg = ag.DeviceGraph(g, weights=True, flags=flags)
    ref = oracle.pagerank_pull(*args, 15, 1e-6)
    for _ in range(2):
        r, res, _ = dg.pagerank(15, 1e-6, order=ag.AG_ORDER_EXACT)
        assert res.iterations == ref["iterations"] and np.array_equal(r, ref["ranks"])
    init = np.random.default_rng(3).random(g.num_vertices).astype(np.float32)
    r, _, _ = dg.pagerank(5, 1e-6, order=ag.AG_ORDER_EXACT, init_ranks=init)
    assert np.array_equal(r, oracle.pagerank_pull(*args, 5, 1e-6, init=init)["ranks"])
    ref = oracle.pagerank_dd(g.in_edges_idx(), g.in_degree(), g.in_neighbours(), g.out_edges_idx(), g.out_degree(),
                             g.out_neighbours(), 8, 1e-3)
    r, res, _ = dg.pagerank(8, 1e-3, order=ag.AG_ORDER_EXACT, data_driven=True)
    assert res.iterations == ref["iterations"] and np.array_equal(r, ref["ranks"])
    # FAST: at most 31 roundings in a short row, 4 in a longer one, 3 in the update
    want = _f64(g, 15)
    r, _, _ = dg.pagerank(15, 0.0)
    assert np.abs(r - want).sum() / want.sum() <= 34 * 2.0 ** -24 / (1 - 0.85)
    x = np.random.default_rng(4).random(g.num_vertices, dtype=np.float32) - np.float32(0.5)
    y = dg.spmv(x, ag.AG_SPMV_GRAPH_WEIGHTS | ag.AG_SPMV_EXACT)
    assert np.array_equal(y, oracle.spmv_pull(g.in_edges_idx(), g.in_degree(), g.in_neighbours(), g.in_weights(), x))
    dg.release()


@pytest.mark.parametrize("units", [False, True])
def test_hub_rounds_that_leave_their_binade(gpu, oracle, monkeypatch, units):
    """EXACT order: every round of a hub row doubles its sum (more rounds to keep than there is room for), and warm
    starts whose second pass is orders of magnitude away from the first (no round finds its map)."""
    ag = gpu
    monkeypatch.setenv("AG_UNIT_MIN_EDGES", "0" if units else "4294967295")
    lengths = [2049, 4097, 12_288, 600, 40_000]
    n = 40_007
    rng = np.random.default_rng(8)
    dst = np.repeat(np.arange(len(lengths)), lengths)
    src = np.concatenate([np.arange(m) for m in lengths])  # in vertex order
    extra = rng.integers(0, n, (2, 90_000))
    g = ag.Graph.from_edges(n, np.concatenate([src, extra[0]]).astype(np.uint32),
                            np.concatenate([dst, extra[1]]).astype(np.uint32))
    dg = ag.DeviceGraph(g)
    args = (g.in_edges_idx(), g.in_degree(), g.in_neighbours())
    for step in (256, 64, 1024):
        x = np.ldexp(1.0 + rng.random(n), np.minimum(np.arange(n) // step, 90)).astype(np.float32)
        y = dg.spmv(x, ag.AG_SPMV_UNIT | ag.AG_SPMV_EXACT)
        assert np.array_equal(y, oracle.gather(*args, x)), step
    for few, high, low in ((0.01, 1e6, 1e-3), (0.5, 1e-30, 1e20), (0.001, 3e30, 0.0)):
        init = np.where(rng.random(n) < few, high, low).astype(np.float32)
        r, _, _ = dg.pagerank(6, 1e-6, order=ag.AG_ORDER_EXACT, init_ranks=init)
        assert np.array_equal(r, oracle.pagerank_pull(*args, g.out_degree(), 6, 1e-6, init=init)["ranks"])
    dg.release()


@pytest.mark.parametrize("name", LENGTHS)
def test_data_driven_bins(gpu, oracle, name):
    """Tags of every row class of a bin: the oracle's worklists in EXACT order; and with epsilon 0, when every change is
    passed on, the plain solve's ranks bit for bit in either order."""
    ag = gpu
    g = _graph(ag, LENGTHS[name], len(name))
    dg = ag.DeviceGraph(g)
    ref = oracle.pagerank_dd(g.in_edges_idx(), g.in_degree(), g.in_neighbours(), g.out_edges_idx(), g.out_degree(),
                             g.out_neighbours(), 8, 1e-3)
    r, res, hist = dg.pagerank(8, 1e-3, order=ag.AG_ORDER_EXACT, data_driven=True, history=8)
    assert res.iterations == ref["iterations"] and np.array_equal(r, ref["ranks"])
    assert np.array_equal(hist["active"], ref["active"])
    for order in (ag.AG_ORDER_FAST, ag.AG_ORDER_EXACT):
        assert np.array_equal(dg.pagerank(6, 0.0, order=order, data_driven=True)[0], dg.pagerank(6, 0.0, order=order)[0])
    dg.release()


@pytest.mark.parametrize("tiles", [(256, 2048), (64, 128), (32, 32)])
def test_split_rows_of_the_work_list(gpu, oracle, tiles):
    """A row partition's EXACT passes, split into small chunks: the oracle's ranks bit for bit; and the pull-push form,
    whose seed and inner product run on the same list."""
    ag = gpu
    import torch
    import torch.distributed as dist

    from accelgraph_b200 import distributed as agd
    g = ag.Graph.rmat(13, 16, seed=21)
    assert g.in_degree().max() > 4 * tiles[0]
    ref = oracle.pagerank_pull(g.in_edges_idx(), g.in_degree(), g.in_neighbours(), g.out_degree(), 60, 1e-4)
    s = socket.socket()
    s.bind(("127.0.0.1", 0))
    port = s.getsockname()[1]
    s.close()
    torch.cuda.set_device(0)
    dist.init_process_group("nccl", init_method=f"tcp://127.0.0.1:{port}", rank=0, world_size=1,
                            timeout=datetime.timedelta(seconds=120))
    try:
        part = agd.RowPartition(g)
        try:
            shape = ag.TileConfig(*tiles, 0, 65536)
            ag.check(ag.lib.ag_graph_set_tiles(part.h, C.byref(shape)), "ag_graph_set_tiles")
            for _ in range(2):
                its, passes, _, _ = part.solve(60, 1e-4, True)
                ranks, _ = part.ranks()
                assert (its, passes) == (ref["iterations"], ref["passes"])
                assert np.array_equal(ranks.view(np.uint32), ref["ranks"].view(np.uint32))
        finally:
            part.release()
    finally:
        dist.destroy_process_group()
    g = ag.Graph.rmat(12, 8, seed=78)
    want = oracle.pagerank_residual(True, g.in_edges_idx(), g.in_degree(), g.in_neighbours(), g.out_edges_idx(),
                                    g.out_degree(), g.out_neighbours(), 300, 1e-6)["ranks"].astype(np.float64)
    dg = ag.DeviceGraph(g)
    dg.set_tiles(*tiles, 0, 65536)
    r, _, _ = dg.pagerank(300, 1e-6, data_driven=True, direction=ag.AG_DIR_PULL_PUSH)
    assert np.abs(r - want).sum() <= 1e-4 * want.sum()
    dg.release()
