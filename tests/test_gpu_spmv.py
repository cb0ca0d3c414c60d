"""The sparse product at the edges of its row classes, in both plans: bins (rows around 32 and 2048 in-edges, hub
rounds and chunks) and units (rows around 512, a graph of 17 million in-edges).  Vectors of one sign, of both (hub
sums that leave their binade downwards, or pass zero), with zeros of either sign, and with infinities and NaN."""
import numpy as np
import pytest

from test_gpu_solve import LENGTHS, UNITS

pytestmark = pytest.mark.gpu


def _graph(ag, lengths, seed):
    rng = np.random.default_rng(seed)
    n = max(len(lengths), 20_000) + 7
    dst = np.repeat(np.arange(len(lengths)), lengths)
    src = np.where(rng.random(dst.size) < 0.5, rng.integers(0, n, dst.size), rng.integers(0, 300, dst.size))
    w = rng.random(dst.size, dtype=np.float32)
    return ag.Graph.from_edges(n, src.astype(np.uint32), dst.astype(np.uint32), w)


def _vectors(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.random(n, dtype=np.float32)
    zeros = x.copy()
    zeros[::2] = 0.0
    zeros[1::4] = -0.0
    few = x.copy()
    few[::701] *= -1.0
    special = x - np.float32(0.5)
    special[5] = np.inf
    special[n // 2] = np.nan
    return {"positive": x, "both": x - np.float32(0.5), "few": few, "zeros": zeros, "none": np.full(n, -0.0, np.float32),
            "special": special}


def _check(ag, oracle, g, dg, x, mode, w):
    want = oracle.spmv_pull(g.in_edges_idx(), g.in_degree(), g.in_neighbours(), w, x)
    y = dg.spmv(x, mode=mode | ag.AG_SPMV_EXACT)
    same = (y.view(np.uint32) == want.view(np.uint32)) | (np.isnan(y) & np.isnan(want))
    assert same.all()
    y = dg.spmv(x, mode=mode)
    finite = np.isfinite(want)
    assert np.array_equal(np.isnan(y), np.isnan(want)) and np.array_equal(y[np.isinf(want)], want[np.isinf(want)])
    # FAST: a product's rounding, at most 31 adds in a short row, 3 and the last in a longer one
    deg, nb = g.in_degree().astype(np.int64), g.in_neighbours()
    row = np.repeat(np.arange(g.num_vertices), deg)
    with np.errstate(invalid="ignore"):
        t = w.astype(np.float64) * x.astype(np.float64)[nb]
    exact = np.bincount(row, weights=np.where(np.isfinite(t), t, 0.0), minlength=g.num_vertices)
    size = np.bincount(row, weights=np.where(np.isfinite(t), np.abs(t), 0.0), minlength=g.num_vertices)
    assert (np.abs(y[finite] - exact[finite]) <= 33 * 2.0 ** -24 * size[finite]).all()


@pytest.mark.parametrize("name", LENGTHS)
@pytest.mark.parametrize("keep_order", [False, True])
def test_row_classes(gpu, oracle, name, keep_order):
    ag = gpu
    g = _graph(ag, LENGTHS[name], len(name))
    dg = ag.DeviceGraph(g, weights=True, flags=ag.AG_UPLOAD_KEEP_ORDER if keep_order else 0)
    w = g.in_weights()
    for x in _vectors(g.num_vertices, 5).values():
        _check(ag, oracle, g, dg, x, ag.AG_SPMV_GRAPH_WEIGHTS, w)
    _check(ag, oracle, g, dg, x, ag.AG_SPMV_UNIT, np.ones_like(w))
    dg.release()


def test_units(gpu, oracle):
    ag = gpu
    lengths = UNITS + [36] * ((17_200_000 - sum(UNITS)) // 36)
    g = _graph(ag, lengths, 78)
    assert g.num_edges >= 17_000_000
    dg = ag.DeviceGraph(g, weights=True)
    for x in _vectors(g.num_vertices, 6).values():
        _check(ag, oracle, g, dg, x, ag.AG_SPMV_GRAPH_WEIGHTS, g.in_weights())
    # without weights on the device every one is 0.0001
    dg.release()
    dg = ag.DeviceGraph(g)
    _check(ag, oracle, g, dg, _vectors(g.num_vertices, 7)["both"], ag.AG_SPMV_GRAPH_WEIGHTS,
           np.full(g.num_edges, 0.0001, np.float32))
    dg.release()


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("keep_order", [False, True])
def test_device_vectors(gpu, offset, keep_order):
    """Vectors at any 4-byte boundary, solves in between, and a product in place (relabelled graphs)."""
    import torch

    ag = gpu
    g = _graph(ag, LENGTHS["hub_rounds"] + LENGTHS["around_32"], 9)
    n = g.num_vertices
    dg = ag.DeviceGraph(g, weights=True, flags=ag.AG_UPLOAD_KEEP_ORDER if keep_order else 0)
    xh = _vectors(n, 8)["both"]
    mode = ag.AG_SPMV_GRAPH_WEIGHTS | ag.AG_SPMV_EXACT
    want = dg.spmv(xh, mode)
    ranks = dg.pagerank(10, 1e-6, order=ag.AG_ORDER_EXACT)[0]
    x = torch.empty(n + 1, device="cuda")[offset:offset + n]
    x.copy_(torch.from_numpy(xh))
    y = x if not keep_order else torch.empty(n + 1, device="cuda")[offset:offset + n]
    torch.cuda.synchronize()
    ag.check(ag.lib.ag_spmv_pull_device(dg.h, x.data_ptr(), y.data_ptr(), mode), "ag_spmv_pull_device")
    again = dg.pagerank(10, 1e-6, order=ag.AG_ORDER_EXACT)[0]
    assert np.array_equal(y.cpu().numpy().view(np.uint32), want.view(np.uint32))
    assert np.array_equal(ranks, again)
    dg.release()
