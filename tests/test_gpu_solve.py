"""The solve kernel at the edges of its row classes: rows around 32 in-edges (one lane in stream order in both
orders), around 2048 (long rows and hub rows of a bin), around a hub row's rounds and chunks, bins of one row class,
and a graph large enough to run as units, whose rows above 512 in-edges are hub rows there."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = {
    "empty_and_one": [0, 1] * 700,
    "around_32": [0, 31, 32, 33, 34, 35, 36] * 90,
    "around_2048": [2047, 2048, 2049, 1, 0, 33] * 7,
    "hub_rounds": [2048 + k for k in (1, 255, 256, 257, 511, 512, 513, 2047, 2048, 2049)] + [3] * 50,
    "hub_chunks": [20480, 20481, 40959, 5000, 0, 2] * 2,
    "one_row": [1],
    "short_only": list(range(33)) * 300,
    "long_only": [33, 64, 100, 257, 700, 1500] * 40,
}


UNITS = ([511, 512, 513, 514, 767, 768, 769, 1023, 1025, 2047, 2048, 2049, 4096, 4097, 70_000]
         + [255, 256, 257, 260, 63, 64, 65, 31, 32, 33, 1, 2, 3, 4, 5, 0, 0] * 40 + [100, 0, 1] * 5) * 30


def _graph(ag, lengths, seed):
    rng = np.random.default_rng(seed)
    n = max(len(lengths), 20_000) + 7
    dst = np.repeat(np.arange(len(lengths)), lengths)
    # half of the in-neighbours among few vertices, so that out-degrees vary
    src = np.where(rng.random(dst.size) < 0.5, rng.integers(0, n, dst.size), rng.integers(0, 300, dst.size))
    return ag.Graph.from_edges(n, src.astype(np.uint32), dst.astype(np.uint32))


def _f64(g, passes):
    n, deg, out = g.num_vertices, g.in_degree().astype(np.int64), g.out_degree().astype(np.float64)
    row, nb = np.repeat(np.arange(n), deg), g.in_neighbours()
    damp, base = float(np.float32(0.85)), float(np.float32(1.0) - np.float32(0.85))
    r = np.full(n, base)
    for _ in range(passes):
        c = np.divide(r, out, out=np.zeros(n), where=out > 0)
        r = base + damp * np.bincount(row, weights=c[nb], minlength=n)
    return r / n


@pytest.mark.parametrize("name", LENGTHS)
@pytest.mark.parametrize("keep_order", [False, True])
def test_row_classes(gpu, oracle, name, keep_order):
    ag = gpu
    g = _graph(ag, LENGTHS[name], len(name))
    dg = ag.DeviceGraph(g, flags=ag.AG_UPLOAD_KEEP_ORDER if keep_order else 0)
    ref = oracle.pagerank_pull(g.in_edges_idx(), g.in_degree(), g.in_neighbours(), g.out_degree(), 20, 1e-6)
    for _ in range(2):  # the second solve starts from the hub exponents that the first one left
        r, res, _ = dg.pagerank(20, 1e-6, order=ag.AG_ORDER_EXACT)
        assert res.iterations == ref["iterations"] and np.array_equal(r, ref["ranks"])
    # FAST: at most 31 roundings in a short row, 4 in a longer one, 3 in the update, each pass's error shrinking by
    # 0.85 in the later ones
    r, _, _ = dg.pagerank(20, 0.0)
    want = _f64(g, 20)
    assert np.abs(r - want).sum() / want.sum() <= 34 * 2.0 ** -24 / (1 - 0.85)
    dg.release()


def test_units(gpu, oracle):
    ag = gpu
    lengths = UNITS + [36] * ((17_200_000 - sum(UNITS)) // 36)
    g = _graph(ag, lengths, 77)
    assert g.num_edges >= 17_000_000
    dg = ag.DeviceGraph(g)
    args = (g.in_edges_idx(), g.in_degree(), g.in_neighbours(), g.out_degree())
    ref = oracle.pagerank_pull(*args, 12, 1e-6)
    for _ in range(2):
        r, res, _ = dg.pagerank(12, 1e-6, order=ag.AG_ORDER_EXACT)
        assert res.iterations == ref["iterations"] and np.array_equal(r, ref["ranks"])
    init = np.random.default_rng(3).random(g.num_vertices).astype(np.float32)
    r, res, _ = dg.pagerank(5, 1e-6, order=ag.AG_ORDER_EXACT, init_ranks=init)
    assert np.array_equal(r, oracle.pagerank_pull(*args, 5, 1e-6, init=init)["ranks"])
    ref = oracle.pagerank_dd(g.in_edges_idx(), g.in_degree(), g.in_neighbours(), g.out_edges_idx(), g.out_degree(),
                             g.out_neighbours(), 8, 1e-3)
    r, res, _ = dg.pagerank(8, 1e-3, order=ag.AG_ORDER_EXACT, data_driven=True)
    assert res.iterations == ref["iterations"] and np.array_equal(r, ref["ranks"])
    want = _f64(g, 20)
    r, _, _ = dg.pagerank(20, 0.0)
    assert np.abs(r - want).sum() / want.sum() <= 34 * 2.0 ** -24 / (1 - 0.85)
    # 16-bit contributions: each pass's gather is off by at most 2^-9 (bfloat16), 2^-11 (binary16)
    for prec, ulp in ((ag.AG_PREC_BF16, 2.0 ** -9), (ag.AG_PREC_FP16, 2.0 ** -11)):
        r, _, _ = dg.pagerank(20, 0.0, precision=prec, switch_residual=1e-30)
        assert np.abs(r - want).sum() / want.sum() <= 1.1 * ulp / (1 - 0.85)
    dg.release()
