"""Batched PPR on graphs whose rows get a warp each whatever the number of columns: no row above 512 in-edges, some above
64, and no more rows than resident warps; and just outside that rule."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 7, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("n,longest", [(600, 512), (600, 513), (33, 65), (33, 64), (4736, 300), (4737, 300)])
def test_small_graphs(gpu, oracle, n, longest, k):
    ag = gpu
    rng = np.random.default_rng(n + k)
    src = np.concatenate([rng.integers(0, n, 4 * n), rng.integers(0, n, longest)]).astype(np.uint32)
    dst = np.concatenate([rng.integers(1, n, 4 * n), np.zeros(longest, np.int64)]).astype(np.uint32)
    g = ag.Graph.from_edges(n, src, dst)
    assert g.in_degree().max() == longest
    sources = rng.choice(n, min(k, n), replace=False).astype(np.uint32)
    r, res = ag.DeviceGraph(g).ppr(sources, iterations=12, epsilon=1e-6)
    ro, _, passes = oracle.ppr(g.in_edges_idx(), g.in_degree(), g.in_neighbours(), g.out_degree(), sources,
                               iterations=12, epsilon=1e-6)
    assert res.passes == passes and np.array_equal(r, ro)
