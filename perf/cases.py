"""Performance cases of the library: what its callers run, from the smallest solve to the largest.

Graphs are made on the GPU from the seed (R-MAT with the Graph500 quadrants, or Erdos-Renyi) and go through the
library's own builder, as a program with an edge list in device memory does.  R-MAT ids are taken modulo the vertex
count, so that the count can be any number.  Kinds of case:

  solve   DeviceGraph.pagerank on a graph that is already on the device; the ranks come back to the host
  call    ag_pagerank_pull_ex on a host CSR (page-locked): upload, solve and readback in one call, as the reference's
          pageRankPullGraphCSR is used
  build   edge list in device memory -> DeviceGraph -> PageRank -> ranks
  spmv    ag_spmv_pull_device: y = A x on device vectors, weighted or not
  spmv_host  DeviceGraph.spmv on numpy vectors
  ppr     DeviceGraph.ppr: personalized PageRank of k sources together
  multi   MultiGraph.pagerank: many small graphs in one launch
"""
import ctypes as C
import math

import numpy as np
import torch

import accelgraph_b200 as ag

A, B, C_ = 0.57, 0.19, 0.19
DAMP = float(np.float32(0.85))
BASE = float(np.float32(1.0) - np.float32(0.85))


def listed():
    return [
        # the smallest call: a solve whose cost is launches and latency
        {"name": "solve_n1k_exact", "kind": "solve", "graph": "rmat", "n": 1024, "ef": 16, "order": "exact",
         "iterations": 20, "epsilon": 1e-4, "precision": "fp32"},
        # the reference CLI's defaults (20 iterations, 1e-4) on a graph of ordinary size
        {"name": "solve_n65k_exact", "kind": "solve", "graph": "rmat", "n": 65536, "ef": 16, "order": "exact",
         "iterations": 20, "epsilon": 1e-4, "precision": "fp32"},
        # an odd vertex count, uniform degrees, the Python default order
        {"name": "solve_er_odd_fast", "kind": "solve", "graph": "er", "n": 1200007, "ef": 9, "order": "fast",
         "iterations": 50, "epsilon": 1e-6, "precision": "fp32"},
        # R-MAT scale 22 and 24 in the reference's bits, 100 passes
        {"name": "solve_n4m_exact", "kind": "solve", "graph": "rmat", "n": 4194304, "ef": 16, "order": "exact",
         "iterations": 100, "epsilon": 1e-6, "precision": "fp32"},
        {"name": "solve_n16m_exact", "kind": "solve", "graph": "rmat", "n": 16777216, "ef": 16, "order": "exact",
         "iterations": 100, "epsilon": 1e-6, "precision": "fp32"},
        # the 16-bit storage option
        {"name": "solve_n1m_bf16", "kind": "solve", "graph": "rmat", "n": 1048576, "ef": 16, "order": "exact",
         "iterations": 100, "epsilon": 1e-6, "precision": "bf16"},
        # the drop-in call of a reference program: host CSR in, host ranks out
        {"name": "call_n1m_exact", "kind": "call", "graph": "rmat", "n": 1048576, "ef": 16, "order": "exact",
         "iterations": 20, "epsilon": 1e-4},
        # a new graph every time: edge list to ranks
        {"name": "build_n700k_fast", "kind": "build", "graph": "rmat", "n": 700001, "ef": 12, "order": "fast",
         "iterations": 20, "epsilon": 1e-4},
        # weighted product on device vectors, the size of an iterative solver's matrix
        {"name": "spmv_n4m_weighted", "kind": "spmv", "graph": "rmat", "n": 4194304, "ef": 16, "order": "fast",
         "weighted": True},
        # a small product on host vectors
        {"name": "spmv_host_n5k", "kind": "spmv_host", "graph": "er", "n": 5003, "ef": 14, "order": "exact",
         "weighted": True},
        # recommendations: a batch of personalized solves that does not fill the 64 columns
        {"name": "ppr_n500k_k40", "kind": "ppr", "graph": "er", "n": 500009, "ef": 8, "k": 40, "iterations": 20,
         "epsilon": 1e-6},
        # many small graphs (one per community, tenant or molecule batch) at once
        {"name": "multi_48", "kind": "multi", "graph": "rmat", "count": 48, "n": 12000, "ef": 10, "order": "fast",
         "iterations": 50, "epsilon": 1e-6},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "call", "build", "spmv", "spmv_host", "ppr", "multi"])
    graph = rng.choice(["rmat", "rmat", "er"])
    order = rng.choice(["exact", "fast"])
    ef = rng.randint(4, 20)
    if kind == "solve":
        return {"kind": kind, "graph": graph, "n": _log_int(rng, 900, 6000000), "ef": ef, "order": order,
                "iterations": rng.choice([10, 20, 50, 100]), "epsilon": rng.choice([1e-4, 1e-6]),
                "precision": "fp32" if order == "fast" else rng.choice(["fp32", "fp32", "bf16"])}
    if kind in ("call", "build"):
        return {"kind": kind, "graph": graph, "n": _log_int(rng, 5000, 1500000), "ef": ef, "order": order,
                "iterations": rng.choice([10, 20, 50]), "epsilon": 1e-4}
    if kind == "spmv":
        return {"kind": kind, "graph": graph, "n": _log_int(rng, 5000, 6000000), "ef": ef, "order": order,
                "weighted": rng.random() < 0.7}
    if kind == "spmv_host":
        return {"kind": kind, "graph": graph, "n": _log_int(rng, 900, 300000), "ef": ef, "order": order,
                "weighted": rng.random() < 0.7}
    if kind == "ppr":
        return {"kind": kind, "graph": graph, "n": _log_int(rng, 10000, 700000), "ef": rng.randint(4, 14),
                "k": rng.randint(1, 64), "iterations": rng.choice([10, 20]), "epsilon": 1e-6}
    return {"kind": kind, "graph": graph, "count": rng.randint(4, 60), "n": _log_int(rng, 900, 40000),
            "ef": rng.randint(4, 14), "order": order, "iterations": rng.choice([20, 50]), "epsilon": 1e-6}


# ------------------------------------------------------------------ graphs
def _edges(graph, n, ef, seed):
    """ef * n generated edges (duplicates and self loops among them), int32 on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    m = n * ef
    if graph == "er":
        src = torch.randint(0, n, (m,), generator=g, device="cuda", dtype=torch.int32)
        dst = torch.randint(0, n, (m,), generator=g, device="cuda", dtype=torch.int32)
        return src, dst
    src = torch.zeros(m, dtype=torch.int32, device="cuda")
    dst = torch.zeros(m, dtype=torch.int32, device="cuda")
    for _ in range(max(1, (n - 1).bit_length())):
        r = torch.rand(m, generator=g, device="cuda")
        src.mul_(2).add_(r >= A + B)
        dst.mul_(2).add_(((r >= A) & (r < A + B)) | (r >= A + B + C_))
    if n & (n - 1):
        src.remainder_(n)
        dst.remainder_(n)
    return src, dst


def _weights(m, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed + 7919)
    return torch.rand(m, generator=g, device="cuda")


def _vector(n, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed + 104729)
    return torch.rand(n, generator=g, device="cuda")


def _sources(case, seed):
    r = np.random.default_rng(seed + 13)
    return r.choice(case["n"], size=case["k"], replace=False).astype(np.uint32)


def _multi_sizes(case):
    """Vertex counts of a batch's graphs, the same for every seed."""
    r = np.random.default_rng(case["n"] + case["count"])
    lo = max(64, case["n"] // 12)
    return [int(v) for v in np.exp(r.uniform(np.log(lo), np.log(case["n"]), case["count"]))]


def _order(case):
    return ag.AG_ORDER_EXACT if case.get("order") == "exact" else ag.AG_ORDER_FAST


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    s = {"case": case}
    if kind == "multi":
        graphs = []
        for i, k in enumerate(_multi_sizes(case)):
            src, dst = _edges(case["graph"], k, case["ef"], seed * 1000 + i)
            graphs.append(ag.Graph.from_edges(k, src.cpu().numpy(), dst.cpu().numpy(), flags=ag.AG_BUILD_DEDUPE))
        s["graph"] = ag.MultiGraph(graphs)
        return s
    src, dst = _edges(case["graph"], n, case["ef"], seed)
    w = _weights(src.numel(), seed) if case.get("weighted") else None
    torch.cuda.synchronize()
    if kind == "build":
        s["src"], s["dst"] = src, dst
    elif kind == "call":
        s["graph"] = ag.Graph.build_gpu(n, src, dst, flags=ag.AG_BUILD_DEDUPE | ag.AG_BUILD_PINNED)
        s["arguments"] = ag.default_arguments(case["iterations"], case["epsilon"])
    else:
        s["graph"] = ag.DeviceGraph.from_edges(n, src, dst, w)
        if kind == "spmv":
            s["x"], s["y"] = _vector(n, seed), torch.empty(n, device="cuda")
        elif kind == "spmv_host":
            s["x"] = _vector(n, seed).cpu().numpy()
        elif kind == "ppr":
            s["sources"] = _sources(case, seed)
    if kind in ("spmv", "spmv_host"):
        s["mode"] = ((ag.AG_SPMV_GRAPH_WEIGHTS if case["weighted"] else ag.AG_SPMV_UNIT)
                     | (ag.AG_SPMV_EXACT if case["order"] == "exact" else 0))
    torch.cuda.synchronize()
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "solve":
        precision = ag.AG_PREC_BF16 if case["precision"] == "bf16" else ag.AG_PREC_FP32
        ranks, res, _ = state["graph"].pagerank(case["iterations"], case["epsilon"], precision, _order(case))
        return _counted(case, ranks, res)
    if kind == "build":
        g = ag.DeviceGraph.from_edges(case["n"], state["src"], state["dst"])
        ranks, res, _ = g.pagerank(case["iterations"], case["epsilon"], order=_order(case))
        g.release()
        return _counted(case, ranks, res)
    if kind == "call":
        opts = ag.make_opts(order=_order(case))
        out = C.POINTER(ag.PageRankStats)()
        ag.check(ag.lib.ag_pagerank_pull_ex(C.byref(state["arguments"]), state["graph"].ptr, C.byref(opts),
                                            C.byref(out)), "ag_pagerank_pull_ex")
        ranks = ag.stats_ranks(out)
        ag.lib.freePageRankStats(out)
        return {"ranks": ranks}
    if kind == "spmv":
        y = state["y"]
        ag.check(ag.lib.ag_spmv_pull_device(state["graph"].h, state["x"].data_ptr(), y.data_ptr(), state["mode"]),
                 "ag_spmv_pull_device")
        return {"y": y}
    if kind == "spmv_host":
        return {"y": state["graph"].spmv(state["x"], state["mode"])}
    if kind == "ppr":
        ranks, _ = state["graph"].ppr(state["sources"], case["iterations"], case["epsilon"])
        return {"ranks": ranks}
    parts, _ = state["graph"].pagerank(case["iterations"], case["epsilon"], _order(case))
    return parts


def _counted(case, ranks, res):
    out = {"ranks": ranks}
    if case["order"] == "exact":  # the reference's pass count, which FAST order does not promise
        out["passes"] = int(res.passes)
    return out


# -------------------------------------------------------------------- work
def _kept(graph, n, ef):
    """Edges left of ef * n once duplicates and self loops are dropped (estimate)."""
    if graph == "er":
        return ef * n
    return ef * n * (1.0 - 0.4 * 2.0 ** (-(math.log2(n) - 10) / 3.2))


def work(case):
    kind = case["kind"]
    if kind == "multi":
        lo, hi = max(64, case["n"] // 12), case["n"]
        n = case["count"] * (hi - lo) / math.log(hi / lo)
        e = case["ef"] * n * 0.7
        return {"bytes": case["iterations"] * (4 * e + 24 * n) + 4 * n, "flops": case["iterations"] * (e + 3 * n)}
    n = case["n"]
    e = _kept(case["graph"], n, case["ef"])
    if kind == "spmv":
        return {"bytes": (8 if case["weighted"] else 4) * e + 12 * n, "flops": (2 if case["weighted"] else 1) * e}
    if kind == "spmv_host":
        return {"bytes": (8 if case["weighted"] else 4) * e + 20 * n, "flops": (2 if case["weighted"] else 1) * e}
    if kind == "ppr":
        k = case["k"]
        return {"bytes": case["iterations"] * (4 * e + 8 * n + 16 * k * n) + 4 * k * n,
                "flops": case["iterations"] * k * (e + 3 * n)}
    per_pass = 4 * e + (20 if case.get("precision") == "bf16" else 24) * n
    extra = {"solve": 4 * n, "call": 4 * e + 16 * n, "build": 8 * case["ef"] * n + 4 * n}[kind]
    return {"bytes": case["iterations"] * per_pass + extra, "flops": case["iterations"] * (e + 3 * n)}


# ------------------------------------------------------------------- exact
def _matrix(n, src, dst, w=None):
    """The deduplicated inverse adjacency (row = destination) in 64 bits, and the out-degrees.  The first of several
    equal edges stays, with its weight."""
    key, at = torch.sort(src.long() * n + dst.long(), stable=True)
    keep = torch.ones_like(key, dtype=torch.bool)
    keep[1:] = key[1:] != key[:-1]
    keep &= torch.div(key, n, rounding_mode="floor") != key % n
    key, at = key[keep], at[keep]
    s, d = torch.div(key, n, rounding_mode="floor"), key % n
    del key, keep
    outdeg = torch.bincount(s, minlength=n)
    d, by = torch.sort(d, stable=True)
    col = s[by]
    val = torch.ones(d.numel(), dtype=torch.float64, device=d.device) if w is None else w[at[by]].double()
    row = torch.zeros(n + 1, dtype=torch.int64, device=d.device)
    row[1:] = torch.cumsum(torch.bincount(d, minlength=n), 0)
    return torch.sparse_csr_tensor(row, col, val, (n, n)), outdeg


def _pagerank64(n, src, dst, iterations, epsilon):
    m, outdeg = _matrix(n, src, dst)
    inv = torch.where(outdeg > 0, 1.0 / outdeg.clamp(min=1).double(), 0.0)
    r = torch.full((n,), BASE, dtype=torch.float64, device="cuda")
    for _ in range(iterations):
        new = BASE + DAMP * (m @ (r * inv).unsqueeze(1)).squeeze(1)
        moved = bool(((new - r).abs() >= epsilon).any())
        r = new
        if not moved:
            break
    return (r / n).cpu()


def exact(case, seed):
    kind = case["kind"]
    if kind == "multi":
        out = []
        for i, k in enumerate(_multi_sizes(case)):
            src, dst = _edges(case["graph"], k, case["ef"], seed * 1000 + i)
            out.append(_pagerank64(k, src, dst, case["iterations"], case["epsilon"]))
        return out
    n = case["n"]
    src, dst = _edges(case["graph"], n, case["ef"], seed)
    if kind in ("spmv", "spmv_host"):
        m, _ = _matrix(n, src, dst, _weights(src.numel(), seed) if case["weighted"] else None)
        return {"y": (m @ _vector(n, seed).double().unsqueeze(1)).squeeze(1).cpu()}
    if kind == "ppr":
        m, outdeg = _matrix(n, src, dst)
        inv = torch.where(outdeg > 0, 1.0 / outdeg.clamp(min=1).double(), 0.0).unsqueeze(1)
        teleport = torch.zeros((n, case["k"]), dtype=torch.float64, device="cuda")
        sources = torch.from_numpy(_sources(case, seed).astype(np.int64)).cuda()
        teleport[sources, torch.arange(case["k"], device="cuda")] = BASE * n
        r = teleport
        for _ in range(case["iterations"]):
            new = teleport + DAMP * (m @ (r * inv))
            moved = bool(((new - r).abs() >= case["epsilon"]).any())
            r = new
            if not moved:
                break
        return {"ranks": (r / n).cpu()}
    out = {"ranks": _pagerank64(n, src, dst, case["iterations"], case["epsilon"])}
    if kind in ("solve", "build") and case["order"] == "exact":
        out["passes"] = None
    return out
