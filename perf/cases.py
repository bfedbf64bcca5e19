"""Timed cases of the engine: what its users have it do, through its public calls.

A case names a call (`op`), a graph family with its edge count, and the options of the
call.  The families are those of the repository's workloads, at other sizes and seeds:

* ``er``   uniform bipartite graphs of mean degree 8 (config 1 is the one with 20k edges);
* ``cl``   the Chung-Lu power-law graph of the bench, vertex counts scaled with the edges;
* ``hub``  the hub-skewed graph (power-law U side with very large hubs, uniform V side);
* ``b``    one graph of the batched workload (Chung-Lu, mean degree 8, gamma 2.3).

Calls on a resident graph (``bfc``, ``ebfc``, ``msp``, ``hidx``) are timed without the upload,
``load_ebfc`` is a new host graph uploaded and counted, ``msp_batch`` takes host graphs through
packing, upload and peeling, ``noalloc`` counts on the caller's own device buffers.
"""

import numpy as np
import torch

import gpu_bitruss_gb300 as bt
from gpu_bitruss_gb300 import gen


def listed():
    return [
        # the smallest interactive call: the butterfly count of config 1
        {"name": "bfc_er_20k", "op": "bfc", "family": "er", "m": 20_000},
        # a plugin host's count on its own buffers, enqueued on its stream
        {"name": "noalloc_b_300k", "op": "noalloc", "family": "b", "m": 300_000},
        # per-edge supports of a resident power-law graph
        {"name": "ebfc_cl_2000k", "op": "ebfc", "family": "cl", "m": 2_000_000},
        # per-edge supports where a few hubs hold most wedges
        {"name": "ebfc_hub_4000k", "op": "ebfc", "family": "hub", "m": 4_000_000},
        # a new graph from the host: upload and supports, the path of every first call
        {"name": "load_ebfc_b_500k", "op": "load_ebfc", "family": "b", "m": 500_001},
        # decompositions from a request-sized graph to the largest that peels in a second or so
        {"name": "msp_b_1k", "op": "msp", "family": "b", "m": 1_000, "exact": False},
        {"name": "msp_cl_20k", "op": "msp", "family": "cl", "m": 20_000, "exact": False},
        {"name": "msp_cl_200k", "op": "msp", "family": "cl", "m": 200_000, "exact": False},
        {"name": "msp_cl_1000k", "op": "msp", "family": "cl", "m": 1_000_000, "exact": False},
        # the corrected rule on hub rows
        {"name": "msp_exact_hub_200k", "op": "msp", "family": "hub", "m": 200_003, "exact": True},
        # h-index rounds from the supports
        {"name": "hidx_cl_50k", "op": "hidx", "family": "cl", "m": 50_000},
        # one arena of a batch of request-sized graphs
        {"name": "msp_batch_48", "op": "msp_batch", "family": "b", "count": 48, "lo": 1_000, "hi": 100_000,
         "exact": False},
    ]


# Edge counts that drawn cases span, by call and family: up to what a pass of about a second allows.
SPAN = {
    "bfc": {"er": (1e3, 4e6), "cl": (1e3, 4e6), "hub": (1e4, 4e6), "b": (1e3, 2e6)},
    "noalloc": {"er": (1e3, 4e5), "cl": (1e3, 4e5), "b": (1e3, 5e5)},
    "ebfc": {"er": (1e3, 4e6), "cl": (1e3, 4e6), "hub": (1e4, 4e6), "b": (1e3, 2e6)},
    "load_ebfc": {"er": (1e3, 2e6), "cl": (1e3, 2e6), "hub": (1e4, 2e6), "b": (1e3, 2e6)},
    "msp": {"er": (1e3, 2e6), "cl": (1e3, 5e5), "hub": (1e4, 3e5), "b": (1e3, 1e6)},
    "hidx": {"er": (1e3, 2e5), "cl": (1e3, 1e5), "hub": (5e3, 4e4), "b": (1e3, 2e5)},
}


def _log_uniform(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    op = rng.choice(["bfc", "noalloc", "ebfc", "load_ebfc", "msp", "msp", "msp", "hidx", "msp_batch"])
    if op == "msp_batch":
        return {"op": op, "family": "b", "count": rng.randint(2, 60), "lo": 1_000,
                "hi": _log_uniform(rng, 2e3, 1e5), "exact": rng.random() < 0.3}
    family = rng.choice(sorted(SPAN[op]))
    case = {"op": op, "family": family, "m": _log_uniform(rng, *SPAN[op][family])}
    if op == "msp":
        case["exact"] = rng.random() < 0.3
    return case


def _sizes(case):
    """(m, |U|, |V|) of every graph of the case (the seed does not change them)."""
    if case["op"] == "msp_batch":
        return list(zip(*(a.tolist() for a in gen.batch_sizes(case["count"], case["lo"], case["hi"]))))
    m, family = case["m"], case["family"]
    if family == "er":  # config 1 has 2,000 x 3,000 vertices and 20,000 edges
        return [(m, m // 10, 3 * m // 20)]
    if family == "cl":  # the bench's graph has 1,000,000 x 500,000 vertices and 20,000,000 edges
        return [(m, max(m // 20, 64), max(m // 40, 64))]
    if family == "hub":
        return [(m, max(m // 1000, 32), max(m // 20, 64))]
    return [(m, m // 10, m // 4 - m // 10)]


def _edges(case, size, seed):
    m, nu, nv = size
    if case["family"] == "er":
        return gen.er(nu, nv, m, seed=seed)
    if case["family"] == "cl":
        cap = max(50_000 * (m / 20_000_000) ** 0.5, 16.0)
        return gen.chung_lu(nu, nv, m, 2.1, 2.1, min(cap, nv), min(cap, nu), seed=seed)
    if case["family"] == "hub":
        return gen.hub_skew(nu, nv, m, 1.8, max(m / 100, 16.0), seed=seed)
    cap = max(8.0, min(nu, nv) * 0.5)
    return gen.chung_lu(nu, nv, m, 2.3, 2.3, min(cap, nv), min(cap, nu), seed=seed)


def prepare(case, seed):
    graphs = [bt.Graph.from_edges(*_edges(case, size, 1_000 * seed + i)) for i, size in enumerate(_sizes(case))]
    state = {"op": case["op"], "exact": case.get("exact", False), "graphs": graphs, "graph": graphs[0]}
    if case["op"] == "noalloc":
        g = graphs[0]
        state["offsets"] = torch.from_numpy(g.offsets.view(np.int32)).cuda()
        state["neighbors"] = torch.from_numpy(g.neighbors.view(np.int32)).cuda()
        state["count"] = torch.zeros(1, dtype=torch.int64, device="cuda")
        return state
    state["ctx"] = bt.Context(0)
    if case["op"] not in ("load_ebfc", "msp_batch"):
        state["ctx"].upload(graphs[0])
    return state


def run(state):
    op, g = state["op"], state["graph"]
    if op == "noalloc":
        bt.bfc_noalloc(0, state["offsets"].data_ptr(), state["neighbors"].data_ptr(), g.n, g.m,
                       state["count"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return {"count": state["count"]}
    ctx = state["ctx"]
    if op == "bfc":
        return {"count": ctx.bfc()}
    if op == "hidx":
        values, rounds = ctx.hidx()
        return {"bitruss": values, "rounds": rounds}
    if op == "msp":
        values, levels = ctx.msp(exact=state["exact"])
        return {"bitruss": values, "levels": levels}
    if op == "msp_batch":
        values, levels = ctx.msp_batch(state["graphs"], exact=state["exact"])
        return {"bitruss": values, "levels": levels}
    if op == "load_ebfc":
        ctx.upload(g)
    sup, count, largest = ctx.ebfc()
    return {"support": sup, "count": count, "largest": largest}


def work(case):
    """Bytes of the CSR read once and of the results written once (the operations are integer ones)."""
    sizes = _sizes(case)
    m = sum(s[0] for s in sizes)
    n = sum(s[1] + s[2] for s in sizes)
    csr = 4 * (n + 1) + 8 * m  # offsets, neighbours of both directions
    if case["op"] in ("bfc", "noalloc"):
        return {"bytes": csr + 8, "flops": 0}
    per_edge = 8 if case["op"] in ("ebfc", "load_ebfc") else 4
    return {"bytes": csr + 8 * m + per_edge * m, "flops": 0}  # with the edge ids of both directions


def exact(case, seed):
    """Counts and supports from dense products in 64 bits, where the matrix is small."""
    if case["op"] not in ("bfc", "noalloc", "ebfc", "load_ebfc"):
        return None
    m, nu, nv = _sizes(case)[0]
    if nu * nv > 100_000_000:
        return None
    u, v = (torch.from_numpy(x.astype(np.int64)).cuda() for x in _edges(case, (m, nu, nv), 1_000 * seed))
    a = torch.zeros(nu, nv, dtype=torch.float64, device="cuda")
    a[u, v] = 1.0
    pairs = a @ a.T
    pairs.fill_diagonal_(0.0)
    count = int(round(float((pairs * (pairs - 1.0)).sum()) / 4.0))
    if case["op"] == "noalloc":
        return {"count": torch.tensor([count])}
    if case["op"] == "bfc":
        return {"count": count}
    # support(u, v): paths u-x-w-v of three edges, less those through (u, v) itself
    sup = ((pairs @ a)[u, v] - (a.sum(0)[v] - 1.0)).round().to(torch.int64).cpu().numpy()
    first_u, first_v = (_first_seen(x.cpu().numpy()) for x in (u, v))
    sup = sup[np.lexsort((first_v, first_u))]  # edge ids: by U vertex, then V vertex, as first seen
    return {"support": sup.astype(np.uint64), "count": count, "largest": int(sup.max())}


def _first_seen(ids):
    """Each entry's vertex number when vertices are numbered by first appearance."""
    _, first, inverse = np.unique(ids, return_index=True, return_inverse=True)
    rank = np.empty(first.size, np.int64)
    rank[np.argsort(first)] = np.arange(first.size)
    return rank[inverse]
