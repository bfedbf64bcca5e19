"""The allocation-free count's two ways: vertices renumbered by degree with
counters in shared memory, or counters in its scratch for small graphs, large
ones and rows that are not in the layout.  Exact against the oracle's count or,
for rows no graph file gives, against the definition."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _call(engine, off, nbr, m=None, captured=False):
    torch = pytest.importorskip("torch")
    d_off = torch.from_numpy(np.ascontiguousarray(off, np.uint32).view(np.int32)).cuda()
    d_nbr = torch.from_numpy(np.ascontiguousarray(nbr, np.uint32).view(np.int32)).cuda()
    out = torch.full((1,), -1, dtype=torch.int64, device="cuda")
    n, m = len(off) - 1, len(nbr) // 2 if m is None else m
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    engine.bfc_noalloc(0, d_off.data_ptr(), d_nbr.data_ptr(), n, m, out.data_ptr(), st.cuda_stream)
    if captured:
        st.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            engine.bfc_noalloc(0, d_off.data_ptr(), d_nbr.data_ptr(), n, m, out.data_ptr(), st.cuda_stream)
        out.fill_(-1)
        torch.cuda.synchronize()
        for _ in range(2):
            g.replay()
    torch.cuda.synchronize()
    return int(out.cpu().numpy().view(np.uint64)[0])


def _random(m, u, v, seed):
    rng = np.random.default_rng(seed)
    key = rng.choice(u * v, size=m, replace=False)
    return (key // v).astype(np.uint32), (key % v).astype(np.uint32)


@pytest.mark.parametrize("m", [24575, 24576, 24577])
def test_smallest_renumbered(engine, oracle_mod, m):
    u, v = _random(m, 700, 900, m)
    g = engine.Graph.from_edges(u, v)
    assert _call(engine, g.offsets, g.neighbors) == oracle_mod.ebfc(oracle_mod.build_csr(u, v), 0)[1]


def _far_ends(n, mids):
    """One vertex joined to every middle vertex, the others of its side to two
    each: its wedge ends lie all over the ranks."""
    few = np.arange(1, n - mids)
    u = np.concatenate([np.zeros(mids, np.int64), few, few])
    v = np.concatenate([np.arange(mids), few % mids, (few * 7 + few // mids) % mids])
    key = np.unique(u * mids + v)
    return (key // mids).astype(np.uint32), (key % mids).astype(np.uint32)


# one, two, three and sixteen windows of 52,224 ranks; more than the scratch holds
@pytest.mark.parametrize("n", [52_000, 57_000, 130_000, 820_000, 850_000])
def test_windows(engine, oracle_mod, n):
    u, v = _far_ends(n, 3000)
    for a, b in ((u, v), (v, u)):
        g = engine.Graph.from_edges(a, b)
        assert g.n == n
        assert _call(engine, g.offsets, g.neighbors) == oracle_mod.ebfc(oracle_mod.build_csr(a, b), 0)[1]


def test_captured(engine, oracle_mod):
    u, v = _random(30000, 500, 900, 2)
    g = engine.Graph.from_edges(u, v)
    assert _call(engine, g.offsets, g.neighbors, captured=True) == oracle_mod.ebfc(oracle_mod.build_csr(u, v), 0)[1]


def test_rows_out_of_order_and_wrong_edge_count(engine, oracle_mod):
    u, v = _random(30000, 500, 900, 3)
    g = engine.Graph.from_edges(u, v)
    expect = oracle_mod.ebfc(oracle_mod.build_csr(u, v), 0)[1]
    nbr = g.neighbors.copy()
    for x in range(0, g.n, 3):
        nbr[g.offsets[x]:g.offsets[x + 1]] = nbr[g.offsets[x]:g.offsets[x + 1]][::-1]
    assert _call(engine, g.offsets, nbr) == expect
    for m in (g.m - 1, g.m + 1):
        assert _call(engine, g.offsets, g.neighbors, m=m) == expect


def test_repeated_neighbours(engine):
    # the count by its definition: wedges from the vertex above both others by
    # (degree, id), pairs of them with the same ends
    u, v = _random(26000, 200, 220, 4)
    u, v = np.concatenate([u, u[:2000]]).astype(int), np.concatenate([v, v[:2000]]).astype(int) + 200
    src, dst = np.concatenate([u, v]), np.concatenate([v, u])
    order = np.lexsort((dst, src))
    src, dst = src[order], dst[order]
    off = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=420))])
    deg = np.diff(off)
    pri = np.empty(420, np.int64)
    pri[np.lexsort((np.arange(420), deg))] = np.arange(420)
    a = np.zeros((420, 420), np.int64)
    np.add.at(a, (src, dst), 1)
    total = 0
    for x in range(420):
        c = a[x][pri < pri[x]] @ a[pri < pri[x]]
        c = c[pri < pri[x]]
        total += int((c * (c - 1) // 2).sum())
    assert _call(engine, off, dst) == total
