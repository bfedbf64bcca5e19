"""The counting kernel where its paths meet: a warp matches up to 32 wedges in
registers, hashes up to 320, a CTA takes the rest in batches of 1,024 middle
vertices or, for many short rows, warp by warp; ranks past the shared counters
count in device memory; slot sums are 32 or 64 bits wide."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(engine, ctx, oracle_mod, u, v):
    order = np.random.default_rng(u.size).permutation(u.size)
    u, v = u[order].astype(np.uint32), v[order].astype(np.uint32)
    sup, count = oracle_mod.ebfc(oracle_mod.build_csr(u, v), 0)
    ctx.upload(engine.Graph.from_edges(u, v))
    assert ctx.bfc() == count
    for _ in range(2):  # the counters are clean again after a call
        got, cnt, largest = ctx.ebfc()
        np.testing.assert_array_equal(got, sup)
        assert cnt == count and largest == (int(sup.max()) if sup.size else 0)


# K(a, b): a start vertex has up to (a - 1) * b wedges over b middle vertices
@pytest.mark.parametrize("a,b", [(2, 16), (2, 33), (5, 8), (5, 64), (6, 64), (6, 65), (9, 1024), (3, 1025), (4, 3000)])
def test_complete_bipartite_supports(engine, gpu_ctx, oracle_mod, a, b):
    _check(engine, gpu_ctx, oracle_mod, np.repeat(np.arange(a), b), np.tile(np.arange(b), a))


# hubs over many short rows (warp by warp), and over rows longer than 512 (in batches)
@pytest.mark.parametrize("hubs,leaves,long_rows", [(3, 5000, 0), (40, 4000, 0), (3, 2500, 700)])
def test_hubs(engine, gpu_ctx, oracle_mod, hubs, leaves, long_rows):
    u = np.repeat(np.arange(hubs), leaves)
    v = np.tile(np.arange(leaves), hubs)
    if long_rows:  # two leaves with a long row of their own
        u = np.concatenate([u, np.tile(np.arange(hubs, hubs + long_rows), 2)])
        v = np.concatenate([v, np.repeat([0, 1], long_rows)])
    _check(engine, gpu_ctx, oracle_mod, u, v)


# more ranks than shared counters: wedges end on both sides of the line
def test_ranks_past_the_shared_counters(engine, gpu_ctx, oracle_mod):
    rng = np.random.default_rng(5)
    n = 70_000
    u = np.concatenate([np.arange(n), np.arange(n), np.repeat(np.arange(200), 300)])
    v = np.concatenate([np.arange(n), (np.arange(n) + 1) % n, rng.integers(0, n, 60_000)])
    keys = np.unique(u.astype(np.int64) * n + v)
    _check(engine, gpu_ctx, oracle_mod, keys // n, keys % n)


# degrees whose product passes 2^32 take the 64-bit sums
def test_wide_sums(engine, gpu_ctx, oracle_mod):
    k = 66_000
    u = np.concatenate([np.zeros(k, np.int64), np.arange(1, k), np.repeat(np.arange(1, 4), 500)])
    v = np.concatenate([np.arange(k), np.zeros(k - 1, np.int64), np.tile(np.arange(1, 501), 3)])
    _check(engine, gpu_ctx, oracle_mod, u, v)


def test_small_and_large_side_by_side(engine, oracle_mod):
    """Contexts of several threads count graphs that want different amounts of
    shared memory, over and over, at the same time."""
    from concurrent.futures import ThreadPoolExecutor
    rng = np.random.default_rng(7)

    def count(n):
        u, v = rng_edges[n]
        want = oracle_mod.ebfc(oracle_mod.build_csr(u, v), 0)[1]
        ctx = engine.Context(0)
        try:
            ctx.upload(engine.Graph.from_edges(u, v))
            return [ctx.bfc() for _ in range(300)], want
        finally:
            ctx.close()

    sizes = (1000, 40_000, 60_000, 90_000)
    rng_edges = {}
    for n in sizes:
        key = np.unique(rng.integers(0, n // 2, 2 * n) * n + rng.integers(0, n // 2, 2 * n))
        rng_edges[n] = ((key // n).astype(np.uint32), (key % n).astype(np.uint32))
    with ThreadPoolExecutor(len(sizes)) as pool:
        for got, want in pool.map(count, sizes):
            assert got == [want] * 300
