"""The peeling kernel where its plan changes: frontiers of up to 32 edges are
planned inside the grid barrier, up to 512 by every CTA, larger ones in chunks;
a block of 32 mids is cut into parts; long rows are walked from either side."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# K(a, b) peels in one sub-round whose frontier is all a * b edges, each with
# support (a - 1)(b - 1): 31, 32, 33, 511, 512 and 513 of them, then rows longer
# than a block of mids on one side or both.
@pytest.mark.parametrize("a,b", [(1, 31), (4, 8), (3, 11), (7, 73), (16, 32), (19, 27), (2, 33), (3, 700), (33, 65),
                                 (40, 1300)])
@pytest.mark.parametrize("schedule", [(0, 0, 0), (1, 64, 1), (4096, 1, 32)])
def test_complete_bipartite_at_the_edges_of_the_plan(engine, gpu_ctx, a, b, schedule):
    u = np.repeat(np.arange(a, dtype=np.uint32), b)
    v = np.tile(np.arange(b, dtype=np.uint32), a)
    gpu_ctx.upload(engine.Graph.from_edges(u, v))
    gpu_ctx.set_msp_schedule(*schedule)
    try:
        for exact in (False, True):
            res, levels = gpu_ctx.msp(exact=exact)
            assert np.all(res == (a - 1) * (b - 1))
            assert levels == (a - 1) * (b - 1)
    finally:
        gpu_ctx.set_msp_schedule(0, 0, 0)


# Two hubs sharing `shared` neighbours, each with `own` more of its own: the
# walk's two rows differ in length by up to three orders of magnitude, and the
# row tables hold from one bucket to thousands.
@pytest.mark.parametrize("shared,own", [(2, 0), (2, 5000), (31, 1), (33, 4000), (700, 3), (5000, 5000)])
def test_two_hubs(engine, gpu_ctx, oracle_mod, shared, own):
    rng = np.random.default_rng(shared * 7919 + own)
    u = [0] * shared + [1] * shared + [0] * own + [1] * own + list(range(2, 2 + min(shared, 300)))
    v = list(range(shared)) * 2 + list(range(shared, shared + 2 * own)) + list(range(min(shared, 300)))
    order = rng.permutation(len(u))
    u, v = np.array(u, np.uint32)[order], np.array(v, np.uint32)[order]
    gpu_ctx.upload(engine.Graph.from_edges(u, v))
    want, levels, _ = oracle_mod.msp(oracle_mod.build_csr(u, v), 0, oracle_mod.MSP_REF)
    res, got_levels = gpu_ctx.msp()
    np.testing.assert_array_equal(res.astype(np.uint64), want)
    assert got_levels == levels


# Batches are peeled by teams of CTAs: more graphs than CTAs, fewer, equal ones
# and very unequal ones, empty ones between; every graph as when peeled alone.
@pytest.mark.parametrize("sizes", [[40] * 300, [30_000, 50, 50], [2000, 0, 2000, 0, 300], [20_000] + [200] * 60])
@pytest.mark.parametrize("ctas", [0, 5])
def test_batches_in_teams(engine, gpu_ctx, sizes, ctas):
    from gpu_bitruss_gb300 import gen
    graphs = []
    for i, m in enumerate(sizes):
        u, v = gen.er(max(m // 8, 8), max(m // 8, 8), m, seed=i) if m else (np.zeros(0, np.uint32),) * 2
        graphs.append(engine.Graph.from_edges(u, v))
    gpu_ctx.set_peel_ctas(ctas)
    try:
        for exact in (False, True):
            res, levels = gpu_ctx.msp_batch(graphs, exact=exact)
            assert len(res) == len(graphs)
            for i in {0, 1, len(graphs) // 2, len(graphs) - 1}:
                gpu_ctx.upload(graphs[i])
                alone, lv = gpu_ctx.msp(exact=exact)
                np.testing.assert_array_equal(res[i], alone)
                assert int(levels[i]) == lv
    finally:
        gpu_ctx.set_peel_ctas(0)
