"""The h-index kernel where its paths meet: an edge of few row positions is one
warp's, a larger one a CTA's; the first window is 256 values below the edge's
value, an edge that falls further takes wider ones; values of 32 and 64 bits."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(engine, ctx, oracle_mod, u, v, monkeypatch):
    order = np.random.default_rng(u.size).permutation(u.size)
    u, v = u[order].astype(np.uint32), v[order].astype(np.uint32)
    want, want_rounds = oracle_mod.hidx(oracle_mod.build_csr(u, v), 0)
    ctx.upload(engine.Graph.from_edges(u, v))
    for wide in ("0", "1"):
        monkeypatch.setenv("BT_MSP_WIDE", wide)
        got, rounds = ctx.hidx()
        np.testing.assert_array_equal(got.astype(np.uint64), want)
        assert rounds == want_rounds


# K(a, b) minus a few edges: about (a - 1)(b - 1) butterflies an edge, on either
# side of 4,096 positions, and values on either side of the first window
@pytest.mark.parametrize("a,b", [(3, 40), (17, 17), (33, 31), (64, 64), (65, 66), (20, 400)])
def test_nearly_complete(engine, gpu_ctx, oracle_mod, a, b, monkeypatch):
    keep = np.random.default_rng(a * b).random(a * b) > 0.05
    u, v = np.repeat(np.arange(a), b)[keep], np.tile(np.arange(b), a)[keep]
    _check(engine, gpu_ctx, oracle_mod, u, v, monkeypatch)


# edges into a dense block from outside it: supports of thousands that fall to a
# few, past the first window by several orders of bins
@pytest.mark.parametrize("side,extra", [(40, 30), (70, 5)])
def test_values_that_fall_far(engine, gpu_ctx, oracle_mod, side, extra, monkeypatch):
    u = [np.repeat(np.arange(side), side)]
    v = [np.tile(np.arange(side), side)]
    for k in range(extra):  # a vertex with two edges into the block and a pendant one
        u.append(np.array([side + k] * 3))
        v.append(np.array([k % side, (k * 7 + 1) % side, side + k]))
    u.append(np.zeros(2000, np.int64))  # a hub row
    v.append(np.arange(side + extra, side + extra + 2000))
    u, v = np.concatenate(u), np.concatenate(v)
    keys = np.unique(u.astype(np.int64) * 100_000 + v)
    _check(engine, gpu_ctx, oracle_mod, keys // 100_000, keys % 100_000, monkeypatch)
