"""Edge lists with repeated lines, which are kept: rows then hold a neighbour
twice, and counts and supports are those of the oracle on the same rows."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(engine, ctx, oracle_mod, u, v, tmp_path=None):
    u, v = np.asarray(u, np.uint32), np.asarray(v, np.uint32)
    sup, count = oracle_mod.ebfc(oracle_mod.build_csr(u, v), 0)
    g = engine.Graph.from_edges(u, v)
    if tmp_path is not None:
        g.to_bin(str(tmp_path / "g.bin"))
        g = engine.Graph.from_bin(str(tmp_path / "g.bin"))
    ctx.upload(g)
    assert ctx.bfc() == count
    got, cnt, largest = ctx.ebfc()
    np.testing.assert_array_equal(got, sup)
    assert cnt == count and largest == int(sup.max())


def _repeated(nu, nv, m, again, seed):
    from gpu_bitruss_gb300 import gen
    rng = np.random.default_rng(seed)
    u, v = gen.er(nu, nv, m, seed=seed)
    k = rng.integers(0, m, again)
    u, v = np.concatenate([u, u[k]]), np.concatenate([v, v[k]])
    p = rng.permutation(u.size)
    return u[p], v[p]


# a start vertex with one middle slot closes a butterfly if the slot's end repeats
@pytest.mark.parametrize("k", [2, 3, 33, 400])
def test_one_middle_vertex(engine, gpu_ctx, oracle_mod, k, tmp_path):
    # r - s once, s - w k times; r is above s and w by its other neighbours
    u = [0] * (k + 3) + [1] * k
    v = list(range(k + 3)) + [0] * k
    _check(engine, gpu_ctx, oracle_mod, u, v, tmp_path)
    _check(engine, gpu_ctx, oracle_mod, v, u)


@pytest.mark.parametrize("nu,nv,m,again", [(5, 5, 12, 1), (60, 80, 1500, 700), (500, 400, 8000, 400),
                                           (2000, 3000, 20000, 50), (3, 900, 2000, 2000)])
def test_random(engine, gpu_ctx, oracle_mod, nu, nv, m, again, tmp_path):
    _check(engine, gpu_ctx, oracle_mod, *_repeated(nu, nv, m, again, m + again), tmp_path)


# k parallel edges r - s and s - w: a slot of r - s sums k (k^2 - 1), on either side of 2^32
@pytest.mark.parametrize("k", [1620, 1700])
def test_slot_sums_past_32_bits(engine, gpu_ctx, oracle_mod, k):
    u = [0] * k + [0] * (k + 2) + [1] * k
    v = [0] * k + list(range(1, k + 3)) + [0] * k
    _check(engine, gpu_ctx, oracle_mod, u, v)


def test_batch_with_and_without(engine, gpu_ctx, oracle_mod):
    from gpu_bitruss_gb300 import gen
    lists = [gen.er(60, 80, 900, seed=1), _repeated(300, 200, 3000, 100, 2), gen.er(40, 30, 500, seed=3)]
    sups, counts = gpu_ctx.ebfc_batch([engine.Graph.from_edges(u, v) for u, v in lists])
    for (u, v), sup, count in zip(lists, sups, counts):
        want, total = oracle_mod.ebfc(oracle_mod.build_csr(u, v), 0)
        np.testing.assert_array_equal(sup, want)
        assert int(count) == total


# Parallel edges may share an edge id and a table entry; an h-index value that
# changes has to change wherever it is read.  64-bit values are read through the
# edge ids, so both widths must end alike.
@pytest.mark.parametrize("nu,nv,m,again,seed", [(60, 80, 1500, 20, 4), (500, 400, 8000, 400, 6), (20, 30, 150, 2, 20)])
def test_hidx_values_of_parallel_edges(engine, gpu_ctx, nu, nv, m, again, seed, monkeypatch):
    u, v = _repeated(nu, nv, m, again, seed)
    gpu_ctx.upload(engine.Graph.from_edges(u.astype(np.uint32), v.astype(np.uint32)))
    got = []
    for wide in ("0", "1"):
        monkeypatch.setenv("BT_MSP_WIDE", wide)
        got.append(gpu_ctx.hidx())
    np.testing.assert_array_equal(got[0][0], got[1][0])
    assert got[0][1] == got[1][1]
