"""Frontiers on either side of the plan's limits whose edges decrement others: a
task left out, cut wrongly or run twice changes the values of the dense block
that they hang on.  Exact against the oracle, with the number of decrements."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class Edges:
    def __init__(self, nu, nv):  # the block: K(nu, nv)
        self.u = list(np.repeat(np.arange(nu), nv))
        self.v = list(np.tile(np.arange(nv), nu))
        self.nu, self.nv = nu, nv

    def add(self, pairs):
        for a, b in pairs:
            self.u.append(a)
            self.v.append(b)

    def complete(self, a, b):  # K(a, b) of its own
        self.add((self.nu + i, self.nv + j) for i in range(a) for j in range(b))
        self.nu, self.nv = self.nu + a, self.nv + b

    def shuffled(self, seed):
        order = np.random.default_rng(seed).permutation(len(self.u))
        return np.array(self.u, np.uint32)[order], np.array(self.v, np.uint32)[order]


# Level 4: U vertices with two edges into K(4, B), whose four butterflies each have
# both edges in the frontier and two survivors; K(3, 3) (9 edges) makes it odd.
def two_survivors(n, block):
    rng = np.random.default_rng(n)
    g = Edges(4, block)
    if n % 2:
        g.complete(3, 3)
    seen = set()
    while len(seen) < (n - 9 * (n % 2)) // 2:
        a, b = sorted(int(x) for x in rng.choice(block, 2, replace=False))
        seen.add((a, b))
    for a, b in sorted(seen):
        g.add([(g.nu, a), (g.nu, b)])
        g.nu += 1
    return g.shuffled(n), 4


# Level 1: an edge (u, v) of the block closed to a butterfly by one more vertex on
# either side, three frontier edges and one survivor, which the reference's rule
# decrements only in some orders of the edges' ids; K(2, 2) makes up the number.
def one_survivor(n, block):
    rng = np.random.default_rng(n + 1)
    g = Edges(4, block)
    for _ in range(n % 3):
        g.complete(2, 2)
    for _ in range((n - 4 * (n % 3)) // 3):
        u, v = int(rng.integers(4)), int(rng.integers(block))
        g.add([(g.nu, v), (g.nu, g.nv), (u, g.nv)])
        g.nu, g.nv = g.nu + 1, g.nv + 1
    return g.shuffled(n), 1


# the block's U rows, of 60 or 400, are longer than a block of mids; frontiers of
# more than 512 edges are cut into chunks
@pytest.mark.parametrize("make", [two_survivors, one_survivor])
@pytest.mark.parametrize("n,block", [(31, 60), (32, 60), (33, 60), (511, 60), (512, 60), (513, 60), (3001, 400)])
def test_frontier_that_decrements(engine, gpu_ctx, oracle_mod, make, n, block, tmp_path, monkeypatch):
    from gpu_bitruss_gb300 import trace
    (u, v), level = make(n, block)
    o = oracle_mod.build_csr(u, v)
    gpu_ctx.upload(engine.Graph.from_edges(u, v))
    path = str(tmp_path / "trace.bin")
    monkeypatch.setenv("BT_MSP_TRACE", path)
    try:
        for exact, mode in ((False, oracle_mod.MSP_REF), (True, oracle_mod.MSP_EXACT)):
            want, levels, stats = oracle_mod.msp(o, 0, mode)
            for schedule in ((0, 0, 0), (1, 64, 1), (4096, 1, 32), (1 << 30, 1, 512)):
                gpu_ctx.set_msp_schedule(*schedule)
                res, lv = gpu_ctx.msp(exact=exact)
                np.testing.assert_array_equal(res.astype(np.uint64), want)
                assert lv == levels
                st = gpu_ctx.stats()
                assert st[1] == stats[1] and st[12] == stats[6]
                assert int(trace.load(path)["frontier"][0]) == n == int((res == level).sum())
    finally:
        gpu_ctx.set_msp_schedule(0, 0, 0)
