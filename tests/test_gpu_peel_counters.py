"""The peel's work counters on graphs whose walk is known."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _disjoint(shapes):
    u, v, bu, bv = [], [], 0, 0
    for a, b in shapes:
        u.append(bu + np.repeat(np.arange(a), b))
        v.append(bv + np.tile(np.arange(b), a))
        bu, bv = bu + a, bv + b
    return np.concatenate(u).astype(np.uint32), np.concatenate(v).astype(np.uint32)


# K(2, 20) goes at level 19 and leaves less than half of the edges, so the rows are
# compacted in front of level 21, whose frontier of 32 edges (K(4, 8)) is planned
# inside the barrier.  In each block both ends' rows hold as many positions, so
# the V end is the pivot and an edge's anchor row is its U end's.
def test_anchors_are_counted_once(engine, gpu_ctx):
    u, v = _disjoint([(2, 20), (4, 8)])
    gpu_ctx.upload(engine.Graph.from_edges(u, v))
    for exact in (False, True):
        res, levels = gpu_ctx.msp(exact=exact)
        assert levels == 21
        st = gpu_ctx.stats()
        assert st[2] == 1  # one compaction
        assert st[10] == 40 * 20 + 32 * 8
