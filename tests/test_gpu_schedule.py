"""The schedule's first number keeps its meaning from one engine to the next: a
host's tuned values stay usable, and the built-in one is what it was."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_built_in_schedule(engine):
    ctx = engine.Context(0)
    try:
        assert ctx.msp_schedule() == (2048, 2, 512)
    finally:
        ctx.close()


# K(3, 700) is one frontier of 2,100 edges.  An edge's pivot row is that of its V
# end, one block of 3 mids, 2 of them with the 700 positions of their rows to
# walk: 1,400 of an estimated 3 * 700.
@pytest.mark.parametrize("grain,tasks_an_edge", [(1 << 20, 1), (2 * 2100 * 32, 1), (1050 * 32, 2)])
def test_positions_per_task(engine, gpu_ctx, grain, tasks_an_edge):
    u, v = np.repeat(np.arange(3), 700), np.tile(np.arange(700), 3)
    gpu_ctx.upload(engine.Graph.from_edges(u.astype(np.uint32), v.astype(np.uint32)))
    gpu_ctx.set_msp_schedule(grain, 1, 512)
    try:
        res, _ = gpu_ctx.msp()
        assert np.all(res == 2 * 699)
        st = gpu_ctx.stats()
        assert st[9] == 2100 * 1400
        assert 2100 * tasks_an_edge <= st[8] <= 2 * 2100 * tasks_an_edge
    finally:
        gpu_ctx.set_msp_schedule(0, 0, 0)
