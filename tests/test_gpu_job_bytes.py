"""The admission estimate against what a job allocates: never below it, and not
above it by the sums in 64 bits that only repeated lines need."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("again", [0, 1])
@pytest.mark.parametrize("op", ["ebfc", "msp"])
def test_estimate_and_peak(engine, op, again):
    from gpu_bitruss_gb300 import gen
    m = 400_000
    u, v = gen.er(2000, 2000, m, seed=3)
    g = engine.Graph.from_edges(np.concatenate([u, u[:again]]), np.concatenate([v, v[:again]]))
    ctx = engine.Context(0)
    try:
        est = ctx.job_bytes([g], op)
        ctx.set_budget(est)
        ctx.upload(g)
        ctx.msp() if op == "msp" else ctx.ebfc()
        peak = ctx.memory_peak()
    finally:
        ctx.close()
    assert peak <= est
    # a peel is estimated with 64-bit working supports (4 m more) and rounding
    if op == "msp" and not again:
        assert est - peak < 8 * m
