"""The peel's control words when CTAs leave a barrier far apart: with
BT_MSP_LATE_NS an eighth of the CTAs, other ones at each barrier, read what they
need behind it 20 us late, when the others have long appended to the next lists
(a level's scan takes about 3 us).  Values, levels and sub-rounds are the same."""

import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu


# 0: every CTA; 3 CTAs have fewer threads than the graphs have edges, so the near
# list is split from the far one, rescanned and compacted
@pytest.mark.parametrize("name", ["aw", "er_config1", "cl5k", "cl20k"])
@pytest.mark.parametrize("ctas,wide", [(0, "0"), (0, "1"), (3, "0")])
def test_late_ctas(engine, gpu_ctx, name, ctas, wide, monkeypatch):
    gd = load_golden(name)
    gpu_ctx.upload(engine.Graph.from_edges(gd["u"], gd["v"]))
    gpu_ctx.set_peel_ctas(ctas)
    monkeypatch.setenv("BT_MSP_WIDE", wide)
    try:
        for exact, key in ((False, "msp"), (True, "hidx")):
            seen = []
            for late in ("0", "20000", "20000"):
                monkeypatch.setenv("BT_MSP_LATE_NS", late)
                res, levels = gpu_ctx.msp(exact=exact)
                np.testing.assert_array_equal(res.astype(np.uint64), gd[key])
                st = gpu_ctx.stats()
                seen.append((levels, st[1], st[5]))
            assert seen[0] == seen[1] == seen[2]
    finally:
        gpu_ctx.set_peel_ctas(0)


def test_late_ctas_of_teams(engine, gpu_ctx, monkeypatch):
    from gpu_bitruss_gb300 import gen
    graphs = [engine.Graph.from_edges(*gen.er(m // 10 + 2, m // 8 + 2, m, seed=m)) for m in (9000, 40, 3000, 500, 5000, 77)]
    want = []
    for g in graphs:
        gpu_ctx.upload(g)
        want.append(gpu_ctx.msp())
    monkeypatch.setenv("BT_MSP_LATE_NS", "20000")
    for ctas in (0, 7):
        gpu_ctx.set_peel_ctas(ctas)
        try:
            res, levels = gpu_ctx.msp_batch(graphs)
        finally:
            gpu_ctx.set_peel_ctas(0)
        for i, (values, lv) in enumerate(want):
            np.testing.assert_array_equal(res[i], values)
            assert int(levels[i]) == lv
