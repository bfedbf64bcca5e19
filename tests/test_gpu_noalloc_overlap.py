"""Allocation-free counts that overlap on the GPU race on the library's scratch:
their counts may be wrong.  They still end, stay inside the scratch and the
callers' buffers, and leave later calls right."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_overlapping_calls_leave_later_ones_right(engine, oracle_mod):
    torch = pytest.importorskip("torch")
    from gpu_bitruss_gb300 import gen
    # renumbered by degree (few and many vertices, hubs), and by counters
    lists = [gen.er(3000, 4000, 60_000, seed=1), gen.hub_skew(60, 30_000, 80_000, 1.8, 4000.0, seed=2),
             gen.er(90_000, 90_000, 200_000, seed=3), gen.er(900, 700, 9000, seed=4)]
    calls, want = [], []
    guard = 1 << 16
    for u, v in lists:
        g = engine.Graph.from_edges(u, v)
        want.append(oracle_mod.ebfc(oracle_mod.build_csr(u, v), 0)[1])
        bufs = []
        for a in (g.offsets, g.neighbors):  # each buffer with a margin on both sides that must not change
            t = torch.full((a.size + 2 * guard,), 0x5A5A5A5A, dtype=torch.int32)
            t[guard:guard + a.size] = torch.from_numpy(a.view(np.int32))
            bufs.append(t.cuda())
        calls.append((g, bufs, torch.zeros(1, dtype=torch.int64, device="cuda"), torch.cuda.Stream()))

    def call(k, stream):
        g, (off, nbr), out, _ = calls[k]
        engine.bfc_noalloc(0, off.data_ptr() + 4 * guard, nbr.data_ptr() + 4 * guard, g.n, g.m, out.data_ptr(), stream)

    before = [[b.clone() for b in c[1]] for c in calls]
    torch.cuda.synchronize()
    for _ in range(100):
        for k in range(len(calls)):
            call(k, calls[k][3].cuda_stream)
    torch.cuda.synchronize()
    for k in range(len(calls)):
        call(k, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert int(calls[k][2].item()) == want[k]
        for b, was in zip(calls[k][1], before[k]):
            assert torch.equal(b, was)
