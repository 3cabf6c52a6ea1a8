"""PageRank to a tolerance: stops at the right sweep, with that sweep's ranks. The tolerance is set against the mean rank 1 / V,
so that every size runs several sweeps. Bound: a rank of either side's sweep n is within TOL of FP64's (test_gpu_sweeps),
so a change between two sweeps is within 2 TOL r of FP64's, and the verdict can differ from FP64's only where the change
is that close to epsilon; the ranks returned are those of the sweep count that the call reports, within TOL."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import dpg
from test_gpu_sweeps import CASES, TOL, _graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", CASES)
def test_stops_at_the_right_sweep(ctx, orc, name):
    V, lengths, ef, empty = CASES[name]
    g = _graph(V, lengths, ef, len(name), empty)
    in_off, in_col = dpg.csr_transpose(g.V, g.offsets, g.col)
    od = np.diff(g.offsets).astype(np.int32)
    dg = dpg.Graph(ctx, in_off, in_col)

    def r64(n):
        return orc.pagerank_f64(in_off, in_col, od, damping=0.85, total=1.0, iterations=n)[0]

    counts = []
    for share in (0.3, 0.03, 3e-3, 5e-4):
        opts = dict(damping=0.85, total_rank=1.0, iterations=200, epsilon=share / V)
        a = dpg.pagerank(ctx, dg, od, **opts)
        n = ctx.last_stats().iterations
        counts.append(n)
        now, before = r64(n), r64(n - 1)
        assert np.all(np.abs(a - now) <= TOL * now), share
        assert np.all(np.abs(now - before) <= share / V + 2 * TOL * now), (share, n)
        if n > 1:  # the sweep before was not the last
            assert np.any(np.abs(before - r64(n - 2)) > share / V - 2 * TOL * before), (share, n)
        again = dpg.pagerank(ctx, dg, od, **opts)
        assert ctx.last_stats().iterations == n and np.array_equal(a, again)
        host = dpg.pagerank_host(ctx, in_off, in_col, od, **opts)
        assert ctx.last_stats().iterations == n and np.array_equal(a, host)
    assert counts == sorted(counts) and counts[-1] < 200
    if V >= 256:
        assert counts[-1] >= 5
    # The cap comes first (but a graph of one loop and no other arc starts at its fixed point, 1 / V).
    a = dpg.pagerank(ctx, dg, od, damping=0.85, total_rank=1.0, iterations=2, epsilon=1e-30)
    assert ctx.last_stats().iterations == (2 if ef or lengths else 1)
    now = r64(ctx.last_stats().iterations)
    assert np.all(np.abs(a - now) <= TOL * now)
