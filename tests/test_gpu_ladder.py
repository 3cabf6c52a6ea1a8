"""Single-source SSSP on graphs with hubs around the size from which it relaxes by a ladder of thresholds (650,000 vertices
and 10 M arcs), against Dijkstra, bit for bit: weights of 0, equal weights, weights so small that the first threshold is
1, large and skewed ones, a source without arcs, one that reaches little, unaligned labels, an iteration cap and an
explicit solution on the same graph."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import dpg

pytestmark = pytest.mark.gpu


def _graph(V, E, weights, seed, hub=4000):
    """E arcs: half of them out of `hub` hubs, a chain through the last 300 vertices, which only vertex 5 enters."""
    rng = np.random.default_rng(seed)
    body = V - 300
    n = E - 300
    src = np.where(rng.random(n) < 0.5, rng.integers(0, hub, n), rng.integers(0, body, n))
    dst = rng.integers(0, body, n)
    src[src == 17] = 18  # 17 has no out-arcs
    src = np.concatenate([src, [5], np.arange(body, V - 1)])
    dst = np.concatenate([dst, [body], np.arange(body + 1, V)])
    return dpg.csr_from_arcs(V, src, dst, weights(rng, len(src)).astype(np.int32))


KINDS = {
    "ordinary": lambda rng, n: rng.integers(1, 256, n),
    "zeros": lambda rng, n: rng.integers(0, 3, n),
    "equal": lambda rng, n: np.ones(n),
    "large": lambda rng, n: rng.integers(1, 3_000_000, n),
    "skewed": lambda rng, n: np.where(rng.random(n) < 0.001, 1_000_000, rng.integers(1, 10, n)),
}


@pytest.mark.parametrize(
    "kind, V, E", [("ordinary", 650_000, 9_999_999), ("ordinary", 649_999, 10_000_000), ("ordinary", 700_001, 11_000_001)]
    + [(k, 650_000, 10_000_000) for k in KINDS])
def test_ladder(ctx, orc, kind, V, E):
    import torch

    g = _graph(V, E, KINDS[kind], E)
    assert g.E == E
    dg = dpg.Graph(ctx, g.offsets, g.col, g.weights)
    for source in (0, 5, 17, 60_000, V - 200):
        want = orc.sssp_dijkstra(g.offsets, g.col, g.weights, source)
        assert np.array_equal(dpg.sssp(ctx, dg, source), want), source
    want = orc.sssp_dijkstra(g.offsets, g.col, g.weights, 0)
    buf = torch.full((V + 3,), -7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    dpg.sssp_dev(ctx, dg, 0, buf.data_ptr() + 4)
    ctx.synchronize()
    assert buf[0] == -7 and bool((buf[V + 1:] == -7).all())
    assert np.array_equal(buf[1:V + 1].cpu().numpy(), want)
    assert np.array_equal(dpg.sssp(ctx, dg, 0, max_iterations=V + 2), want)
    assert np.array_equal(dpg.sssp(ctx, dg, 0, solution=dpg.SOL_BINNED), want)
