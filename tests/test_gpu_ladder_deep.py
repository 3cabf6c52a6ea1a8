"""Single-source SSSP by a ladder of thresholds (650,000 vertices and 10 M arcs up) on graphs that have both hubs and a high
diameter: long chains before the first hub, behind the hubs and between two cores of hubs, so that the ladder begins
late, runs dry between hubs and ends ahead of the chains. Against Dijkstra, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import dpg

pytestmark = pytest.mark.gpu

V, E, CHAIN = 660_001, 10_200_000, 1500


def _graph(weights, chain_weight, seed):
    """Two cores with hubs of their own. Chains: a (into core 1), b (core 1 to core 2), c (out of core 2); a grid of 40 x
    1,000 hangs off core 1's first hub. Returns the graph and the first vertices of a, b, c and the grid."""
    rng = np.random.default_rng(seed)
    rows, cols = 40, 1000
    fixed = 3 * CHAIN + rows * cols
    core = (V - fixed) // 2
    a, b, c = (2 * core + k * CHAIN for k in range(3))
    grid = 2 * core + 3 * CHAIN
    src, dst, w = [], [], []

    def add(s, d, ws):
        src.append(np.asarray(s))
        dst.append(np.asarray(d))
        w.append(np.broadcast_to(np.asarray(ws), np.shape(s)))

    for first in (a, b, c):
        add(np.arange(first, first + CHAIN - 1), np.arange(first + 1, first + CHAIN), chain_weight)
    add([a + CHAIN - 1, 3, b + CHAIN - 1, core + 3, 0], [7, b, core + 9, c, grid], chain_weight)
    v = np.arange(rows * cols).reshape(rows, cols) + grid
    for s, d in ((v[:, :-1], v[:, 1:]), (v[:, 1:], v[:, :-1]), (v[:-1], v[1:]), (v[1:], v[:-1])):
        add(s.ravel(), d.ravel(), rng.integers(1, 1000, s.size))
    n = E - sum(len(s) for s in src)
    side = rng.integers(0, 2, n) * core
    s = np.where(rng.random(n) < 0.5, rng.integers(0, 800, n), rng.integers(0, core, n)) + side
    add(s, rng.integers(0, core, n) + side, weights(rng, n))
    src, dst, w = (np.concatenate(x) for x in (src, dst, w))
    return dpg.csr_from_arcs(V, src, dst, w.astype(np.int32)), (a, b, c, grid)


@pytest.mark.parametrize("kind, weights, chain_weight", [
    ("ordinary", lambda rng, n: rng.integers(1, 256, n), 40),
    ("long_chains", lambda rng, n: rng.integers(1, 256, n), 100_000),
    ("unit", lambda rng, n: np.ones(n, int), 1),
    ("zeros", lambda rng, n: rng.integers(0, 3, n), 0),
])
def test_hubs_and_high_diameter(ctx, orc, kind, weights, chain_weight):
    g, (a, b, c, grid) = _graph(weights, chain_weight, len(kind))
    assert (g.V, g.E) == (V, E)
    dg = dpg.Graph(ctx, g.offsets, g.col, g.weights)
    for source in (a, a + CHAIN - 2, 0, 1000, b, grid + 500, c):
        assert np.array_equal(dpg.sssp(ctx, dg, source), orc.sssp_dijkstra(g.offsets, g.col, g.weights, source)), source
