"""Small frontiers are cut into warp items of 1 to 32 vertices (by the mean degree and the number of idle warps) and
items of at most 32 arcs take a shorter path: distances and levels must stay those of the oracle at the edges."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import dpg

pytestmark = pytest.mark.gpu


def _layers(width: int, degree: int, depth: int, seed: int):
    """A root over `width` vertices, then `depth` layers of `width` vertices with `degree` random arcs each into the
    next layer: every frontier is about `width` vertices of `degree` arcs."""
    rng = np.random.default_rng(seed)
    V = 1 + width * (depth + 1)
    src = [np.zeros(width, np.int64)]
    dst = [1 + np.arange(width)]
    for k in range(depth):
        s = np.repeat(1 + k * width + np.arange(width), degree)
        src.append(s)
        dst.append(1 + (k + 1) * width + rng.integers(0, width, s.size))
    src, dst = np.concatenate(src), np.concatenate(dst)
    return dpg.csr_from_arcs(V, src, dst, rng.integers(0, 50, src.size))


# Degrees around 8 and 32 arcs per item and past the hub threshold of 128; widths around 32, one item per warp
# (3,648 and 4,864 warps) and their doubles.
@pytest.mark.parametrize("width", [1, 31, 33, 3647, 3649, 4865, 9731])
@pytest.mark.parametrize("degree", [1, 2, 7, 9, 31, 33, 130])
def test_layers(ctx, orc, width, degree):
    g = _layers(width, degree, 3, seed=width * 1000 + degree)
    dg = dpg.Graph(ctx, g.offsets, g.col, g.weights)
    want = orc.sssp_dijkstra(g.offsets, g.col, g.weights, 0)
    for solution in (dpg.SOL_BINNED, dpg.SOL_NEARFAR):
        assert np.array_equal(dpg.sssp(ctx, dg, 0, solution=solution), want)
    assert np.array_equal(dpg.bfs(ctx, dg, 0), orc.bfs(g.offsets, g.col, 0))


# Warps going on with their own improvements (near-far, small iterations): chains, rings with shortcuts that improve
# labels late, rows that do not fit beside another in one arc per lane, thresholds that send everything or nothing to
# the far pile, zero weights. An iteration cap turns it off; the distances are the same.
@pytest.mark.parametrize("delta", [1, 60, 10**9])
@pytest.mark.parametrize("degree", [1, 4, 16, 17, 33])
def test_warps_go_on_with_their_own_improvements(ctx, orc, degree, delta):
    rng = np.random.default_rng(degree)
    V = 6000
    v = np.arange(V)
    src = np.concatenate([v[:-1], np.repeat(v, degree), [0, 17]])
    dst = np.concatenate([v[1:], np.clip(np.repeat(v, degree) + rng.integers(-40, 41, V * degree), 0, V - 1), [V - 1, 17]])
    w = np.concatenate([rng.integers(0, 3, V - 1), rng.integers(0, 90, V * degree), [2000, 0]])
    g = dpg.csr_from_arcs(V, src, dst, w)
    dg = dpg.Graph(ctx, g.offsets, g.col, g.weights)
    for source in (0, 17, V - 1):
        want = orc.sssp_dijkstra(g.offsets, g.col, g.weights, source)
        assert np.array_equal(dpg.sssp(ctx, dg, source, solution=dpg.SOL_NEARFAR, delta=delta), want)
        capped = dpg.sssp(ctx, dg, source, solution=dpg.SOL_NEARFAR, delta=delta, max_iterations=1 << 30)
        assert np.array_equal(capped, want)


def _chain_then(tail: str, seed: int):
    """A chain of 100 levels with side branches and back arcs (past the iteration from which levels are relaxed in any
    order), then a grid (long paths of differing length) or a random graph whose frontier grows large."""
    rng = np.random.default_rng(seed)
    n = 100
    src, dst = [np.arange(n)], [np.arange(1, n + 1)]
    if tail == "grid":
        rows, cols = 60, 211
        s, d, _ = dpg.grid_arcs(rows, cols, 1)
        keep = rng.random(s.size) < 0.85  # holes: shortest paths bend, some vertices are unreachable
        s, d, V = s[keep] + n, d[keep] + n, n + rows * cols
    else:
        V = n + 150_000
        s, d = rng.integers(n, V, 6 * 150_000), rng.integers(n, V, 6 * 150_000)
    back = rng.integers(0, n, 50)
    src += [s, back, back, [n]]
    dst += [d, np.maximum(back - rng.integers(0, 9, 50), 0), n + rng.integers(0, 20, 50), [n]]
    src, dst = np.concatenate(src), np.concatenate(dst)
    return dpg.csr_from_arcs(V, src, dst, rng.integers(0, 9, src.size))


@pytest.mark.parametrize("tail", ["grid", "random"])
@pytest.mark.parametrize("seed", range(4))
def test_levels_of_long_graphs(ctx, orc, tail, seed):
    g = _chain_then(tail, seed)
    dg = dpg.Graph(ctx, g.offsets, g.col, g.weights)
    for source in (0, 50, 99):
        want = orc.bfs(g.offsets, g.col, source)
        assert np.array_equal(dpg.bfs(ctx, dg, source), want)
        assert np.array_equal(dpg.bfs(ctx, dg, source, max_iterations=1 << 30), want)
        assert np.array_equal(dpg.sssp(ctx, dg, source), orc.sssp_dijkstra(g.offsets, g.col, g.weights, source))


def test_iteration_cap_still_counts_levels(ctx):
    g = dpg.csr_from_arcs(301, np.arange(300), np.arange(1, 301), np.ones(300))
    dg = dpg.Graph(ctx, g.offsets, g.col, g.weights)
    with pytest.raises(dpg.DpgError):
        dpg.bfs(ctx, dg, 0, max_iterations=200)
    assert np.array_equal(dpg.bfs(ctx, dg, 0, max_iterations=302), np.arange(301))
    assert np.array_equal(dpg.bfs(ctx, dg, 0), np.arange(301))
