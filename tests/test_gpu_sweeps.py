"""The sweeps over item streams (PageRank, weighted PageRank, the batch) and the tiled SpMV, at the edges of their layout:
tiles of 256 merge items that hold only empty rows, rows one short of, at and past the hub line (255 nonzeros) and its
segments, vertex counts around a tile and a block, ranks too few and too many for the shared-memory cache, batches with
and without cache windows. Bound: a sweep's row is a tree over lane sums of at most 8 products and fixed-order hub
segments, all terms positive, so its relative error is a few tens of 2^-24, and damping keeps 20 sweeps' total below
1 / (1 - d) = 6.7 times that: within 1e-5 of FP64, as required elsewhere. Repeated calls are bit-equal: the sweeps are
launched as a chain, each reading what the one before it wrote."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import dpg
from test_gpu_prgrad import CONV, _check_vs_fp64, _run

pytestmark = pytest.mark.gpu
TOL = 1e-5
SWEEPS = 20
LENGTHS = [1, 2, 7, 8, 9, 31, 32, 33, 253, 254, 255, 256, 257, 509, 510, 511, 512, 513, 1023, 2039, 2040, 2041, 2049,
           5000]


def _graph(V, lengths, ef, seed, empty=0):
    """`empty` rows without in-arcs first, then one row of each given length, then uniform arcs over the other rows."""
    rng = np.random.default_rng(seed)
    src, dst = [], []
    rows = empty + np.arange(len(lengths)) * max(1, (V - empty) // max(1, 2 * len(lengths)))
    for v, n in zip(rows[rows < V], lengths):
        src.append(rng.integers(0, V, n))
        dst.append(np.full(n, v))
    if V > empty:
        src.append(rng.integers(0, V, ef * V))
        dst.append(rng.integers(empty, V, ef * V))
    src, dst = np.concatenate(src or [[0]]), np.concatenate(dst or [[0]])
    return dpg.csr_from_arcs(V, src, dst, np.ones(len(src), np.int32))


CASES = {
    "one": (1, [], 0, 0),
    "31": (31, [1, 40], 1, 0),
    "tile_of_empty_rows": (700, [300], 1, 512),
    "255": (255, [], 0, 0),
    "256": (256, [256], 1, 0),
    "257": (257, [257], 1, 1),
    "lengths": (4097, LENGTHS, 2, 0),
    "lengths_shifted": (4097, LENGTHS, 2, 257),
    "past_the_cache": (60_001, LENGTHS * 3, 6, 1000),
    "many_tiles": (1_000_003, LENGTHS * 20, 3, 100_000),
}


@pytest.mark.parametrize("name", CASES)
def test_sweeps(ctx, orc, name):
    V, lengths, ef, empty = CASES[name]
    g = _graph(V, lengths, ef, len(name), empty)
    in_off, in_col = dpg.csr_transpose(g.V, g.offsets, g.col)
    od = np.diff(g.offsets).astype(np.int32)
    dg = dpg.Graph(ctx, in_off, in_col)
    r64, _ = orc.pagerank_f64(in_off, in_col, od, damping=0.85, total=1.0, iterations=SWEEPS)
    first = dpg.pagerank(ctx, dg, od, damping=0.85, total_rank=1.0, iterations=SWEEPS)
    assert np.all(np.abs(first - r64) <= TOL * r64)
    for _ in range(5):
        assert np.array_equal(first, dpg.pagerank(ctx, dg, od, damping=0.85, total_rank=1.0, iterations=SWEEPS))
    tol = dict(damping=0.85, total_rank=1.0, iterations=200, epsilon=1e-7)
    r64, _ = orc.pagerank_f64(in_off, in_col, od, damping=0.85, total=1.0, iterations=200)
    a, b = (dpg.pagerank(ctx, dg, od, **tol) for _ in range(2))
    assert np.array_equal(a, b)
    # The last change of any rank is at most epsilon: at most epsilon d / (1 - d) in the 1-norm's decay per vertex.
    assert np.all(np.abs(a - r64) <= TOL * r64 + V * 1e-7 * 0.85 / 0.15)

    rng = np.random.default_rng(7)
    vals = rng.uniform(0.5, 1.5, g.E).astype(np.float32)
    x = rng.uniform(-1, 1, g.V).astype(np.float32)
    y = dpg.spmv(ctx, dg, vals, x)
    y64, ay = orc.spmv_f32in(in_off, in_col, vals, x)
    assert np.all(np.abs(y.astype(np.float64) - y64) <= TOL * np.maximum(ay, np.finfo(np.float32).tiny))
    assert np.array_equal(y, dpg.spmv(ctx, dg, vals, x))


@pytest.mark.parametrize("name", ["31", "tile_of_empty_rows", "257", "lengths", "lengths_shifted"])
def test_weighted_sweeps(ctx, name):
    V, lengths, ef, empty = CASES[name]
    g = _graph(V, lengths, ef, len(name), empty)
    rng = np.random.default_rng(11)
    w = rng.uniform(0.1, 2.0, g.E).astype(np.float32)
    seed = (rng.random(g.V) < 0.1).astype(np.float32)
    seed[0] = 1
    r, gr, n = _run(ctx, g, w, seed, **CONV)
    _check_vs_fp64(g, w, seed, r, gr)
    r2, gr2, n2 = _run(ctx, g, w, seed, **CONV)
    assert np.array_equal(r, r2) and np.array_equal(gr, gr2) and n == n2


# 8 tiles per warp (about 10 M merge items) is the line from which a batch's gather goes window by window: graphs that
# share a window, graphs larger than the cache, single vertices between them, the first and last graph of either kind.
@pytest.mark.parametrize("order", ["small", "large_first", "large_last"])
def test_batch_windows(ctx, orc, order):
    import torch

    sizes = [1, 255, 5, 3000, 256, 1, 20_001, 700, 44_444, 60_001, 1, 257, 513, 9000]
    if order != "small":
        sizes = sizes + [400_003, 130_001, 2, 1, 33, 800_009]
    if order == "large_first":
        sizes = sizes[::-1]
    gs = [_graph(V, LENGTHS[:V], 8 if V < 100_000 else 6, V + k, V // 7) for k, V in enumerate(sizes)]
    if order == "small":
        assert sum(g.V + g.E for g in gs) < 8 << 20
    else:
        assert sum(g.V + g.E for g in gs) > 10 << 20
    b = dpg.Batch(ctx, gs)
    rank = torch.empty(b.V, device="cuda")
    b.pagerank_dev(rank.data_ptr(), damping=0.85, total_rank=1.0, iterations=SWEEPS)
    ctx.synchronize()
    r = rank.cpu().numpy()
    for k, g in enumerate(gs):
        v0, v1 = int(b.vstart[k]), int(b.vstart[k + 1])
        in_off, in_col = dpg.csr_transpose(g.V, g.offsets, g.col)
        od = np.diff(g.offsets).astype(np.int32)
        r64, _ = orc.pagerank_f64(in_off, in_col, od, damping=0.85, total=1.0, iterations=SWEEPS)
        assert np.all(np.abs(r[v0:v1] - r64) <= TOL * r64), k
    for _ in range(3):
        again = torch.empty_like(rank)
        b.pagerank_dev(again.data_ptr(), damping=0.85, total_rank=1.0, iterations=SWEEPS)
        ctx.synchronize()
        assert torch.equal(again, rank)
