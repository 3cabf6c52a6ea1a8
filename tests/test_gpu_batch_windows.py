"""Batches large enough for hot-cache windows (8 tiles per warp of the gather, about 10 M merge items) when the cache size
changes between calls: each size has windows of its own, whose addresses a captured solve keeps. The cache size only
decides where a value is read from, so every result is bit-equal to the default's."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import dpg
from test_gpu_sweeps import LENGTHS, SWEEPS, _graph

pytestmark = pytest.mark.gpu

PR = dict(damping=0.85, total_rank=1.0, iterations=SWEEPS)


def _batch(ctx):
    sizes = [300, 5, 60_001, 1, 400_003, 130_001, 33, 800_009]
    gs = []
    for k, V in enumerate(sizes):
        g = _graph(V, LENGTHS[:V], 7, V + k, V // 7)
        gs.append(g._replace(weights=np.random.default_rng(k).integers(1, 100, g.E).astype(np.int32)))
    assert sum(g.V + g.E for g in gs) > 10 << 20
    return gs, dpg.Batch(ctx, gs)


def _tune(b, hot):
    b.tuning = dict(b.tuning, pr_hot=hot)


def test_cache_sizes(ctx):
    import torch

    _, b = _batch(ctx)
    want = None
    for hot in (-1, 0, 1, 4096, 16384, 20_000_000, -1):
        _tune(b, hot)
        rank = torch.full((b.V,), -1.0, device="cuda")
        torch.cuda.synchronize()
        b.pagerank_dev(rank.data_ptr(), **PR)
        ctx.synchronize()
        want = rank if want is None else want
        assert torch.equal(rank, want), hot


def test_replay_after_the_cache_size_changed(ctx):
    import torch

    gs, b = _batch(ctx)
    sources = np.zeros((b.n, 1), np.int32)
    dist = torch.empty(b.V, dtype=torch.int32, device="cuda")
    rank = torch.empty(b.V, device="cuda")

    def run(hot):
        _tune(b, hot)
        dist.fill_(-1)
        rank.fill_(-1)
        torch.cuda.synchronize()
        b.run(sources, dist.data_ptr(), rank.data_ptr(), {}, PR)
        ctx.synchronize()
        return dist.clone(), rank.clone()

    want = run(4096)
    keep = []
    for hot in (0, 16384, -1):
        _tune(b, hot)
        b.pagerank_dev(rank.data_ptr(), **PR)  # windows for this size
        ctx.synchronize()
        # Other users of the freed memory, had any been freed.
        keep += [torch.full((n,), 0x7F7F7F7F, dtype=torch.int32, device="cuda") for n in (16, 64, 256, 1024, 4096)]
        got = run(4096)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]), hot


def test_a_callers_own_capture_survives_another_cache_size(ctx):
    import torch

    _, b = _batch(ctx)
    rank = torch.full((b.V,), -1.0, device="cuda")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    _tune(b, 4096)
    ctx.set_stream(stream.cuda_stream)
    try:
        b.pagerank_dev(rank.data_ptr(), **PR)
        ctx.synchronize()
        want = rank.clone()
        graph = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            b.pagerank_dev(rank.data_ptr(), **PR)
        for hot in (0, -1, 4096):
            _tune(b, hot)
            b.pagerank_dev(rank.data_ptr(), **PR)
            ctx.synchronize()
            keep = [torch.full((n,), 0x7F7F7F7F, dtype=torch.int32, device="cuda") for n in (16, 64, 256, 1024, 4096)]
            rank.fill_(-1)
            torch.cuda.synchronize()
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(rank, want), hot
            del keep
    finally:
        ctx.set_stream(None)
