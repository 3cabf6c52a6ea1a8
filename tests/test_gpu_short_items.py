"""Backward of more than 32 columns on small matrices, whose long rows are cut into items of 64, 128 or 256 nonzeros (512 on
large ones) and added up in a tree of eight: rows around the items' limits and hubs of up to all arcs. Bound as in
test_gpu_rows: sums of products within 1e-5 of their |terms|; against items of 512 (the plan that a captured first call
has to use) no further from FP64 beyond rounding."""
from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp

from conftest import dpg

pytestmark = pytest.mark.gpu

TOL = 1e-5
LENGTHS = [1, 63, 64, 65, 127, 128, 129, 191, 255, 256, 257, 511, 512, 513, 1023, 1025, 2047, 4097, 9000]


def _graph(E, hub, seed):
    """Column lengths LENGTHS, one column of `hub` arcs, the rest uniform: E arcs over 3,001 vertices."""
    rng = np.random.default_rng(seed)
    V = 3001
    dst = np.concatenate([np.full(n, k) for k, n in enumerate(LENGTHS)] + [np.full(hub, 2000)])
    assert len(dst) <= E
    dst = np.concatenate([dst, rng.integers(100, V, E - len(dst))])
    src = rng.integers(0, V, E)
    name = rng.permutation(V)
    return dpg.csr_from_arcs(V, name[src], name[dst])


# Arcs that give items of 64, 128, 256 and 512 on 152 SMs; a hub of nearly all arcs among them.
@pytest.mark.parametrize("E, hub", [(40_000, 5_000), (311_000, 280_000), (640_000, 1_000), (1_300_000, 1_200_000),
                                    (2_600_000, 2_400_000)])
@pytest.mark.parametrize("nrhs", [36, 64, 100, 128])
def test_backward(ctx, E, hub, nrhs):
    import torch

    g = _graph(E, hub, E + nrhs)
    rng = np.random.default_rng(nrhs)
    vals = np.exp(rng.normal(0, 1, E)).astype(np.float32)
    X, G = (rng.uniform(-1, 1, (g.V, nrhs)).astype(np.float32) for _ in range(2))
    tv, tX, tG = (torch.from_numpy(a).cuda() for a in (vals, X, G))

    def run(dg):
        dX = torch.full((g.V, nrhs), float("nan"), device="cuda")
        dA = torch.full((E,), float("nan"), device="cuda")
        torch.cuda.synchronize()
        dpg.spmv_bwd_dev(ctx, dg, tv.data_ptr(), nrhs, tX.data_ptr(), tG.data_ptr(), dX.data_ptr(), dA.data_ptr())
        ctx.synchronize()
        return dX.cpu().numpy(), dA.cpu().numpy()

    dg = dpg.Graph(ctx, g.offsets, g.col)
    dX, dA = run(dg)
    A = sp.csr_matrix((vals.astype(np.float64), g.col.copy(), g.offsets.copy()), shape=(g.V, g.V))
    want, terms = A.T @ G.astype(np.float64), abs(A).T @ np.abs(G.astype(np.float64))
    assert np.all(np.abs(dX - want) <= TOL * terms)
    row = np.repeat(np.arange(g.V), np.diff(g.offsets))
    for a in range(0, E, 1 << 19):
        e = slice(a, a + (1 << 19))
        p = G[row[e]].astype(np.float64) * X[g.col[e]]
        assert np.all(np.abs(dA[e] - p.sum(1)) <= TOL * np.abs(p).sum(1))
    dX2, dA2 = run(dg)
    assert np.array_equal(dX, dX2) and np.array_equal(dA, dA2)

    # Items of 512: a graph whose first wide backward is captured (the narrow one before it made that plan).
    stream = torch.cuda.Stream()
    long = dpg.Graph(ctx, g.offsets, g.col)
    out = torch.empty((g.V, nrhs), device="cuda")
    torch.cuda.synchronize()
    ctx.set_stream(stream.cuda_stream)
    try:
        dpg.spmv_bwd_dev(ctx, long, tv.data_ptr(), 1, tX.data_ptr(), tG.data_ptr(), out.data_ptr(), None)
        ctx.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            dpg.spmv_bwd_dev(ctx, long, tv.data_ptr(), nrhs, tX.data_ptr(), tG.data_ptr(), out.data_ptr(), None)
        graph.replay()
        torch.cuda.synchronize()
    finally:
        ctx.set_stream(None)
    err, err512 = (np.linalg.norm(d - want) / np.linalg.norm(want) for d in (dX, out.cpu().numpy()))
    assert err <= err512 * 1.05 + 1e-9, (err, err512)


@pytest.mark.parametrize("nrhs", [1, 3, 32, 36, 64])
def test_captured_after_a_wide_call(ctx, nrhs):
    """A graph whose only backward so far was of 64 columns: a captured one of any width takes the plan that is there."""
    import torch

    g = _graph(60_000, 20_000, 9)
    rng = np.random.default_rng(4)
    tv = torch.from_numpy(rng.uniform(0.5, 1.5, g.E).astype(np.float32)).cuda()
    X, G = (torch.from_numpy(rng.uniform(-1, 1, (g.V, 64)).astype(np.float32)).cuda() for _ in range(2))
    x, gg = X[:, :nrhs].contiguous(), G[:, :nrhs].contiguous()
    dX64, dA = torch.empty_like(X), torch.empty(g.E, device="cuda")
    dX, dAn = torch.full_like(x, -7), torch.full_like(dA, -7)
    torch.cuda.synchronize()
    dg = dpg.Graph(ctx, g.offsets, g.col)
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    try:
        dpg.spmv_bwd_dev(ctx, dg, tv.data_ptr(), 64, X.data_ptr(), G.data_ptr(), dX64.data_ptr(), dA.data_ptr())
        ctx.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            dpg.spmv_bwd_dev(ctx, dg, tv.data_ptr(), nrhs, x.data_ptr(), gg.data_ptr(), dX.data_ptr(),
                             dAn.data_ptr())
        graph.replay()
        torch.cuda.synchronize()
    finally:
        ctx.set_stream(None)
    A = sp.csr_matrix((tv.cpu().numpy().astype(np.float64), g.col.copy(), g.offsets.copy()), shape=(g.V, g.V))
    G64 = gg.cpu().numpy().astype(np.float64)
    assert np.all(np.abs(dX.cpu().numpy() - A.T @ G64) <= TOL * (abs(A).T @ np.abs(G64)))
    row = np.repeat(np.arange(g.V), np.diff(g.offsets))
    p = G64[row] * x.cpu().numpy()[g.col]
    assert np.all(np.abs(dAn.cpu().numpy() - p.sum(1)) <= TOL * np.abs(p).sum(1))
