"""Y = A X and its adjoint over the widths and row lengths where the row kernel changes its layout: lanes per row (powers
of two of float4 vectors or single floats), groups per warp, arcs per step, rows at the limit of a group (64 nonzeros)
and of a listed item (512), 16-byte aligned row blocks or not. Bound: every result is a sum of n <= 1,300 products in
FP32, so within (n + 1) * 2^-24 < 1e-4 of its sum of |terms|; the fixed trees of 8-lane groups do far better, 1e-5 is
required as elsewhere."""
from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp

from conftest import dpg

pytestmark = pytest.mark.gpu

TOL = 1e-5
LENGTHS = [0, 1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 66, 127, 128, 511, 512, 513, 1024, 1025, 1300]


@pytest.fixture(scope="module")
def graph():
    """Every row length above, in rows and (as the last 1,000 vertices' arcs turned round) in columns, shuffled."""
    rng = np.random.default_rng(3)
    V = 1500
    src, dst = [], []
    for k, n in enumerate(LENGTHS * 3):
        src.append(np.full(n, k))
        dst.append(rng.integers(0, V, n))
        src.append(rng.integers(0, V, n))
        dst.append(np.full(n, 200 + k))
    src, dst = np.concatenate(src), np.concatenate(dst)
    name = rng.permutation(V)
    return dpg.csr_from_arcs(V, name[src], name[dst])


@pytest.mark.parametrize("nrhs", [1, 2, 3, 4, 5, 8, 9, 16, 17, 20, 32, 33, 36, 64, 68, 96, 100, 127, 128])
@pytest.mark.parametrize("shift", [0, 1])
def test_widths(ctx, graph, nrhs, shift):
    import torch

    g = graph
    rng = np.random.default_rng(nrhs)
    dev = torch.device("cuda", 0)
    vals = np.exp(rng.normal(0, 1, g.E)).astype(np.float32)
    X = rng.uniform(-1, 1, (g.V, nrhs)).astype(np.float32)
    G = rng.uniform(-1, 1, (g.V, nrhs)).astype(np.float32)

    def block(a=None):
        t = torch.full((g.V * nrhs + shift,), float("nan"), device=dev)
        if a is not None:
            t[shift:] = torch.from_numpy(a.ravel()).to(dev)
        return t[shift:]

    tv = torch.from_numpy(vals).to(dev)
    tX, tG, Y, dX, dX2 = block(X), block(G), block(), block(), block()
    dA = torch.full((g.E,), float("nan"), device=dev)
    dA2 = dA.clone()
    dg = dpg.Graph(ctx, g.offsets, g.col)
    dpg.spmm_dev(ctx, dg, tv.data_ptr(), nrhs, tX.data_ptr(), Y.data_ptr())
    dpg.spmv_bwd_dev(ctx, dg, tv.data_ptr(), nrhs, tX.data_ptr(), tG.data_ptr(), dX.data_ptr(), dA.data_ptr())
    dpg.spmv_bwd_dev(ctx, dg, tv.data_ptr(), nrhs, None, tG.data_ptr(), dX2.data_ptr(), None)
    dpg.spmv_bwd_dev(ctx, dg, tv.data_ptr(), nrhs, tX.data_ptr(), tG.data_ptr(), None, dA2.data_ptr())
    ctx.synchronize()
    A = sp.csr_matrix((vals.astype(np.float64), g.col.copy(), g.offsets.copy()), shape=(g.V, g.V))
    Aa = abs(A)
    X64, G64 = X.astype(np.float64), G.astype(np.float64)
    rows = np.repeat(np.arange(g.V), np.diff(g.offsets))

    def close(got, want, size):
        got = got.cpu().numpy().reshape(want.shape)
        assert np.all(np.abs(got - want) <= TOL * size + 1e-30)

    close(Y, A @ X64, Aa @ np.abs(X64))
    for t in (dX, dX2):
        close(t, A.T @ G64, Aa.T @ np.abs(G64))
    for t in (dA, dA2):
        prod = G64[rows] * X64[g.col]
        close(t, prod.sum(1), np.abs(prod).sum(1))


# From 3 x 2^22 arcs up the backward permutes the values to transposed order and dA back, in blocks of 24,576: a full
# last block, one of a single arc, one short of it, and one arc less than the line. dX sums up to about 1,200 products, dA is one product of nrhs = 1.
@pytest.mark.parametrize("E", [(3 << 22) - 1, 3 << 22, 1366 * 24576 - 1, 1366 * 24576, 1366 * 24576 + 1])
def test_permuted_values(ctx, E):
    import torch

    dev = torch.device("cuda", 0)
    gen = torch.Generator(device=dev)
    gen.manual_seed(E)
    V = 40_009
    row, _ = torch.sort(torch.randint(0, V, (E,), device=dev, generator=gen, dtype=torch.int32))
    col = torch.randint(0, V, (E,), device=dev, generator=gen, dtype=torch.int32)
    off = torch.zeros(V + 1, dtype=torch.int32, device=dev)
    off[1:] = torch.cumsum(torch.bincount(row, minlength=V), 0)
    vals = torch.rand(E, device=dev, generator=gen)
    X, G = (torch.rand(V, 1, device=dev, generator=gen) - 0.5 for _ in range(2))
    dX, dA = torch.empty_like(X), torch.empty_like(vals)
    torch.cuda.synchronize()
    dg = dpg.Graph.from_device(ctx, V, E, off.data_ptr(), col.data_ptr())
    dpg.spmv_bwd_dev(ctx, dg, vals.data_ptr(), 1, X.data_ptr(), G.data_ptr(), dX.data_ptr(), dA.data_ptr())
    ctx.synchronize()
    r, c = row.long(), col.long()
    assert torch.equal(dA, G[r, 0] * X[c, 0])  # one product each, correctly rounded
    terms = vals.double() * G[r, 0].double()
    want = torch.zeros(V, dtype=torch.float64, device=dev).index_add_(0, c, terms)
    size = torch.zeros(V, dtype=torch.float64, device=dev).index_add_(0, c, terms.abs())
    assert bool(((dX[:, 0].double() - want).abs() <= TOL * size).all())
