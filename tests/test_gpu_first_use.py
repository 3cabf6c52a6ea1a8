"""What a graph keeps (row plan, renaming, renamed columns, merge items, permutation) is built by the first call that needs
it and then read by calls on other streams and by captured ones. Results are bit-equal however a call comes to it."""
from __future__ import annotations

from contextlib import contextmanager

import numpy as np
import pytest

from conftest import dpg

pytestmark = pytest.mark.gpu

PR = dict(damping=0.85, total_rank=1.0, iterations=7)


class _Problem:
    def __init__(self, ctx, seed=5):
        import torch

        V = 20_011
        rng = np.random.default_rng(seed)
        src = np.concatenate([rng.integers(0, V, 6 * V), rng.integers(0, 40, 3 * V)])
        g = dpg.csr_from_arcs(V, src, rng.permutation(len(src)) % V)
        in_off, in_col = dpg.csr_transpose(V, g.offsets, g.col)
        self.ctx, self.V, self.E = ctx, V, len(src)
        self.csr = in_off, in_col
        self.od = torch.from_numpy(np.diff(g.offsets).astype(np.int32)).cuda()
        self.vals = torch.from_numpy(rng.uniform(0.5, 1.5, self.E).astype(np.float32)).cuda()
        self.x = torch.from_numpy(rng.uniform(-1, 1, V).astype(np.float32)).cuda()
        self.want = {}
        g = self.graph()
        for what in ("pagerank", "spmv"):
            out = self.out()
            self.call(what, g, out)
            ctx.synchronize()
            self.want[what] = out
        torch.cuda.synchronize()

    def graph(self):
        return dpg.Graph(self.ctx, *self.csr)

    def out(self):
        import torch

        t = torch.full((self.V,), -7.0, device="cuda")
        torch.cuda.synchronize()
        return t

    def call(self, what, g, out):
        if what == "pagerank":
            dpg.pagerank_dev(self.ctx, g, self.od.data_ptr(), out.data_ptr(), **PR)
        else:
            dpg.spmv_dev(self.ctx, g, self.vals.data_ptr(), self.x.data_ptr(), out.data_ptr())

    def check(self, what, g):
        import torch

        out = self.out()
        self.call(what, g, out)
        self.ctx.synchronize()
        assert torch.equal(out, self.want[what]), what


@pytest.fixture
def prob(ctx):
    return _Problem(ctx)


@contextmanager
def _on(ctx, stream):
    ctx.set_stream(stream.cuda_stream)
    try:
        yield
    finally:
        import torch

        torch.cuda.synchronize()
        ctx.set_stream(None)


def _capture(prob, what, g, out, stream, mode="global"):
    import torch

    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode=mode):
        prob.call(what, g, out)
    return graph


def _replay(prob, what, graph, out):
    import torch

    out.fill_(-7)
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, prob.want[what]), what


@pytest.mark.parametrize("what", ["pagerank", "spmv"])
@pytest.mark.parametrize("relabel", [True, False])
def test_a_capture_survives_the_other_choice_of_renaming(prob, what, relabel):
    import torch

    stream = torch.cuda.Stream()
    g = prob.graph()
    with _on(prob.ctx, stream):
        g.set_relabel(relabel)
        prob.check(what, g)
        out = prob.out()
        graph = _capture(prob, what, g, out, stream)
        for other in (not relabel, relabel, not relabel):
            g.set_relabel(other)
            prob.check(what, g)
            _replay(prob, what, graph, out)
