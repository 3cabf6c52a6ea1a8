"""What a graph keeps (row plan, renaming, renamed columns, merge items, permutation) is built by the first call that needs
it and then read by calls on other streams and by captured ones. Results are bit-equal however a call comes to it."""
from __future__ import annotations

import subprocess
import sys
from contextlib import contextmanager

import numpy as np
import pytest

from conftest import ROOT, dpg

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


@pytest.mark.parametrize("what, warm", [("pagerank", "spmv"), ("spmv", "pagerank"), ("pagerank", "pagerank")])
@pytest.mark.parametrize("mode", ["global", "relaxed"])
def test_first_use_inside_a_capture(prob, what, warm, mode):
    """The graph was used by another call, or with the other choice of renaming, and the scratch buffers exist."""
    import torch

    stream = torch.cuda.Stream()
    g = prob.graph()
    with _on(prob.ctx, stream):
        prob.check(warm, g)
        if what == warm:
            g.set_relabel(False)
        out = prob.out()
        graph = _capture(prob, what, g, out, stream, mode)
        prob.check(what, g)  # ahead of the first replay
        _replay(prob, what, graph, out)
        g.set_relabel(True)
        prob.check(what, g)
        _replay(prob, what, graph, out)
        del graph
        prob.check(what, g)


@pytest.mark.parametrize("first, then", [("pagerank", "pagerank"), ("pagerank", "spmv"), ("spmv", "spmv")])
def test_next_call_on_another_stream(prob, first, then):
    """Ordered behind the first by an event; the first one's stream is busy when it comes."""
    import torch

    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    g = prob.graph()
    o1, o2 = prob.out(), prob.out()
    with torch.cuda.stream(a):
        torch.cuda._sleep(20_000_000)
    prob.ctx.set_stream(a.cuda_stream)
    prob.call(first, g, o1)
    ev = torch.cuda.Event()
    ev.record(a)
    b.wait_event(ev)
    with _on(prob.ctx, b):
        prob.call(then, g, o2)
    assert torch.equal(o1, prob.want[first]) and torch.equal(o2, prob.want[then])


def test_destroyed_while_its_first_use_is_queued_on_another_stream(prob):
    """The graph's memory goes back to the context's pool, and the next graph's builds take it, only behind its builds."""
    import torch

    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    for what in ("pagerank", "spmv"):
        out = prob.out()
        g = prob.graph()
        with torch.cuda.stream(a):
            torch.cuda._sleep(20_000_000)
        prob.ctx.set_stream(a.cuda_stream)
        prob.call(what, g, out)
        ev = torch.cuda.Event()
        ev.record(a)
        with _on(prob.ctx, b):
            b.wait_event(ev)  # its sweeps; the builds are the destruction's own affair
            g.close()
            prob.check(what, prob.graph())
        assert torch.equal(out, prob.want[what])


def test_backward_captured_before_and_after_its_permutation(ctx):
    """Past 12.6 M arcs the backward permutes values through blocks; a capture that comes first works in arc order."""
    import torch

    V, E, n = 400_009, 12_700_001, 1
    gen = torch.Generator(device="cuda").manual_seed(3)
    deg = torch.bincount(torch.randint(0, V, (E,), device="cuda", generator=gen), minlength=V)
    off = torch.zeros(V + 1, dtype=torch.int32, device="cuda")
    off[1:] = torch.cumsum(deg, 0)
    col = torch.randint(0, V, (E,), device="cuda", generator=gen, dtype=torch.int32)
    vals, X, G = (torch.randn(k, device="cuda", generator=gen) for k in (E, V, V))
    dX, dA = torch.empty(V, device="cuda"), torch.empty(E, device="cuda")
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    with _on(ctx, stream):
        def bwd(g):
            dpg.spmv_bwd_dev(ctx, g, vals.data_ptr(), n, X.data_ptr(), G.data_ptr(), dX.data_ptr(), dA.data_ptr())

        def graph_of():
            return dpg.Graph.from_device(ctx, V, E, off.data_ptr(), col.data_ptr(), None)

        g = graph_of()
        bwd(g)
        ctx.synchronize()
        want = dX.clone(), dA.clone()
        row = torch.repeat_interleave(torch.arange(V, device="cuda"), deg)
        assert torch.equal(want[1], G[row] * X[col.long()])
        late = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(late, stream=stream):
            bwd(g)
        for _ in range(2):
            dX.fill_(7)
            dA.fill_(7)
            torch.cuda.synchronize()
            late.replay()
            torch.cuda.synchronize()
            assert torch.equal(dX, want[0]) and torch.equal(dA, want[1])
            bwd(g)
            ctx.synchronize()
        h = graph_of()
        early = torch.cuda.CUDAGraph()
        with pytest.raises(dpg.DpgError):  # the transposed CSR is not there yet
            with torch.cuda.graph(early, stream=stream):
                bwd(h)
        torch.cuda.synchronize()
        bwd(h)
        ctx.synchronize()
        assert torch.equal(dX, want[0]) and torch.equal(dA, want[1])


FAILED_CALL = """
import sys
import numpy as np
import torch
sys.path.insert(0, sys.argv[1])
from conftest import dpg

ctx = dpg.Context(0)
V = 3000
rng = np.random.default_rng(1)
g = dpg.csr_from_arcs(V, rng.integers(0, V, 9 * V), rng.integers(0, V, 9 * V))
dg = dpg.Graph(ctx, g.offsets, g.col)
vals, x, y = torch.ones(g.E, device="cuda"), torch.ones(V, device="cuda"), torch.empty(V, device="cuda")
stream = torch.cuda.Stream()
torch.cuda.synchronize()
ctx.set_stream(stream.cuda_stream)
failed = False
try:
    with torch.cuda.graph(torch.cuda.CUDAGraph(), stream=stream):
        try:
            dpg.spmv_dev(ctx, dg, vals.data_ptr(), x.data_ptr(), y.data_ptr())
        except dpg.DpgError:
            failed = True
except Exception:  # the capture is void
    pass
assert failed
dpg.spmv_dev(ctx, dg, vals.data_ptr(), x.data_ptr(), y.data_ptr())
ctx.synchronize()
assert np.array_equal(y.cpu().numpy(), np.diff(g.offsets))
"""


def test_a_failed_call_leaves_no_error_to_the_next():
    """A first call under capture fails where it has to allocate scratch; the next one, not captured, is not refused. In a
    process of its own: a void capture leaves torch's generator unusable."""
    r = subprocess.run([sys.executable, "-c", FAILED_CALL, str(ROOT / "tests")], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
