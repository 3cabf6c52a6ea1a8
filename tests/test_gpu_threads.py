"""One context per host thread: first calls on graphs of different sizes at the same time, whose gathers take different
amounts of shared memory. Each thread's results are bit-equal to those of its problem alone."""
from __future__ import annotations

import threading

import numpy as np
import pytest

from conftest import dpg

pytestmark = pytest.mark.gpu

SIZES = [37, 1_000, 5_003, 12_007, 33_333, 90_001]


def _problem(V):
    rng = np.random.default_rng(V)
    g = dpg.csr_from_arcs(V, rng.integers(0, V, 9 * V), rng.integers(0, V, 9 * V))
    in_off, in_col = dpg.csr_transpose(V, g.offsets, g.col)
    return in_off, in_col, dpg.out_degrees(g.offsets), rng.random(len(in_col), np.float32), rng.random(V, np.float32)


def _solve(ctx, p):
    in_off, in_col, od, vals, x = p
    out = []
    for epsilon in (0.0, 1e-9):
        g = dpg.Graph(ctx, in_off, in_col)
        out.append(dpg.pagerank(ctx, g, od, iterations=12, epsilon=epsilon))
        out.append(dpg.spmv(ctx, g, vals, x))
        g.close()
    return out


def test_first_calls_from_several_threads():
    problems = [_problem(V) for V in SIZES]
    got, errors = [None] * len(SIZES), []
    start = threading.Barrier(len(SIZES))

    def work(k):
        try:
            with dpg.Context(0) as ctx:
                start.wait(60)
                for _ in range(3):
                    got[k] = _solve(ctx, problems[k])
        except Exception as e:  # reported by the main thread
            errors.append((SIZES[k], e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(SIZES))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    with dpg.Context(0) as ctx:
        for p, out in zip(problems, got):
            for a, b in zip(out, _solve(ctx, p)):
                assert np.array_equal(a, b)
