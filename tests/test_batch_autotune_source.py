"""Autotune times every cache size of the batch's PageRank on the windows that a run with that size uses. No call reports
which windows a sweep had, so the order of the calls is checked on the source."""
from __future__ import annotations

import re

from conftest import ROOT

SRC = ROOT / "show-me-dynamic-parallelism_gb300" / "csrc" / "dpg_batch.cu"


def test_windows_are_cut_for_each_candidate_before_its_warm_up():
    body = re.search(r"dpg_status dpg_batch_autotune\(.*?\n}\n", SRC.read_text(), re.S)[0]
    loop = re.search(r"for \(int32_t hot : .*?\n    }\n", body, re.S)[0]
    cut = re.search(r"st = (?:pr_buffers|ensure_windows)\(b", loop)
    assert cut and loop.index("tune.pr_hot = hot") < cut.start() < loop.index("run_batch_pagerank")
