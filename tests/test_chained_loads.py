"""Kernels launched as a chain (programmatic dependent launch) start while their predecessor still runs. The read-only path
(__ldg, ld.global.nc, ld_stream) is specified for data that does not change during the kernel, so nothing that a
kernel of the chain writes may be read by it. Checked on the source: a stale read need not show in a run."""
from __future__ import annotations

import re

import pytest

from conftest import ROOT

CSRC = ROOT / "show-me-dynamic-parallelism_gb300" / "csrc"
# Fields of RowGatherLaunch that a kernel of a sweep writes: x is the y of the sweep (or the renaming) before it,
# rank_prev its rank_out, dsum_in its dsum_out.
WRITTEN = ["x", "y", "rank_prev", "rank_out", "partial", "dpart", "dfix", "dsum_in", "dsum_out", "gbase", "nonstop"]


def _code(name):
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


@pytest.mark.parametrize("field", WRITTEN)
def test_sweeps_read_no_written_field_through_the_read_only_path(field):
    bad = re.findall(r"(?:__ldg|ld_stream4?(?:<\w+>)?)\s*\(\s*L\." + field + r"\b[^;]*;", _code("dpg_rowgather.cu"))
    assert not bad, bad


def test_hot_cache_fill_and_batch_reduction():
    fill = re.search(r"void fill_hot\(([^)]*)\)\s*\{(.*?)\n\}", _code("dpg_rowgather.cu"), re.S)
    assert "__restrict__ x" not in fill[1] and "__ldg" not in fill[2]
    body = re.search(r"batch_dangling_kernel\((.*?)\n\}", _code("dpg_batch.cu"), re.S)[1]
    assert not re.search(r"__ldg\(\s*(y|gpart|gbase)\b", body)
    assert re.search(r"const float\* __restrict__ y", body) is None
