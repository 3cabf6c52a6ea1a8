"""dpg_graph_hot_cache counts the arcs whose column is among the most frequent; it keeps no array per arc."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import dpg

pytestmark = pytest.mark.gpu


def test_count_and_memory():
    import torch

    V, E = 300_007, 40_000_000
    gen = torch.Generator(device="cuda").manual_seed(1)
    col = torch.empty(E, device="cuda").geometric_(2e-5, generator=gen).long().remainder(V).to(torch.int32)
    off = (torch.arange(V + 1, device="cuda", dtype=torch.int64) * E // V).to(torch.int32)
    torch.cuda.synchronize()
    with dpg.Context(0) as ctx:
        g = dpg.Graph.from_device(ctx, V, E, off.data_ptr(), col.data_ptr(), None)
        # The renaming goes by the bit length of a column's count, then by the column.
        counts = torch.bincount(col.long(), minlength=V).cpu().numpy()
        order = np.argsort(-np.floor(np.log2(np.maximum(counts, 0.5))), kind="stable")
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        before = torch.cuda.mem_get_info()[0]
        hot = g.hot_cache()
        held = before - torch.cuda.mem_get_info()[0]
        assert 0 < hot["hot_entries"] < V
        assert hot["hot_arcs"] == counts[order[:hot["hot_entries"]]].sum()
        assert held < 2 * E  # less than half of a renamed column array; the renaming itself takes 12 V
        assert g.hot_cache() == hot
        g.close()
