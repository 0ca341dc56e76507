"""Streamed graphs under a device budget between what the graph takes without and with its bitmaps."""
import numpy as np
import pytest

import efficientstructuralgraphclusteringongpus_gb300 as sg
from oracle import oracle

pytestmark = pytest.mark.gpu


def check(g, cn, eps="0.3", mu=3):
    off, adj = g.offsets(), g.adjacency()
    for mode in (sg.PRED_EXACT, sg.PRED_REF_F64):
        res = g.run(eps, mu, mode)
        label, role, _ = oracle.scan_ex(off, adj, eps, mu, mode, cn=cn)
        assert np.array_equal(res.label, label) and np.array_equal(res.role, role)


@pytest.mark.parametrize("make", [lambda: sg.Graph.rmat(17, 16, seed=42),
                                  lambda: sg.Graph.chung_lu(60000, 2.1, 1000000, 30000, seed=43)], ids=["rmat", "hubs"])
def test_streamed_budgets(make):
    g = make()
    cn = oracle.common_neighbors(g.offsets(), g.adjacency())
    whole = g.upload_streamed(0, 0)
    with_bitmaps = g.bitmap_bytes
    assert with_bitmaps > 0
    g.release_bitmaps()
    lists = g.device_bytes
    words = 4 * g.num_edges
    for budget in (whole + (64 << 20), whole + (20 << 20), (whole + lists) // 2 + (16 << 20), lists + (17 << 20)):
        used = g.upload_streamed(0, budget)
        assert used == g.device_bytes <= budget
        check(g, cn)
        # full counts leave no more than fits the budget in the cache (by lists one word per edge)
        sg.release_cached_memory()
        assert np.array_equal(g.common_neighbors()[0], cn)
        assert sg.cached_memory_bytes(0) <= max(budget - used, words + 256)
    g.upload_streamed(0, whole + (64 << 20))
    assert g.bitmap_bytes == with_bitmaps
    g.release_device()
