"""Low eps, where most edges stay open after the neighbourhood bitmaps: runs equal the oracle in every
form of the kernels that count them.

Exact counts and a bound first (from 2^22 edges on, chosen by what was counted so far), pivots of every
hash class and hubs.
"""
import numpy as np
import pytest

import efficientstructuralgraphclusteringongpus_gb300 as sg
from oracle import oracle

pytestmark = pytest.mark.gpu


def check(g, cases, cn=None):
    off, adj = g.offsets(), g.adjacency()
    cn = oracle.common_neighbors(off, adj) if cn is None else cn
    for eps, mu, mode in cases:
        res = g.run(eps, mu, mode)
        label, role, c = oracle.scan_ex(off, adj, eps, mu, mode, cn=cn)
        assert np.array_equal(res.label, label), (eps, mu, mode)
        assert np.array_equal(res.role, role), (eps, mu, mode)
        assert res.stats["num_similar_edges"] == c["similar_edges"], (eps, mu, mode)
    return cn


def both(*eps):
    return [(e, 2 + 3 * i, mode) for i, e in enumerate(eps) for mode in (sg.PRED_EXACT, sg.PRED_REF_F64)]


def random_graph(n, edges, seed):
    return sg.Graph.from_edges(n, np.random.RandomState(seed).randint(0, n, (edges, 2)))


@pytest.mark.parametrize("n,edges", [(40000, 4_210_000), (40000, 4_150_000)], ids=["above 2^22", "below"])
def test_rejected_by_the_bound(n, edges):
    # hardly a common neighbour: every count ends below its threshold
    g = random_graph(n, edges, 5)
    assert (g.num_edges >= 1 << 22) == (edges == 4_210_000)
    check(g, both("0.04", "0.06", "0.1"))


def test_counts_near_the_threshold():
    # 55% of a list are common neighbours; the first eps is met by most edges, the last by few
    g = random_graph(4000, 6_500_000, 6)
    assert g.num_edges >= 1 << 22 and 1024 < g.max_degree <= 4096
    check(g, both("0.54", "0.56", "0.57"))


def test_every_class_and_hubs_without_tails():
    g = sg.Graph.rmat(19, 16, seed=31)
    assert g.num_edges >= 1 << 22 and g.max_degree > 6144
    check(g, both("0.05", "0.12", "0.17", "0.25"))


@pytest.mark.parametrize("bitmap", ["on", "off"])      # off: pivots above the chunk are split
def test_split_pivots(monkeypatch, bitmap):
    monkeypatch.setenv("SCAN_GB300_BITMAP", bitmap)
    g = sg.Graph.rmat(18, 20, seed=33)
    assert g.num_edges >= 1 << 22
    cn = check(g, both("0.06", "0.15", "0.3"))
    g.set_plan(64, sg.SMALL_SERIAL, 4096, 12288)
    check(g, both("0.15"), cn)
