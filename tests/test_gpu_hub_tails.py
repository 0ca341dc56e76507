"""Hubs whose neighbours do not all have hot ids: runs and full counts by the list kernels equal the
oracle for tails of every length, those too long for the bitmap kernel among them.
"""
import numpy as np
import pytest

import efficientstructuralgraphclusteringongpus_gb300 as sg
from oracle import oracle

pytestmark = pytest.mark.gpu


def hubs_with_tails():
    """24 hubs, all joined, each with 7,000 hot neighbours and a tail of 0 to 15,000 others."""
    r = np.random.RandomState(8)
    hubs, hot, cold = 24, 700_000, 600_000
    first_hot, first_cold = hubs, hubs + hot
    n = hubs + hot + cold
    i = np.arange(hot)
    edges = [np.stack([first_hot + i, first_hot + (i + k) % hot], 1) for k in (1, 2)]
    edges.append(np.array([(a, b) for a in range(hubs) for b in range(a)]))
    for h in range(hubs):
        near = r.permutation(20_000)[:7_000]        # of a common part: hubs share some
        edges.append(np.stack([np.full(7_000, h), first_hot + near], 1))
    # cold vertices have two neighbours: two hubs, or a ring of their own.  Tails grow with the hub's id.
    linked = 100_000
    weight = np.arange(hubs, dtype=float)
    a = r.choice(hubs, linked, p=weight / weight.sum())
    b = (a + 1 + r.randint(0, hubs - 1, linked)) % hubs
    b[b == 0] = 2                                    # hub 0 keeps no tail
    b[a == b] = 1
    c = first_cold + np.arange(linked)
    edges += [np.stack([a, c], 1), np.stack([b, c], 1)]
    rest = first_cold + linked + np.arange(cold - linked)
    edges.append(np.stack([rest, np.roll(rest, 1)], 1))
    return sg.Graph.from_edges(n, np.concatenate(edges))


def test_hubs_with_tails():
    g = hubs_with_tails()
    deg = g.degrees()
    assert (deg[:24] > 6144).all() and (deg >= 3).sum() < 1 << 20 < (deg >= 1).sum()
    off, adj = g.offsets(), g.adjacency()
    cn = oracle.common_neighbors(off, adj)
    for eps, mu in (("0.05", 2), ("0.2", 5), ("0.4", 8)):
        for mode in (sg.PRED_EXACT, sg.PRED_REF_F64):
            res = g.run(eps, mu, mode)
            label, role, _ = oracle.scan_ex(off, adj, eps, mu, mode, cn=cn)
            assert np.array_equal(res.label, label) and np.array_equal(res.role, role), (eps, mode)
    sg.release_cached_memory()
    for _ in range(2):
        assert np.array_equal(g.common_neighbors()[0], cn)
    # full counts by the list kernels
    try:
        sg.set_device_memory_left(4 * g.num_edges + 512)
        assert np.array_equal(g.common_neighbors()[0], cn)
    finally:
        sg.set_device_memory_left(None)
