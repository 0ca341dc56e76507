"""Boundary cases of the neighbourhood bitmaps on graphs that have them.

Below 2^19 edges a graph has bitmaps only if some vertex has more than 128 neighbours, and never below
2^12 edges: each graph here holds a star of 200 leaves (and, where it has too few edges, a ring beside
it), so that its batches, bitmap sizes and pending runs go through the bitmap kernels, and says so.
"""
import numpy as np
import pytest

import efficientstructuralgraphclusteringongpus_gb300 as sg
from oracle import oracle

pytestmark = pytest.mark.gpu

STAR = 200


def with_star(n, edges, least=0):
    """The graph of `edges` on n vertices, a star of its own and a ring of what `least` edges lack."""
    parts = [np.asarray(edges), np.stack([np.full(STAR, n), n + 1 + np.arange(STAR)], 1)]
    n += STAR + 1
    ring = max(least - len(edges) - STAR, 0)
    if ring:
        parts.append(n + np.stack([np.arange(ring + 3), (np.arange(ring + 3) + 1) % (ring + 3)], 1))
        n += ring + 3
    return sg.Graph.from_edges(n, np.concatenate(parts))


def check(g, points, bitmaps=True):
    off, adj = g.offsets(), g.adjacency()
    cn = oracle.common_neighbors(off, adj)
    for eps, mu in points:
        for mode in (sg.PRED_EXACT, sg.PRED_REF_F64):
            res = g.run(eps, mu, predicate=mode)
            label, role, counts = oracle.scan_ex(off, adj, eps, mu, mode, cn=cn)
            assert np.array_equal(res.label, label) and np.array_equal(res.role, role), (eps, mu, mode)
            assert res.stats["num_similar_edges"] == counts["similar_edges"], (eps, mu, mode)
            assert res.stats["pred_disagreements"] == counts["disagreements"], (eps, mu, mode)
    assert (g.bitmap_bytes > 0) == bitmaps


def random_pairs(n, count, seed):
    r = np.random.RandomState(seed)
    pool = np.unique(np.sort(r.randint(0, n, (4 * count, 2)), axis=1), axis=0)
    pool = pool[pool[:, 0] != pool[:, 1]]
    return pool[r.permutation(len(pool))[:count]]


@pytest.mark.parametrize("edges", [4094, 4095, 4096, 4097, 4223, 4224, 4225, 6001])
def test_edge_counts_around_batches(edges):
    g = with_star(501, random_pairs(501, edges - STAR, edges))
    assert g.num_edges == edges and g.max_degree == STAR
    check(g, [("0.15", 2), ("0.3", 3), ("0.6", 2)], bitmaps=edges >= 1 << 12)


@pytest.mark.parametrize("degrees", [[10, 11, 12], [21, 22, 42, 43, 44], [84, 85, 86, 127, 128]])
@pytest.mark.parametrize("shared", [0.05, 0.5, 0.95])
def test_small_bitmap_sizes(degrees, shared):
    # hubs of exactly these degrees, two of each, over one pool of leaves, each pair joined
    r = np.random.RandomState(len(degrees))
    hubs = degrees * 2
    k, pool = len(hubs), 2 * max(hubs) + 64
    edges = [(i, j) for i in range(k) for j in range(i + 1, k)]
    for i, d in enumerate(hubs):
        own = d - (k - 1)
        same = int(own * shared)
        rest = same + r.permutation(pool - same)[: own - same]
        edges += [(i, k + int(x)) for x in np.concatenate([np.arange(same), rest])]
    g = with_star(k + pool, np.array(edges), 4200)
    assert (g.degrees()[:k] == hubs).all()
    check(g, [("0.1", 2), ("0.3", 2), ("0.5", 3), ("0.7", 2), ("0.95", 2)])


@pytest.mark.parametrize("clique", [3, 4, 5, 6, 9, 33, 34, 66, 70, 120])
def test_pending_runs(clique):
    # cliques with a few random edges: a vertex has about half a clique of pending lower edges,
    # around the run length that takes a table (4), a window of 32 edges and a tile of 128
    r = np.random.RandomState(clique)
    count = 12000 // (clique * (clique - 1) // 2) + 40
    i, j = np.triu_indices(clique, 1)
    base = np.arange(count)[:, None] * clique
    inside = np.stack([(base + i).ravel(), (base + j).ravel()], 1)
    n = count * clique
    check(with_star(n, np.concatenate([inside, r.randint(0, n, (n // 2, 2))]), 4200),
          [("0.05", 2), ("0.3", 2), ("0.5", 2), ("0.7", 3), ("0.9", 2)])


@pytest.mark.parametrize("n,pairs", [(300, 20_000), (40_000, 200_000)])
def test_random_graphs(n, pairs):
    edges = np.random.RandomState(n).randint(0, n, (pairs, 2))
    check(with_star(n, edges), [("0", 2), ("0.1", 3), ("0.25", 2), ("0.5", 4), ("0.9", 2), ("1", 2), ("1.5", 2)])


@pytest.mark.parametrize("strategy", [sg.SMALL_SERIAL, sg.SMALL_BATCHED, sg.SMALL_SEARCH])
@pytest.mark.parametrize("small_deg", [1, 64, 128])
def test_small_pivot_strategies_without_bitmaps(strategy, small_deg):
    # no vertex above 128 neighbours and fewer than 2^19 edges: k_cn_small, k_cn_filter_classes below its cut
    r = np.random.RandomState(9)
    i, j = np.triu_indices(40, 1)
    base = np.arange(60)[:, None] * 40
    inside = np.stack([(base + i).ravel(), (base + j).ravel()], 1)
    g = sg.Graph.from_edges(2400, np.concatenate([inside, r.randint(0, 2400, (60_000, 2))]))
    assert 64 < g.max_degree <= 128
    g.set_plan(small_deg, strategy, 6144, 6144)
    check(g, [("0", 2), ("0.2", 2), ("0.45", 3), ("0.7", 2)], bitmaps=False)
