"""One-shot runs through the neighbourhood sketches (kernels_sketch.cuh) equal the oracle.

Sizes sit where the sketches change form: degrees around the bitmap sizes (12 bits per
neighbour, powers of two from 2^7), edges compared by a lane, a group of lanes or a warp,
more long edges than their list holds, runs of pending edges around the table threshold,
edge counts around a 128-edge batch and around the smallest graph that has sketches (2^12
edges), plans with and without split pivots.  All results are whole numbers: they are equal.
"""
import numpy as np
import pytest

import efficientstructuralgraphclusteringongpus_gb300 as sg
from oracle import oracle

pytestmark = pytest.mark.gpu

EXACT, REF = sg.PRED_EXACT, sg.PRED_REF_F64
COUNTS = {"num_cores": "cores", "num_clusters": "clusters", "num_borders": "borders", "num_hubs": "hubs",
          "num_outliers": "outliers", "num_similar_edges": "similar_edges", "pred_disagreements": "disagreements",
          "multi_cluster_borders": "multi_borders"}


def check(g, points, modes=(EXACT, REF)):
    off, adj = g.offsets(), g.adjacency()
    cn = oracle.common_neighbors(off, adj)
    for eps, mu in points:
        for mode in modes:
            res = g.run(eps, mu, predicate=mode)
            label, role, counts = oracle.scan_ex(off, adj, eps, mu, mode, cn=cn)
            what = f"eps={eps} mu={mu} mode={mode}"
            assert np.array_equal(res.label, label), what
            assert np.array_equal(res.role, role), what
            for key, name in COUNTS.items():
                assert res.stats[key] == counts[name], f"{what}: {key}"


def random_graph(n, pairs, seed):
    return sg.Graph.from_edges(n, np.random.RandomState(seed).randint(0, n, (pairs, 2)))


def stars_sharing(degrees, shared, seed):
    """Hubs of the given degrees over one pool of leaves, each pair of hubs joined: the edges
    between hubs have lists of exactly those degrees with a set share in common."""
    r = np.random.RandomState(seed)
    k, pool = len(degrees), 2 * max(degrees) + 64
    edges = [(i, j) for i in range(k) for j in range(i + 1, k)]
    common = r.permutation(pool)
    for i, d in enumerate(degrees):
        own = max(d - (k - 1), 0)
        same = int(own * shared)
        rest = r.permutation(common[same:])[: own - same]
        edges += [(i, k + int(x)) for x in np.concatenate([common[:same], rest])]
    return sg.Graph.from_edges(k + pool, edges)


@pytest.mark.parametrize("degrees", [
    [10, 11, 12, 21, 22, 42, 43, 44],                  # the smallest sizes: 2^7, 2^8, 2^9
    [84, 85, 86, 170, 171, 172],                       # lane and group work
    [341, 342, 682, 683, 684, 1365, 1366],             # built by a warp, then by a CTA
    [5460, 5461, 5462, 10922, 10923, 10924],           # whole-SM CTAs; k_sketch_long
])
@pytest.mark.parametrize("shared", [0.05, 0.5, 0.95])
def test_bitmap_sizes(degrees, shared):
    g = stars_sharing(degrees * 2, shared, seed=len(degrees))
    check(g, [("0.1", 2), ("0.3", 2), ("0.5", 3), ("0.7", 2), ("0.95", 2)])


@pytest.mark.parametrize("edges", [4094, 4095, 4096, 4097, 4223, 4224, 4225, 6001])
def test_edge_counts_around_batches(edges):
    r = np.random.RandomState(edges)
    pool = np.unique(np.sort(r.randint(0, 500, (4 * edges, 2)), axis=1), axis=0)
    pool = pool[pool[:, 0] != pool[:, 1]]
    g = sg.Graph.from_edges(501, pool[r.permutation(len(pool))[:edges]])
    assert g.num_edges == edges
    check(g, [("0.15", 2), ("0.3", 3), ("0.6", 2)])


@pytest.mark.parametrize("n,pairs", [(2000, 800_000), (300, 20_000), (40_000, 200_000)])
def test_random_graphs(n, pairs):
    check(random_graph(n, pairs, n), [("0", 2), ("0.1", 3), ("0.25", 2), ("0.5", 4), ("0.9", 2), ("1", 2), ("1.5", 2)])


def test_complete_graph_overflows_the_long_list():
    # every edge is similar, so every bitmap fails at its first size and again at the largest
    # (2^16 bits at degree 2999): 4.5M long edges for a list of a sixteenth of that
    n = 3000
    i, j = np.triu_indices(n, 1)
    off = np.arange(n + 1, dtype=np.uint64) * (n - 1)
    adj = np.arange(n * n, dtype=np.uint32) % n
    adj = adj[np.arange(n * n) // n != adj]
    g = sg.Graph.from_csr(off, adj)
    for mode in (EXACT, REF):
        res = g.run("0.9", 5, predicate=mode)
        assert (res.label == 0).all() and (res.role == sg.ROLE_CORE).all()
        assert res.stats["num_similar_edges"] == len(i) and res.stats["pred_disagreements"] == 0


@pytest.mark.parametrize("knob", ["on", "off"])
def test_split_pivots(monkeypatch, knob):
    # with the bitmap path off, pivots above 6,144 neighbours are split into chunks
    monkeypatch.setenv("SCAN_GB300_BITMAP", knob)
    check(sg.Graph.rmat(15, 16, seed=3), [("0.1", 2), ("0.2", 2), ("0.5", 5)])
    check(sg.Graph.chung_lu(60000, 2.1, 400000, 30000, seed=5), [("0.2", 2), ("0.4", 5)])


@pytest.mark.parametrize("clique", [3, 4, 5, 6, 9, 33, 70])
def test_pending_runs(clique):
    # cliques of k vertices with a few random edges: a vertex has about k / 2 pending lower
    # edges, around the run length that takes a table (4) and a window of 32 edges
    r = np.random.RandomState(clique)
    count = 12000 // (clique * (clique - 1) // 2) + 40
    i, j = np.triu_indices(clique, 1)
    base = np.arange(count)[:, None] * clique
    inside = np.stack([(base + i).ravel(), (base + j).ravel()], 1)
    n = count * clique
    check(sg.Graph.from_edges(n, np.concatenate([inside, r.randint(0, n, (n // 2, 2))])),
          [("0.3", 2), ("0.5", 2), ("0.7", 3), ("0.9", 2)])


def test_streamed_without_room_for_sketches():
    g = sg.Graph.rmat(16, 16, seed=1)
    g.upload_streamed(0, 0)
    with_sketches = g.device_bytes
    g.release_device()
    # a budget just above the estimate for the graph itself (30 MiB, of which 16 are slack)
    # leaves no room for its sketches: accepted, smaller, and the same result
    used = g.upload_streamed(0, 31 << 20)
    assert used < with_sketches - 2 * g.m
    check(g, [("0.3", 2), ("0.5", 5)], modes=(REF,))


def test_hubs_of_many_chunks_with_their_edges_pending(monkeypatch):
    """96 joined hubs over 120,000 shared leaves, each hub's list in 20 chunks: nearly every edge
    between hubs is left open, so each chunk task of a hub has edges to be cut into slices, and
    charged with their whole lists the tasks would ask for about twice the slices there is room
    for."""
    monkeypatch.setenv("SCAN_GB300_BITMAP", "off")
    hubs, leaves = 96, 120_000
    i, j = np.triu_indices(hubs, 1)
    h, x = np.divmod(np.arange(hubs * leaves), leaves)
    pairs = np.concatenate([np.stack([i, j], 1), np.stack([h, hubs + x], 1)])
    check(sg.Graph.from_edges(hubs + leaves, pairs), [("0.5", 2)])


@pytest.mark.parametrize("eps,modes", [("0.149999", (EXACT, REF)), ("0.15", (REF,))])
def test_large_graph_around_the_least_eps_of_sketches(eps, modes):
    # 2^25 edges and more: lists alone below eps 0.15, bitmaps first from there on
    g = sg.Graph.rmat(22, 9, seed=1)
    assert g.num_edges >= 1 << 25
    for mode in modes:
        res = g.run(eps, 2, predicate=mode)
        label, role, counts = oracle.scan_ex(g.offsets(), g.adjacency(), eps, 2, mode, prune=True)
        assert np.array_equal(res.label, label) and np.array_equal(res.role, role)
        for key, name in COUNTS.items():
            assert res.stats[key] == counts[name], key
