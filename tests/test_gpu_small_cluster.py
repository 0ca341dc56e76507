"""The cluster stage in one launch (k_cluster_small) and as a chain of launches give the oracle's
answer on either side of the sizes where the choice changes: 2^16 edges for a run, 2^20 edges and
2^17 vertices for a served query, and the edges of the fused kernel's 8,192 threads.
Labels, roles and counters are whole numbers: they are equal.
"""
import numpy as np
import pytest

import efficientstructuralgraphclusteringongpus_gb300 as sg
from oracle import oracle

pytestmark = pytest.mark.gpu


def communities(n, size, edges, seed):
    """Exactly `edges` edges, nearly all inside communities of `size` consecutive vertices."""
    r = np.random.RandomState(seed)
    u = r.randint(0, n, 4 * edges)
    v = np.where(r.random_sample(u.size) < 0.97, u // size * size + r.randint(0, size, u.size), r.randint(0, n, u.size))
    v = np.minimum(v, n - 1)
    e = np.unique(np.stack([np.minimum(u, v), np.maximum(u, v)], 1)[u != v], axis=0)
    assert len(e) >= edges
    return sg.Graph.from_edges(n, e[r.permutation(len(e))[:edges]])


@pytest.mark.parametrize("n,edges", [(2, 1), (31, 60), (1000, 5000), (8191, 40_000), (8193, 65_535), (9000, 65_536),
                                     (9000, 65_537), (70_000, 60_000)])
@pytest.mark.parametrize("mode", [sg.PRED_EXACT, sg.PRED_REF_F64])
def test_run(n, edges, mode):
    g = communities(n, 24, edges, n) if n > 31 else sg.Graph.from_edges(n, [(i, j) for i in range(n) for j in range(i)][:edges])
    off, adj = g.offsets(), g.adjacency()
    for eps, mu in (("0.2", 2), ("0.45", 3), ("0.7", 2), ("1.5", 2)):
        res = g.run(eps, mu, predicate=mode)
        label, role, counts = oracle.scan(off, adj, eps, mu, mode)
        assert np.array_equal(res.label, label) and np.array_equal(res.role, role)
        st = res.stats
        assert (st["num_cores"], st["num_clusters"], st["num_borders"], st["num_hubs"], st["num_outliers"],
                st["multi_cluster_borders"]) == (counts["cores"], counts["clusters"], counts["borders"], counts["hubs"],
                                                 counts["outliers"], counts["multi_borders"])


def test_served_around_the_limits():
    graphs = [communities(1000, 24, 5000, 1), communities(60_000, 40, (1 << 20) - 1, 2),
              communities(60_000, 40, 1 << 20, 3), communities(60_000, 40, (1 << 20) + 1, 4),
              communities((1 << 17) - 1, 24, 400_000, 5), communities(1 << 17, 24, 400_000, 6),
              communities((1 << 17) + 1, 24, 400_000, 7)]
    counts = [oracle.common_neighbors(g.offsets(), g.adjacency()) for g in graphs]
    with sg.Server(0, 512 << 20, 4) as srv:
        ids = [srv.add_graph(g) for g in graphs]
        queries = [(k, eps, mu, mode) for k in range(len(graphs)) for eps, mu in (("0.2", 2), ("0.4", 4), ("0.8", 2))
                   for mode in (sg.PRED_EXACT, sg.PRED_REF_F64)]
        tickets = [srv.submit(ids[k], eps, mu, mode) for k, eps, mu, mode in queries]
        for (k, eps, mu, mode), t in zip(queries, tickets):
            label, role, st = srv.wait(t)
            want = oracle.scan_ex(graphs[k].offsets(), graphs[k].adjacency(), eps, mu, mode, cn=counts[k])
            assert np.array_equal(label, want[0]) and np.array_equal(role, want[1])
            assert st["num_cores"] == want[2]["cores"] and st["num_clusters"] == want[2]["clusters"]
            assert st["num_similar_edges"] == want[2]["similar_edges"]
