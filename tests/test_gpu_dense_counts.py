"""Full counts of graphs of nearly complete neighbourhoods, which the list kernels count faster.

From 2^19 edges and 96 neighbours on average a sample of the lists decides; the graphs sit on both
sides of each limit.  Counts are whole numbers: they are equal, by either way, and a served graph's
queries give the oracle's labels.
"""
import numpy as np
import pytest

import efficientstructuralgraphclusteringongpus_gb300 as sg
from oracle import oracle

pytestmark = pytest.mark.gpu


def complete(n):
    adj = np.arange(n * n, dtype=np.uint32) % n
    adj = adj[np.arange(n * n) // n != adj]
    return sg.Graph.from_csr(np.arange(n + 1, dtype=np.uint64) * (n - 1), adj)


def csr(n, lists):
    """Lists of equal length, one per vertex, any order: rows of an array."""
    return sg.Graph.from_csr(np.arange(n + 1, dtype=np.uint64) * lists.shape[1], np.sort(lists, axis=1).astype(np.uint32).ravel())


def ring(n, k):
    steps = np.concatenate([np.arange(-k, 0), np.arange(1, k + 1)])
    return csr(n, (np.arange(n)[:, None] + steps) % n)


def cliques(count, size):
    inside = np.array([[j for j in range(size) if j != i] for i in range(size)])
    return csr(count * size, (np.arange(count)[:, None, None] * size + inside).reshape(count * size, size - 1))


@pytest.mark.parametrize("n", [1024, 1025, 1400])          # 523,776 edges; 524,800; 979,300
def test_complete_graphs(n):
    cn, _ = complete(n).common_neighbors()
    assert cn.size == n * (n - 1) // 2 and (cn == n - 2).all()


@pytest.mark.parametrize("make", [lambda: ring(11000, 48), lambda: ring(11000, 47), lambda: cliques(120, 97),
                                  lambda: cliques(120, 96), lambda: ring(3000, 200),
                                  lambda: sg.Graph.from_edges(3000, np.random.RandomState(1).randint(0, 3000, (700_000, 2)))],
                         ids=["degree96", "degree94", "cliques97", "cliques96", "ring400", "random"])
def test_equal_the_oracle(make):
    g = make()
    cn = oracle.common_neighbors(g.offsets(), g.adjacency())
    for _ in range(2):
        assert np.array_equal(g.common_neighbors()[0], cn)
    with sg.Server(0, 64 << 20, 2) as srv:
        gid = srv.add_graph(g)
        for eps, mu, mode in (("0.3", 2, sg.PRED_EXACT), ("0.6", 5, sg.PRED_REF_F64)):
            label, role, _ = srv.wait(srv.submit(gid, eps, mu, mode))
            want = oracle.scan_ex(g.offsets(), g.adjacency(), eps, mu, mode, cn=cn)
            assert np.array_equal(label, want[0]) and np.array_equal(role, want[1])


def test_a_complete_graph_takes_no_longer_than_by_lists():
    # the lists alone, where memory leaves no other way; by triangles it took 1.8 times as long
    g = complete(3000)
    g.upload()
    sg.release_cached_memory()
    sg.set_device_memory_left(4 * g.num_edges + 512)
    by_lists = min(g.common_neighbors()[1]["ms_similarity"] for _ in range(4))
    sg.set_device_memory_left(None)
    ms = min(g.common_neighbors()[1]["ms_similarity"] for _ in range(4))
    assert ms < 1.3 * by_lists, (ms, by_lists)
