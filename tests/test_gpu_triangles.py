"""Full common-neighbour counts by triangles (kernels_tri.cuh) equal the oracle's.

Sizes sit at the edges of its form: pivots of 128 and 129 neighbours (a warp, a CTA), slices of
1,024 lower edges, higher-neighbour lists of 1,024 entries (one staged chunk, then more), batches
of 32 edges, lists at every alignment.  Counts are whole numbers: they are equal.
"""
import numpy as np
import pytest

import efficientstructuralgraphclusteringongpus_gb300 as sg
from oracle import oracle

pytestmark = pytest.mark.gpu


def check(g):
    cn, st = g.common_neighbors()
    assert np.array_equal(cn, oracle.common_neighbors(g.offsets(), g.adjacency()))
    assert st["num_edges"] == g.num_edges and st["kernel_launches"] > 0


def complete(n):
    adj = np.arange(n * n, dtype=np.uint32) % n
    adj = adj[np.arange(n * n) // n != adj]
    return sg.Graph.from_csr(np.arange(n + 1, dtype=np.uint64) * (n - 1), adj)


@pytest.mark.parametrize("n", [3, 4, 129, 130, 131, 1024, 1025, 1026, 2050, 2051])
def test_complete_graphs(n):
    # every vertex is a pivot; the middle ones hold up to n - 2 higher neighbours
    cn, _ = complete(n).common_neighbors()
    assert cn.size == n * (n - 1) // 2 and (cn == n - 2).all()


@pytest.mark.parametrize("lower", [31, 32, 33, 127, 128, 129, 1023, 1024, 1025, 2048, 2049])
@pytest.mark.parametrize("higher", [1, 2, 5])
def test_slices(lower, higher):
    # `higher` hubs over the same leaves: each is a pivot for all of them with the others above it
    # (equal degrees, larger ids); a second ring joins leaves so that lists vary in length
    r = np.random.RandomState(lower * 10 + higher)
    hubs = np.arange(higher + 1) + lower
    edges = [(i, int(h)) for i in range(lower) for h in hubs]
    edges += [(int(a), int(b)) for i, a in enumerate(hubs) for b in hubs[i + 1:]]
    edges += [(i, int(j)) for i in range(lower) for j in r.randint(0, lower, 3)]
    check(sg.Graph.from_edges(lower + higher + 1, edges))


@pytest.mark.parametrize("n,pairs", [(50, 200), (400, 30_000), (3000, 400_000), (70_000, 300_000)])
def test_random_graphs(n, pairs):
    check(sg.Graph.from_edges(n, np.random.RandomState(n).randint(0, n, (pairs, 2))))


def test_counts_then_memberships_and_runs():
    # the counts stay cached for later calls on the same resident graph, which agree with a run
    g = sg.Graph.rmat(13, 16, seed=4)
    fresh = sg.Graph.rmat(13, 16, seed=4)
    check(g)
    for mode in (sg.PRED_EXACT, sg.PRED_REF_F64):
        for a, b in zip(g.memberships("0.3", 2, mode), fresh.memberships("0.3", 2, mode)):
            assert np.array_equal(a, b)
    res = g.run("0.3", 2)
    label, role, _ = oracle.scan(g.offsets(), g.adjacency(), "0.3", 2, 0)
    assert np.array_equal(res.label, label) and np.array_equal(res.role, role)
    check(g)


def test_streamed_counts():
    g = sg.Graph.rmat(14, 16, seed=9)
    g.upload_streamed(0, 0)
    check(g)
