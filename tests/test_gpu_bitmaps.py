"""The neighbourhood bitmaps of a resident graph as memory: what they take, giving them back, and calls
that find no memory with them.
"""
import numpy as np
import pytest

import efficientstructuralgraphclusteringongpus_gb300 as sg
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def no_limit():
    sg.release_cached_memory()      # cached blocks may be larger than what is asked for
    yield
    sg.set_device_memory_left(None)


@pytest.fixture(scope="module")
def rmat():
    g = sg.Graph.rmat(16, 16, seed=41)
    yield g, oracle.common_neighbors(g.offsets(), g.adjacency())


def check(g, cn, eps="0.3", mu=3):
    off, adj = g.offsets(), g.adjacency()
    for mode in (sg.PRED_EXACT, sg.PRED_REF_F64):
        res = g.run(eps, mu, mode)
        label, role, _ = oracle.scan_ex(off, adj, eps, mu, mode, cn=cn)
        assert np.array_equal(res.label, label) and np.array_equal(res.role, role)


def test_release(rmat):
    g, cn = rmat
    g.upload()
    whole, bitmaps = g.device_bytes, g.bitmap_bytes
    assert 0 < bitmaps < whole
    check(g, cn)
    g.release_bitmaps()
    assert g.bitmap_bytes == 0 and g.device_bytes == whole - bitmaps
    check(g, cn)
    assert np.array_equal(g.common_neighbors()[0], cn)
    g.set_plan(64, sg.SMALL_SEARCH, 4096, 12288)
    check(g, cn)
    g.release_bitmaps()
    g.release_device()
    g.release_bitmaps()
    assert g.bitmap_bytes == 0
    check(g, cn)
    assert g.bitmap_bytes == bitmaps
    g.release_device()


def test_a_new_plan_takes_the_room_of_the_bitmaps(rmat):
    # above every degree: the hubs are split, and pending edges get an array of their own
    g, cn = rmat
    g.upload()
    assert g.max_degree > 6144
    sg.set_device_memory_left(1 << 20)
    g.set_plan(64, sg.SMALL_SERIAL, 1 << 30, 6144)
    assert g.bitmap_bytes == 0
    check(g, cn)
    g.release_device()


def test_a_plan_that_finds_no_room_leaves_the_graph_usable(rmat):
    g, cn = rmat
    g.upload()
    g.release_bitmaps()
    sg.release_cached_memory()
    before = g.plan()
    sg.set_device_memory_left(0)
    with pytest.raises(sg.ScanError) as e:
        g.set_plan(1, sg.SMALL_SERIAL, 1 << 30, 6144)
    assert e.value.status == 5
    sg.set_device_memory_left(None)
    check(g, cn)
    assert g.plan() == before
    g.release_device()


def test_memberships_take_the_room_of_the_bitmaps(rmat):
    g, cn = rmat
    want = g.memberships("0.2", 2)
    g.release_device()
    g.upload()
    sg.set_device_memory_left(0)
    got = g.memberships("0.2", 2)
    assert got[0].size and all(np.array_equal(a, b) for a, b in zip(want, got))
    assert g.bitmap_bytes == 0
    g.release_device()
