"""Uploads: graphs the device refuses, too little memory for the bitmaps, launches counted, several threads."""
import threading

import numpy as np
import pytest

import efficientstructuralgraphclusteringongpus_gb300 as sg
from oracle import oracle

pytestmark = pytest.mark.gpu


def arrays(g):
    return g.offsets().astype(np.uint32), g.adjacency().astype(np.int32)


def without(off, adj, v, k):
    """The arrays without entry k of v's list."""
    off = off.copy()
    adj = np.delete(adj, off[v] + k)
    off[v + 1:] -= 1
    return off, adj


@pytest.mark.parametrize("scale", [6, 13, 16])           # without bitmaps, with them, with hubs
@pytest.mark.parametrize("entries", [1, 2, 7, 64])
def test_asymmetric_graphs_are_refused(scale, entries):
    g = sg.Graph.rmat(scale, 16, seed=61)
    off, adj = arrays(g)
    r = np.random.RandomState(entries)
    for _ in range(entries):                             # odd and even numbers of entries are left
        v = int(r.choice(np.flatnonzero(np.diff(off.astype(np.int64)) > 0)))
        off, adj = without(off, adj, v, int(r.randint(off[v + 1] - off[v])))
    with pytest.raises(sg.ScanError) as e:
        sg.GPUScan(off, adj, 0.5, 2)
    assert "symmetric" in str(e.value)
    label, _, _ = oracle.scan(g.offsets(), g.adjacency(), "0.5", 2, sg.PRED_REF_F64)
    assert np.array_equal(sg.GPUScan(*arrays(g), 0.5, 2), label)


def test_one_sided_lists_are_refused():
    # every edge in its lower endpoint's list only, and in its higher endpoint's only
    n = 3000
    lists = [np.arange(v + 1, min(v + 400, n)) for v in range(n)]
    off = np.concatenate([[0], np.cumsum([len(x) for x in lists])]).astype(np.uint32)
    for mirror in (False, True):
        a = [n - 1 - x[::-1] for x in lists][::-1] if mirror else lists
        o = np.concatenate([[0], np.cumsum([len(x) for x in a])]).astype(np.uint32)
        assert o[-1] == off[-1]
        with pytest.raises(sg.ScanError) as e:
            sg.GPUScan(o, np.concatenate(a).astype(np.int32), 0.3, 2)
        assert "symmetric" in str(e.value)


def test_upload_without_room_for_the_bitmaps():
    g = sg.Graph.rmat(16, 16, seed=62)
    g.upload()
    whole, bitmaps = g.device_bytes, g.bitmap_bytes
    g.release_device()
    sg.release_cached_memory()
    try:
        sg.set_device_memory_left(whole - bitmaps // 2 + 8 * (g.n + 2))     # the 64-bit offsets, for a while
        g.upload()
    finally:
        sg.set_device_memory_left(None)
    assert g.bitmap_bytes == 0 and g.device_bytes <= whole - bitmaps
    label, role, _ = oracle.scan(g.offsets(), g.adjacency(), "0.3", 3, sg.PRED_EXACT)
    res = g.run("0.3", 3, sg.PRED_EXACT)
    assert np.array_equal(res.label, label) and np.array_equal(res.role, role)
    g.release_device()


def test_launches_of_an_upload():
    # 64-bit offsets and their check, tile map, degree histogram, hot ids, one orientation pass, two
    # scans of three, the fill, two plans: 15 where there are no bitmaps; with them the size classes,
    # the ranks, the small ones and, of 3,000 neighbours, the middle ones
    path = sg.Graph.from_edges(300, [(i, i + 1) for i in range(299)])
    star = sg.Graph.from_edges(4000, [(0, i) for i in range(1, 3001)] + [(i, i + 1) for i in range(1, 3001)])
    for g, want in ((path, 15), (star, 19)):
        first = g.run("0.5", 2).stats["kernel_launches"]
        assert first - g.run("0.5", 2).stats["kernel_launches"] == want
    assert star.bitmap_bytes > 0


def test_graphs_of_several_threads():
    # uploads, runs and frees side by side: pooled streams, pinned staging and cached buffers change hands
    graphs = [sg.Graph.rmat(10 + i % 5, 16, seed=70 + i) for i in range(6)]
    want = [oracle.scan(g.offsets(), g.adjacency(), "0.3", 2, sg.PRED_REF_F64)[:2] for g in graphs]
    host = [arrays(g) for g in graphs]
    wrong = []

    def work(k):
        try:
            for i in range(24):
                q = (i + k) % len(graphs) if i % 3 == 0 else k
                if i % 3 == 0:
                    ok = np.array_equal(sg.GPUScan(*host[q], 0.3, 2), want[q][0])
                else:
                    res = graphs[q].run("0.3", 2, sg.PRED_REF_F64)
                    ok = np.array_equal(res.label, want[q][0]) and np.array_equal(res.role, want[q][1])
                    if i % 6 == 5:
                        graphs[q].release_device()
                if not ok:
                    wrong.append((k, i))
        except Exception as e:   # noqa: BLE001 - reported below
            wrong.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(graphs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
