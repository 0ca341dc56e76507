"""Calls on a device with little memory left give the same results by the paths that need less.

set_device_memory_left makes the engine's allocations on this thread fail as on a nearly full
device, so no test fills one.
"""
import itertools

import numpy as np
import pytest

import efficientstructuralgraphclusteringongpus_gb300 as sg
from oracle import oracle

pytestmark = pytest.mark.gpu

PLANS = list(itertools.product((64, 128), (sg.SMALL_SERIAL, sg.SMALL_BATCHED, sg.SMALL_SEARCH), (4096, 6144),
                               (6144, 12288)))


@pytest.fixture(autouse=True)
def no_limit():
    sg.release_cached_memory()      # cached blocks may be larger than what is asked for
    yield
    sg.set_device_memory_left(None)


def graphs():
    ring = [(i, (i + k) % 30000) for i in range(30000) for k in (1, 2, 5)]
    return {"rmat14": sg.Graph.rmat(14, 16, seed=21),
            "chung_lu": sg.Graph.chung_lu(200000, 2.1, 1500000, 60000, seed=23),
            "ring": sg.Graph.from_edges(30000, ring)}      # no bitmaps: small pivots only


@pytest.fixture(scope="module")
def cases():
    yield {name: (g, oracle.common_neighbors(g.offsets(), g.adjacency())) for name, g in graphs().items()}


def room(g, words):
    """Device memory for `words` words per edge, as the engine rounds it, and a little."""
    return words * (4 * g.num_edges + 256) + 256


@pytest.mark.parametrize("words", [1, 2, 3])
def test_full_counts_with_room_for_the_list_kernels(cases, words):
    # the triangles take two words per edge and their task lists, the lists one word
    for g, cn in cases.values():
        g.upload()
        sg.set_device_memory_left(room(g, words))
        for _ in range(2):
            got, st = g.common_neighbors()
            assert np.array_equal(got, cn) and st["num_edges"] == g.num_edges
        sg.set_device_memory_left(None)
        g.release_device()


@pytest.mark.parametrize("bitmap", ["on", "off"])      # off: pivots above the chunk are split
@pytest.mark.parametrize("small_deg,strategy,hub,chunk", PLANS)
def test_full_counts_by_lists_under_every_plan(cases, monkeypatch, bitmap, small_deg, strategy, hub, chunk):
    monkeypatch.setenv("SCAN_GB300_BITMAP", bitmap)
    for g, cn in cases.values():
        g.set_plan(small_deg, strategy, hub, chunk)
        sg.set_device_memory_left(room(g, 1))
        assert np.array_equal(g.common_neighbors()[0], cn)
        sg.set_device_memory_left(None)
        g.release_device()
