"""The autotuner times what runs execute: the stage of a one-shot run, not full counts by lists."""
import numpy as np
import pytest

import efficientstructuralgraphclusteringongpus_gb300 as sg

pytestmark = pytest.mark.gpu


def stage_ms(g):
    return min(g.run("0.5", 5, sg.PRED_REF_F64).stats["ms_similarity"] for _ in range(8))


@pytest.mark.parametrize("make", [lambda: sg.Graph.rmat(18, 16, seed=51),
                                  lambda: sg.Graph.chung_lu(200000, 2.1, 3000000, 20000, seed=52)], ids=["rmat18", "hubs"])
def test_times_the_stage_of_a_run(make):
    g = make()
    g.upload()
    assert g.bitmap_bytes > 0
    before = stage_ms(g)
    label = g.run("0.5", 5, sg.PRED_REF_F64).label
    info = g.autotune()
    # full counts by lists of these graphs take ten times as long as the stage of such a run
    assert info["similarity_ms"] < 2 * before, (info, before)
    assert info["small_strategy"] == sg.SMALL_SERIAL             # the only form behind the bitmaps
    assert stage_ms(g) < 1.2 * before
    assert np.array_equal(g.run("0.5", 5, sg.PRED_REF_F64).label, label)


def test_without_bitmaps_every_strategy_is_tried():
    g = sg.Graph.from_edges(6000, [(i, (i + k) % 6000) for i in range(6000) for k in range(1, 9)])
    info = g.autotune()
    assert g.bitmap_bytes == 0 and info["small_strategy"] in (sg.SMALL_SERIAL, sg.SMALL_BATCHED, sg.SMALL_SEARCH)
    assert (g.run("0.4", 3).role == sg.ROLE_CORE).all()
