"""The packaged tuning table against the tuner that should find it: its chunks,
runs and blocks are among the sweeps' candidates, its widths within their
spread of the cost model's, and size classes outside the sweeps follow from
those inside.  On the CPU (the table and the model are host code)."""
import inspect
import json

import pytest


@pytest.fixture()
def packaged():
    from liblightzk_b200 import autotune
    saved = autotune.current()
    windows = {(k, g, lg): autotune.get_value(k, g, lg) for k in ("window", "table_window") for g in (1, 2) for lg in range(33)}
    for (k, g, lg) in windows:
        autotune.set_value(k, g, lg, 0)
    with open(autotune.DEFAULT_TABLES["B200"]) as f:
        yield json.load(f)
    for g in (1, 2):
        for k in saved["msm"][str(g)]:
            for lg in range(33):
                autotune.set_value(k, g, lg, windows.get((k, g, lg), 0))
    for lg in range(33):
        autotune.set_value("ntt", 0, lg, 0)


def _default(f, name):
    return inspect.signature(f).parameters[name].default


def test_candidates(packaged):
    from liblightzk_b200 import autotune as a
    for f in (a.tune_msm, a.tune_msm_table):
        for g in ("1", "2"):
            pre = "table_" if f is a.tune_msm_table else ""
            assert set(packaged["msm"][g][pre + "chunk"].values()) <= set(_default(f, "chunks"))
            assert set(packaged["msm"][g][pre + "run"].values()) <= set(_default(f, "runs"))
    assert set(packaged["ntt"].values()) <= set(_default(a.tune_ntt, "blocks"))
    lgs = {1: (20, 21), 2: (20,)}        # the benchmark prover's classes
    for g in (1, 2):
        for lg in lgs[g]:
            assert packaged["msm"][str(g)]["table_chunk"][str(lg)] in _default(a.tune_prover, "chunks")
            assert packaged["msm"][str(g)]["table_run"][str(lg)] in _default(a.tune_prover, "runs")


def test_widths_near_the_model(packaged):
    from liblightzk_b200 import autotune as a, msm
    # the spreads bench.py's tune case takes
    for g, below, above in ((1, 2, 2), (2, 3, 3)):
        for lg in a.PLAIN_CLASSES[g]:
            c = packaged["msm"][str(g)]["window"][str(lg)]
            m = msm.autotune_window(g, 1 << lg)
            assert m - below <= c <= m + above, (g, lg, c, m)
    below, above = _default(a.tune_msm_table, "spread")
    for g in (1, 2):
        for lg in a.TABLE_CLASSES[g]:
            c = packaged["msm"][str(g)]["table_window"][str(lg)]
            m = msm.autotune_window(g, 1 << lg, precomputed=True)
            assert m - below <= c <= m + above, (g, lg, c, m)


def test_edges_follow(packaged, tmp_path):
    from liblightzk_b200 import autotune as a
    a.load(a.DEFAULT_TABLES["B200"])
    for g in (1, 2):
        for k in ("window", "chunk", "run"):
            for lg in set(range(33)) - set(a.PLAIN_CLASSES[g]):
                a.set_value(k, g, lg, 0)
        for k in ("table_window", "table_chunk", "table_run"):
            for lg in range(a.TABLE_CLASSES[g][0]):
                a.set_value(k, g, lg, 0)
    for lg in set(range(33)) - set(a.NTT_CLASSES):
        a.set_value("ntt", 0, lg, 0)
    a.fill_edges()
    assert a.current() == packaged
