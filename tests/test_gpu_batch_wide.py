"""Batches deep enough that their DAGs run wide tiles -- rows all on chip, and rows off
chip in each CTA's scratch -- beside DAGs too short for them and one whose window is off
chip: statistics equal those of 32-sample tiles (window in global memory, alone), and
the plan says what ran."""
from __future__ import annotations

import numpy as np
import pytest

from mc_dagprop_gb300 import _core, batching
from mcd_testlib import kitchen_sink

pytestmark = pytest.mark.gpu

KEYS = ("mean", "p50", "p90", "p99", "p_on_time", "hist")


@pytest.mark.parametrize("n_warps", [24, 12, 8])
def test_deep_batches_run_wide_tiles(cuda, n_warps):
    import torch

    deep = 100 * torch.cuda.get_device_properties(0).multi_processor_count  # three tiles an SM of one DAG
    widths = [130, 80, 130, 130, 80, 130, 130, 130]
    ns = [deep + 1, deep + 33, deep - 31, 1, 32, 33, 95, 64]
    dags = [kitchen_sink(seed=30 + i, n_layers=5, width=w) for i, w in enumerate(widths)]
    props = [batching.compile_dag(f, g, n_warps, "global" if i == 7 else "auto") for i, (f, g) in enumerate(dags)]
    assert not props[7].info()["window_in_smem"] and props[0].info()["window_in_smem"]
    batch = _core.Batch(props, list(range(8)), ns)
    plan = batch.plan
    if n_warps == 24:  # (a CTA has its SM to itself, and the rule is three tiles of work an SM)
        assert plan["wide_dags"] == 5  # all but the two of a single tile and the one off chip
        assert plan["queued_items"] == sum(-(-n // (64 if i in (0, 1, 2, 5, 6) else 32)) for i, n in enumerate(ns))
        assert plan["most_warps"] == 24
    assert batch.items == sum(-(-n // 32) for n in ns)
    for _ in range(2):
        batch.run()
    for i, ((f, g), n) in enumerate(zip(dags, ns)):
        alone = batching.compile_dag(f, g, 0, "global").run_stats(n=n, seed0=i, hist=True)
        got = batch.stats(i, True)
        assert all(np.array_equal(alone[k], got[k]) for k in KEYS), i


def test_whole_rounds_of_narrow_tiles_stay_narrow(cuda):
    """Three 32-sample tiles an SM of one DAG take less time than two rounds of wide ones; a
    tile more is a fourth round."""
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    prop = batching.compile_dag(*kitchen_sink(seed=40, n_layers=5, width=130), 24)
    wide = [_core.Batch([prop], [0], [n]).plan["wide_dags"] for n in (96 * sms - 31, 96 * sms, 96 * sms + 1)]
    assert wide == [0, 0, 1]
