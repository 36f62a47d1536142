"""Device memory for the off-chip window rows of wide tiles: taken only by runs that wide
tiles run."""
from __future__ import annotations

import numpy as np
import pytest

from mc_dagprop_gb300 import batching
from mcd_testlib import kitchen_sink

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _free(torch):
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_statistics_by_narrow_tiles_take_no_rows(cuda):
    import torch

    flat, gen = kitchen_sink(seed=21, n_layers=7, width=130)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    # three 32-sample tiles an SM run narrow (two wide ones would take longer), six run wide
    warm = batching.compile_dag(flat, gen)
    for tiles in (3, 6):
        warm.run_stats(n=tiles * 32 * sms, seed0=5)  # loads the kernels
    took = {}
    for tiles in (3, 6):
        prop = batching.compile_dag(flat, gen)
        before = _free(torch)
        prop.run_stats(n=tiles * 32 * sms, seed0=5)
        took[tiles] = before - _free(torch)
    assert took[3] <= 6 * MIB < took[6], took


def test_the_gradients_rows_count_in_its_budget(cuda, monkeypatch):
    import torch

    flat, gen = kitchen_sink(seed=21, n_layers=7, width=130)
    n = 65536
    first = batching.compile_dag(flat, gen)
    want = first.gradient(n, 5)
    records = 6 * first.node_count() * n
    full = want["buffer_bytes"]
    assert want["level_blocks"] == 1 and full > records  # the records and the rows
    budget = (records + (full - records) // 2) // MIB
    monkeypatch.setenv("MCD_ADJ_BUDGET_MB", str(budget))
    prop = batching.compile_dag(flat, gen)
    before = _free(torch)
    got = prop.gradient(n, 5)
    assert before - _free(torch) <= (budget + 8) * MIB
    assert got["buffer_bytes"] <= budget * MIB
    assert got["objective"] == want["objective"]
    assert all(np.array_equal(got[k], want[k]) for k in ("grad_earliest", "grad_base"))
