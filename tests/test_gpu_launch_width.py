"""Launches that choose their warps per CTA by the tile count (one tile, a ragged
few, one per SM and one more) give the bits of a fixed three-warp CTA."""
from __future__ import annotations

import numpy as np
import pytest

from mc_dagprop_gb300 import batching
from mcd_testlib import kitchen_sink

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("window", ["auto", "global"])
@pytest.mark.parametrize("n", [1, 33, 152 * 32, 152 * 32 + 1])
def test_automatic_width_gives_the_bits_of_a_fixed_width(cuda, n, window):
    flat, gen = kitchen_sink(seed=11, n_layers=6, width=37)
    seeds = np.arange(n, dtype=np.int64) * 7919 + 5
    auto = batching.compile_dag(flat, gen, 0, window)
    fixed = batching.compile_dag(flat, gen, 3, window)
    for a, b in zip(auto.run_many_arrays(seeds), fixed.run_many_arrays(seeds)):
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
    a, b = auto.run_stats(n=n, seed0=3), fixed.run_stats(n=n, seed0=3)
    for k in ("mean", "p50", "p90", "p99", "p_on_time"):
        assert np.array_equal(a[k], b[k])
    a, b = auto.gradient(n, 3), fixed.gradient(n, 3)
    assert a["objective"] == b["objective"] and np.array_equal(a["grad_base"], b["grad_base"])
    assert np.array_equal(a["grad_earliest"], b["grad_earliest"])
