"""Moments of delays relative to bases of any magnitude: those whose square or
reciprocal no double holds, beside ordinary ones in the same type, every kind of delay
that scales with its base, equal numpy's quotients to the rounding of their sums."""
from __future__ import annotations

import numpy as np
import pytest

from mc_dagprop_gb300 import batching, inspection
from mcd_testlib import kitchen_sink

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-200, 1e-155, 3e-311, 1e150, 1e290, 1.0])
def test_relative_moments_over_the_range_of_bases(cuda, scale):
    flat, gen = kitchen_sink(seed=12, n_layers=4, width=40)
    keep = [g for g in gen if g[0] != "empirical_absolute"]  # (those delays do not scale)
    keep.append(("empirical_relative", 8, np.linspace(0.0, 0.5, 16), np.full(16, 1.0 / 16.0)))  # counted by entry
    flat["act_duration"] = flat["act_duration"] * np.where(np.arange(len(flat["act_duration"])) % 3, scale, 1.0)
    prop = batching.compile_dag(flat, keep)
    seeds = np.arange(300, dtype=np.int64) * 31 + 7
    _, dur, _ = prop.run_many_arrays(seeds)
    acts = {k: flat[k] for k in ("act_idx", "act_duration", "act_type")}
    res = inspection.delay_histograms(prop, acts, seeds, bins=20)
    for t, entry in res.items():
        sel = flat["act_type"] == t
        base = flat["act_duration"][sel]
        x = ((dur[:, flat["act_idx"][sel]] - base) / base).ravel()
        e = entry["relative"]
        tol = 2.0 * x.size * 2.0**-53  # of a sum of n terms in any order, and its terms' own rounding
        assert e["count"] == x.size
        assert abs(e["mean"] - x.mean()) <= tol * np.abs(x).max(), t
        assert abs(e["var"] - x.var()) <= 4.0 * tol * (x * x).max(), t
