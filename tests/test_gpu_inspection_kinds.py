"""Delay histograms over every delay kind, sample counts at the edges of a warp's
rounds, bases of zero and of either sign, links outside every class, and ranges
whose edges lie on table values: counts equal numpy's on the same durations."""
from __future__ import annotations

import numpy as np
import pytest

from mc_dagprop_gb300 import batching, inspection
from mcd_testlib import kitchen_sink
from test_gpu_inspection import numpy_bins

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,big,shift", [(1, False, 0.0), (127, False, 0.0), (1025, True, 0.0), (700, False, -120.0)])
def test_counts_equal_numpy_for_every_kind(cuda, n, big, shift):
    flat, gen = kitchen_sink(seed=9, n_layers=5, width=40, big_table=big)
    flat["act_duration"] = flat["act_duration"] + shift
    flat["act_duration"][::11] = 0.0
    prop = batching.compile_dag(flat, gen)
    seeds = np.arange(n, dtype=np.int64) * 31 + 7
    _, dur, _ = prop.run_many_arrays(seeds)
    keep = np.arange(len(flat["act_idx"])) % 7 != 3  # the other links belong to no class
    acts = {k: flat[k][keep] for k in ("act_idx", "act_duration", "act_type")}
    # table values on bin edges (types 8 and 10), a range that misses most delays (type 2)
    ranges = {8: (0.0, 300.0, -1.0, 1.0), 10: (20.0, 620.0, 0.0, 4.0), 2: (5.0, 5.5, 0.19, 0.2)}
    res = inspection.delay_histograms(prop, acts, seeds, bins=30, ranges=ranges)
    for t, entry in res.items():
        sel = acts["act_type"] == t
        base = acts["act_duration"][sel]
        d = dur[:, acts["act_idx"][sel]] - base
        rel = d[:, base != 0.0] / base[base != 0.0]
        for name, x in (("absolute", d.ravel()), ("relative", rel.ravel())):
            e = entry[name]
            got = np.concatenate([[e["under"]], e["counts"], [e["over"]]])
            lo, hi = (ranges[t][:2] if name == "absolute" else ranges[t][2:]) if t in ranges else \
                (e["edges"][0], e["edges"][-1])
            assert np.array_equal(got, numpy_bins(x, lo, hi, 30)), (t, name)
            assert e["count"] == x.size
            if x.size:
                assert abs(e["mean"] - x.mean()) <= 1e-12 * max(1.0, np.abs(x).max())
