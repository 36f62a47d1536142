"""The pilot's ranges (extremes of every delay, absolute and relative, by type) against
their definition over all delays, on made-up durations: bases of both signs and zero,
NaN, a type without relative delays, no samples."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from mc_dagprop_gb300 import inspection


class _Propagator:
    def __init__(self, dur):
        self.dur = dur

    def activity_count(self):
        return self.dur.shape[1]

    def _handle(self):
        return 0

    def run_many_arrays(self, seeds):
        return None, self.dur[:len(seeds)], None


class _Library:
    def mcd_delay_histograms(self, h, seeds, n, cls, base, nc, bins, ranges, counts, moments):
        self.ranges = np.ctypeslib.as_array(ctypes.cast(ranges, ctypes.POINTER(ctypes.c_double)), (nc, 4)).copy()
        return 0


@pytest.mark.parametrize("samples", [0, 1, 40])
@pytest.mark.parametrize("nan", [False, True])
def test_ranges_are_the_extremes_of_every_delay(monkeypatch, samples, nan):
    rng = np.random.default_rng(samples)
    L = 30
    base = np.round(rng.normal(size=L) * 100.0) * (rng.random(L) > 0.2)
    typ = np.arange(L) % 4
    base[typ == 3] = 0.0
    dur = base * (1.0 + rng.exponential(size=(samples, L))) + rng.exponential(size=(samples, L))
    if nan and samples:
        dur[0, 1] = np.nan
    lib = _Library()
    monkeypatch.setattr(inspection, "_api", lambda: lib)
    flat = {"act_idx": np.arange(L), "act_duration": base, "act_type": typ}
    inspection.delay_histograms(_Propagator(dur), flat, np.arange(samples), bins=4)
    for t in range(4):
        d = dur[:, typ == t] - base[typ == t]
        b = base[typ == t]
        rel = d[:, b != 0.0] / b[b != 0.0]
        want = []
        for x in (d, rel):
            lo, hi = (x.min(), x.max()) if x.size else (0.0, 1.0)
            want += [lo, hi + max(1e-9, 1e-6 * (hi - lo))]
        assert np.array_equal(lib.ranges[t], want, equal_nan=True), t
