"""Networks of narrow levels over many samples, whose launches take two or three warps a
CTA and many CTAs an SM, give the bits of a fixed count: sampled rows, given durations,
statistics."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from mc_dagprop_gb300 import batching
from mcd_testlib import kitchen_sink, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,layers", [(2, 30), (5, 40), (9, 5), (26, 6)])
@pytest.mark.parametrize("tiles", [5, 12, 13])
def test_few_warps_give_the_bits_of_a_fixed_count(cuda, width, layers, tiles):
    import torch

    flat, gen = kitchen_sink(seed=13, n_layers=layers, width=width)
    n = 32 * torch.cuda.get_device_properties(0).multi_processor_count * tiles - 17
    props = [batching.compile_dag(flat, gen, k) for k in (0, 7)]
    E, L = props[0].node_count(), props[0].activity_count()
    seeds = torch.arange(n, dtype=torch.int64, device="cuda") * 7919 + 5
    rows, given = [], []
    for p in props:
        h = C.c_void_p(p._handle())
        o = [torch.full((r, n), -7, dtype=t, device="cuda")
             for r, t in ((E, torch.float64), (L, torch.float64), (E, torch.int32), (E, torch.float64), (E, torch.int32))]
        torch.cuda.synchronize()
        assert lib().mcd_run_device(h, seeds.data_ptr(), n, *(t.data_ptr() for t in o[:3]), n, None) == 0
        assert lib().mcd_propagate_device(h, o[1].data_ptr(), n, n, o[3].data_ptr(), o[4].data_ptr(), n, None) == 0
        torch.cuda.synchronize()
        rows.append(o[:3])
        given.append(o[3:])
    for got in (rows, given):
        for a, b in zip(*got):
            assert torch.equal(a, b)
    assert torch.equal(rows[0][0], given[0][0]) and torch.equal(rows[0][2], given[0][1])
    a, b = (p.run_stats(n=n, seed0=3) for p in props)
    assert all(np.array_equal(a[k], b[k]) for k in ("mean", "p50", "p90", "p99", "p_on_time"))
