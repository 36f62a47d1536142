"""Sample counts on either side of where the few-sample kernels give way to the general
ones -- 16, 18 and 20 samples an SM by level width, stages and the share of entries that
draw -- against the general kernels (warps per CTA of the caller's choice), bit for bit."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from mc_dagprop_gb300 import batching
from mc_dagprop_gb300 import workloads as W
from mcd_testlib import lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers,width,types,limit", [(30, 20, 2, 20), (25, 60, 2, 16), (60, 60, 2, 18), (60, 30, 2, 20),
                                                      (60, 60, 5, 20)])
def test_rows_on_both_sides_of_the_limit(cuda, layers, width, types, limit):
    import torch

    rng = np.random.default_rng(layers)
    flat = W.layered_dag_fast(rng, layers, width, 3, [1, 2] if types == 2 else [1, 2, 3, 4, 5], 1800.0)
    gen = list(W.GEN_TWO_TYPES) if types == 2 else W.gen_five_types(rng)
    few, general = batching.compile_dag(flat, gen), batching.compile_dag(flat, gen, 24)
    E, L = few.node_count(), few.activity_count()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for n in (limit * sms - 1, limit * sms, limit * sms + 1):
        seeds = torch.arange(n, dtype=torch.int64, device="cuda") * 104729 + 17
        outs = []
        for p in (few, general):
            o = [torch.full((r, n), -7, dtype=t, device="cuda")
                 for r, t in ((E, torch.float64), (L, torch.float64), (E, torch.int32))]
            torch.cuda.synchronize()
            assert lib().mcd_run_device(C.c_void_p(p._handle()), seeds.data_ptr(), n, *(t.data_ptr() for t in o), n,
                                        None) == 0
            torch.cuda.synchronize()
            outs.append(o)
        for a, b in zip(*outs):
            assert torch.equal(a, b)
