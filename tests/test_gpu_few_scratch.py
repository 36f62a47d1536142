"""Device memory that few-sample runs on device buffers keep: at most 2 GiB however much
a run took, 32 MiB once the handles are gone."""
from __future__ import annotations

import ctypes as C
import gc

import numpy as np
import pytest

from mc_dagprop_gb300 import batching
from mc_dagprop_gb300 import workloads as W
from mcd_testlib import lib

pytestmark = pytest.mark.gpu

GIB = 1 << 30


def test_what_is_kept_between_runs_is_bounded(cuda):
    import torch

    rng = np.random.default_rng(3)
    flat = W.layered_dag_fast(rng, 2000, 100, 3, [1, 2, 3, 4, 5], 1800.0)
    gen = W.gen_five_types(rng)
    n, st = 1216, torch.cuda.Stream()  # eight samples a CTA, some 5 GB of durations
    prop = batching.compile_dag(flat, gen)
    real = torch.empty((prop.node_count(), n), dtype=torch.float64, device="cuda")
    seeds = torch.arange(n, dtype=torch.int64, device="cuda")

    def run(p):
        assert lib().mcd_run_device(C.c_void_p(p._handle()), seeds.data_ptr(), n, real.data_ptr(), None, None, n,
                                    C.c_void_p(st.cuda_stream)) == 0
        torch.cuda.synchronize()

    small = batching.compile_dag(W.layered_dag_fast(rng, 20, 20, 3, [1, 2], 1800.0), list(W.GEN_TWO_TYPES))
    run(small)  # loads the kernels
    free = torch.cuda.mem_get_info()[0]
    run(prop)
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] <= 2 * GIB + (64 << 20)
    run(prop)
    assert free - torch.cuda.mem_get_info()[0] <= 2 * GIB + (64 << 20)
    del prop, small
    gc.collect()
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] <= 64 << 20
