"""Propagation of given durations at the edges of what the kernel reads ahead: events
of 1 to 12 predecessors (four are read ahead), durations of every sign with infinities,
NaN and zeros of both signs, narrow and wide tiles, the window on chip, partly off chip
and off chip -- bit for bit the oracle's rows."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import oracle
from mc_dagprop_gb300 import batching
from mcd_testlib import kitchen_sink, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,window", [(130, "auto"), (40, "auto"), (130, "global")])
@pytest.mark.parametrize("n", [1, 31, 9728 - 33])
def test_rows_equal_the_oracle(cuda, width, window, n):
    import torch

    flat, gen = kitchen_sink(seed=4, n_layers=5, width=width, max_preds=12)
    prop = batching.compile_dag(flat, gen, 0, window)
    E, L = prop.node_count(), prop.activity_count()
    rng = np.random.default_rng(n)
    dur = rng.uniform(-200.0, 900.0, (n, L))
    odd = rng.random((n, L)) < 0.02
    dur[odd] = rng.choice([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -1e300], int(odd.sum()))
    check = np.unique(rng.integers(0, n, 64))
    ro, co = oracle.OracleSim(flat, gen).propagate_given(np.ascontiguousarray(dur[check]))
    d = torch.from_numpy(np.ascontiguousarray(dur.T)).cuda()
    real = torch.empty((E, n), dtype=torch.float64, device="cuda")
    cause = torch.empty((E, n), dtype=torch.int32, device="cuda")
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    assert lib().mcd_propagate_device(C.c_void_p(prop._handle()), d.data_ptr(), n, n, real.data_ptr(),
                                      cause.data_ptr(), n, C.c_void_p(st.cuda_stream)) == 0
    torch.cuda.synchronize()
    got = np.ascontiguousarray(real.cpu().numpy()[:, check].T)
    same = (got.view(np.int64) == ro.view(np.int64)) | (np.isnan(got) & np.isnan(ro))
    assert same.all()
    assert np.array_equal(cause.cpu().numpy()[:, check].T, co)
