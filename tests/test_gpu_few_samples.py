"""A handful of samples (lanes over predecessors) against the general kernels and the
oracle, bit for bit: every sampler, lists longer than the lanes, stages with more units
than threads, one stage, a window too large for tiles of 32, times of both signs, sample counts around the steps of a CTA's
samples and past the last, page-locked, ordinary and device buffers, two streams at once,
a captured stream."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import oracle
from mc_dagprop_gb300 import batching
from mcd_testlib import kitchen_sink, lib

pytestmark = pytest.mark.gpu


def _bits(a):
    return np.ascontiguousarray(a).view(np.int64)


@pytest.mark.parametrize("layers,width,preds,shift,big", [(6, 150, 12, 0.0, False), (40, 7, 4, -500.0, False),
                                                          (1, 3, 1, 0.0, False), (5, 900, 4, 0.0, True),
                                                          (9, 1100, 4, 0.0, False)])
@pytest.mark.parametrize("n", [1, 3, 8, 9, 153, 800, 1217, 3040, 3041])
def test_rows_equal_the_general_kernels_and_the_oracle(cuda, layers, width, preds, shift, big, n):
    flat, gen = kitchen_sink(seed=6, n_layers=layers, width=width, big_table=big, max_preds=preds)
    flat = dict(flat, earliest=flat["earliest"] + shift)
    prop, general = batching.compile_dag(flat, gen, 0, "auto"), batching.compile_dag(flat, gen, 24, "auto")
    E, L = prop.node_count(), prop.activity_count()
    seeds = np.arange(n, dtype=np.int64) * 104729 + 17 - (1 << 40)
    real, dur, cause = prop.run_many_arrays(seeds)
    for a, b in zip((real, dur), general.run_many_arrays(seeds)):
        assert np.array_equal(_bits(a), _bits(b))
    ro, co = oracle.OracleSim(flat, gen).propagate_given(dur)
    assert np.array_equal(_bits(real), _bits(ro)) and np.array_equal(cause, co)
    # ordinary memory, and outputs left out
    r2, c2 = np.empty((n, E)), np.empty((n, E), dtype=np.int32)
    for cp in (c2.ctypes.data, None):
        assert lib().mcd_run_many_host(C.c_void_p(prop._handle()), seeds.ctypes.data, n, r2.ctypes.data, None, cp) == 0
        assert np.array_equal(_bits(r2), _bits(ro)) and np.array_equal(c2, co)
    # given durations, of any value
    rng = np.random.default_rng(n)
    odd = rng.random((n, L)) < 0.05
    dur = np.where(odd, rng.choice([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -1e300], (n, L)), dur)
    ro, co = oracle.OracleSim(flat, gen).propagate_given(dur)
    real, cause = prop.propagate(dur)
    assert ((_bits(real) == _bits(ro)) | (np.isnan(real) & np.isnan(ro))).all()
    assert np.array_equal(cause, co)


@pytest.mark.parametrize("n", [5, 200, 1217])
def test_device_buffers_streams_and_capture(cuda, n):
    import torch

    flat, gen = kitchen_sink(seed=6, n_layers=40, width=37)
    prop, general = batching.compile_dag(flat, gen, 0, "auto"), batching.compile_dag(flat, gen, 24, "auto")
    E, L, ld = prop.node_count(), prop.activity_count(), n + 3

    def out():
        return [torch.full((r, ld), -7, dtype=t, device="cuda")
                for r, t in ((E, torch.float64), (L, torch.float64), (E, torch.int32))]

    def run(p, seeds, o, st):
        rc = lib().mcd_run_device(C.c_void_p(p._handle()), seeds.data_ptr(), n, *(t.data_ptr() for t in o), ld,
                                  C.c_void_p(st.cuda_stream))
        assert rc == 0

    def given(p, d, o, st):
        rc = lib().mcd_propagate_device(C.c_void_p(p._handle()), d.data_ptr(), ld, n, o[0].data_ptr(), o[2].data_ptr(),
                                        ld, C.c_void_p(st.cuda_stream))
        assert rc == 0

    seeds = [torch.arange(n, dtype=torch.int64, device="cuda") + 1000 * k for k in (1, 2)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    want, got, again, graphed = [out(), out()], [out(), out()], [out(), out()], out()
    torch.cuda.synchronize()
    for _ in range(3):  # the same handle on two streams
        for k in (0, 1):
            run(prop, seeds[k], got[k], streams[k])
    for k in (0, 1):
        run(general, seeds[k], want[k], streams[k])
        given(prop, got[k][1], again[k], streams[k])
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=streams[0]):
        run(prop, seeds[0], graphed, streams[0])
    g.replay()
    torch.cuda.synchronize()
    for k in (0, 1):
        for a, b in zip(got[k], want[k]):
            assert torch.equal(a.view(torch.int32), b.view(torch.int32))
        assert torch.equal(again[k][0], want[k][0]) and torch.equal(again[k][2], want[k][2])
    for a, b in zip(graphed, want[0]):
        assert torch.equal(a, b)


@pytest.mark.parametrize("n", [1, 40])
def test_a_dag_without_links_may_leave_the_durations_out(cuda, n):
    E = 700
    flat = dict(earliest=np.arange(E, dtype=np.float64), act_idx=np.zeros(0, np.int32), act_duration=np.zeros(0),
                act_type=np.zeros(0, np.int32), target=np.arange(1, E, dtype=np.int32),
                pred_offsets=np.arange(E, dtype=np.int64), pred_src=np.arange(E - 1, dtype=np.int32),
                pred_act=np.zeros(E - 1, np.int32), max_delay=1000.0)  # a chain over links past the last
    prop = batching.compile_dag(flat, [], 0, "auto")
    real, cause = np.empty((n, E)), np.empty((n, E), np.int32)
    assert lib().mcd_propagate_host(C.c_void_p(prop._handle()), None, n, real.ctypes.data, cause.ctypes.data) == 0
    assert np.array_equal(real, np.tile(flat["earliest"], (n, 1)))
    # a later event's own time exceeds its predecessor's: no cause
    assert (cause == -1).all()
