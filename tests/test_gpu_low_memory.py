"""Calls on a device with little free memory: what a faster path would need beside the
general one's buffers must not make a call fail that the general one can answer.  The
memory is taken beforehand and given back after the call."""
from __future__ import annotations

import ctypes as C
from contextlib import contextmanager

import numpy as np
import pytest

from mc_dagprop_gb300 import _core, batching
from mc_dagprop_gb300 import workloads as W
from mcd_testlib import kitchen_sink, lib

pytestmark = pytest.mark.gpu

MIB = 1 << 20
KEYS = ("mean", "p50", "p90", "p99", "p_on_time")


@contextmanager
def only(left):
    """At most `left` bytes of device memory free."""
    import torch

    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    cu = C.CDLL("libcuda.so.1")
    took = []
    try:
        while torch.cuda.mem_get_info()[0] > left + 2 * MIB:
            d = C.c_uint64()
            size = (torch.cuda.mem_get_info()[0] - left) // (2 * MIB) * (2 * MIB)
            if cu.cuMemAlloc_v2(C.byref(d), C.c_size_t(size)) != 0:
                break
            took.append(d)
        yield
    finally:
        for d in took:
            assert cu.cuMemFree_v2(d) == 0


def test_few_samples_without_room_for_their_scratch(cuda):
    rng = np.random.default_rng(1)
    flat, gen = W.layered_dag_fast(rng, 500, 40, 3, [1, 2, 3, 4, 5], 1800.0), W.gen_five_types(rng)
    n, warm = 600, batching.compile_dag(flat, gen)
    seeds = np.arange(n, dtype=np.int64) * 31 + 7
    E, L = warm.node_count(), warm.activity_count()
    host = []
    for rows, size in ((E, 8), (L, 8), (E, 4)):  # page-locked, so that no copies are staged
        p = C.c_void_p()
        assert lib().mcd_host_alloc(rows * n * size, C.byref(p)) == 0
        host.append(p)

    def run(p):
        assert lib().mcd_run_many_host(C.c_void_p(p._handle()), seeds.ctypes.data, n, *host) == 0
        return [np.ctypeslib.as_array(C.cast(h, C.POINTER(t)), (rows * n,)).copy()
                for h, t, rows in zip(host, (C.c_int64, C.c_int64, C.c_int32), (E, L, E))]

    try:
        want = run(warm)
        run(batching.compile_dag(flat, gen, 24))  # (the general kernels, loaded)
        prop = batching.compile_dag(flat, gen)
        with only(n * (12 * E + 8 * L) + 100 * MIB):  # the rows, and less than the scratch
            got = run(prop)
        assert all(np.array_equal(a, b) for a, b in zip(got, want))
    finally:
        for p in host:
            lib().mcd_host_free(p)


def test_statistics_without_room_for_off_chip_rows(cuda):
    flat, gen = kitchen_sink(seed=21, n_layers=7, width=130)
    n = 400_000
    want = batching.compile_dag(flat, gen).run_stats(n=n, seed0=5)
    batching.compile_dag(flat, gen, 0, "global").run_stats(n=3000, seed0=5)
    batching.compile_dag(flat, gen).run_stats(n=3000, seed0=5)  # (narrow tiles, loaded)
    prop = batching.compile_dag(flat, gen)
    with only(64 * MIB):
        got = prop.run_stats(n=n, seed0=5)
    assert all(np.array_equal(got[k], want[k]) for k in KEYS)


def test_batches_without_room_for_off_chip_rows(cuda):
    import torch

    deep = 100 * torch.cuda.get_device_properties(0).multi_processor_count
    dags = [kitchen_sink(seed=30 + i, n_layers=5, width=130) for i in range(3)]
    props = [batching.compile_dag(f, g, 24) for f, g in dags]
    wide = _core.Batch(props, [0, 1, 2], [deep] * 3)
    assert wide.plan["wide_dags"] == 3
    wide.run()
    small = _core.Batch(props, [0, 1, 2], [100] * 3)  # (narrow tiles, loaded)
    small.run()
    narrow = None
    for left in range(4, 64, 2):  # the first that leaves room for anything leaves none for the rows
        with only(left * MIB):
            try:
                narrow = _core.Batch(props, [0, 1, 2], [deep] * 3)
                break
            except (RuntimeError, MemoryError):
                pass
    assert narrow.plan["wide_dags"] == 0
    narrow.run()
    for i in range(3):
        a, b = wide.stats(i), narrow.stats(i)
        assert all(np.array_equal(a[k], b[k]) for k in KEYS)
