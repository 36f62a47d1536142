"""Wide tiles (two samples a lane) against 32-sample tiles: the same bits from the
sampled outputs, the statistics and the gradient, with every window row on chip and
with rows off chip, at sample counts that leave a wide tile full, half empty or one
sample long."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from mc_dagprop_gb300 import batching

from mcd_testlib import kitchen_sink, lib

pytestmark = pytest.mark.gpu

WAVE = 152 * 32  # more samples than this on 152 SMs run wide tiles


def _device_run(prop, seeds):
    import torch

    n, E, L = len(seeds), prop.node_count(), prop.activity_count()
    s = torch.from_numpy(seeds).cuda()
    real = torch.empty((E, n), dtype=torch.float64, device="cuda")
    dur = torch.empty((L, n), dtype=torch.float64, device="cuda")
    cause = torch.empty((E, n), dtype=torch.int32, device="cuda")
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    assert lib().mcd_run_device(C.c_void_p(prop._handle()), s.data_ptr(), n, real.data_ptr(), dur.data_ptr(),
                                cause.data_ptr(), n, C.c_void_p(st.cuda_stream)) == 0
    torch.cuda.synchronize()
    return real.cpu().numpy(), dur.cpu().numpy(), cause.cpu().numpy()


# width 80 over 3 layers keeps a wide window on chip, width 130 does not (width 60: two
# narrow CTAs an SM, which stay narrow)
@pytest.mark.parametrize("width,preds", [(60, 4), (80, 4), (130, 4), (130, 12)])
@pytest.mark.parametrize("n", [2 * WAVE - 64, 2 * WAVE - 31, 2 * WAVE - 33, 2 * WAVE + 2 * WAVE - 127])
def test_wide_tiles_give_the_bits_of_narrow_ones(cuda, width, preds, n):
    flat, gen = kitchen_sink(seed=21, n_layers=7, width=width, max_preds=preds)
    seeds = np.random.default_rng(n).integers(0, 2**40, n)
    prop = batching.compile_dag(flat, gen)
    wide = _device_run(prop, seeds)
    cut = [0, WAVE // 2, WAVE, n // 2, n - WAVE // 2, n]  # at most a wave each: narrow tiles
    for b, e in zip(cut[:-1], cut[1:]):
        for k in range(b, e, WAVE):
            end = min(e, k + WAVE)
            for x, y in zip(wide, _device_run(prop, seeds[k:end])):
                assert np.array_equal(np.ascontiguousarray(x[:, k:end]).view(np.uint8), y.view(np.uint8))
    # statistics and gradient: integer sums over the same samples, off-chip windows run narrow tiles
    glob = batching.compile_dag(flat, gen, 0, "global")
    a, b = prop.run_stats(n=n, seed0=5, hist=True), glob.run_stats(n=n, seed0=5, hist=True)
    assert all(np.array_equal(a[k], b[k]) for k in ("mean", "p50", "p90", "p99", "p_on_time", "hist"))
    a, b = prop.gradient(n, 5), glob.gradient(n, 5)
    assert a["objective"] == b["objective"]
    assert np.array_equal(a["grad_earliest"], b["grad_earliest"]) and np.array_equal(a["grad_base"], b["grad_base"])


def test_large_windows_keep_rows_off_chip(cuda):
    """The cases above cover both plans: 130-wide levels need more rows than fit, 80-wide
    ones fit and leave no room for a second narrow CTA."""
    small, gen = kitchen_sink(seed=21, n_layers=7, width=80)
    large, _ = kitchen_sink(seed=21, n_layers=7, width=130)
    row = 64 * 8
    info = [batching.compile_dag(f, gen).info() for f in (small, large)]
    rest = [i["smem_bytes"] - i["window_slots"] * 256 for i in info]
    assert 2 * (info[0]["smem_bytes"] + 1024) > 228 * 1024
    assert info[0]["window_in_smem"] and info[0]["window_slots"] * row + rest[0] <= 226 * 1024
    assert info[1]["window_in_smem"] and info[1]["window_slots"] * row + rest[1] > 226 * 1024


def test_batches_run_wide_tiles_with_the_same_statistics(cuda):
    """A batch's items are wide where the DAG has them; alone, these sample counts run narrow."""
    from mc_dagprop_gb300 import _core

    ns = [1, 32, 33, 64, 95, 3000]
    props = [batching.compile_dag(*kitchen_sink(seed=30 + i, n_layers=5, width=w), 8)
             for i, w in enumerate([60, 130, 130, 80, 130, 130])]
    batch = _core.Batch(props, list(range(len(ns))), ns)
    for _ in range(2):
        batch.run()
    for i, (p, n) in enumerate(zip(props, ns)):
        a, b = batch.stats(i, True), p.run_stats(n=n, seed0=i, hist=True)
        assert all(np.array_equal(a[k], b[k]) for k in ("mean", "p50", "p90", "p99", "p_on_time", "hist")), i
