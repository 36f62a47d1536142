"""The analytic fold where its work is cut: grids of one bin to several CTAs of a
cluster and past shared memory, one to many predecessors (groups of four, and more
than a CTA has threads), values off the step grid, sparse activity PMFs, every flow
rule -- against the oracle (supports exactly, probabilities within 1e-12)."""
from __future__ import annotations

import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))

import analytic_oracle as AO  # noqa: E402
from test_gpu_analytic import compare, run_flat  # noqa: E402

pytestmark = pytest.mark.gpu


def star(seed, n_preds, bins, rule=1, step=1, window=None, offset=0.0, sparse=False):
    """n_preds origins into one event, and that event into a second one: the maximum
    over n_preds shifted activity PMFs, then a convolution of its result."""
    rng = np.random.default_rng(seed)
    acts, prec = {}, []
    for p in range(n_preds):
        w = rng.random(bins)
        if sparse:
            w[rng.random(bins) < 0.9] = 0.0
            w[rng.integers(bins)] = 1.0
        first = float(rng.integers(0, 2 * bins + 1)) * step + (offset if p % 2 else 0.0)
        acts[(p, n_preds)] = (p, first + step * np.arange(bins), w / w.sum())
    prec.append((n_preds, [(p, p) for p in range(n_preds)]))
    w = rng.random(max(1, bins // 2))
    acts[(n_preds, n_preds + 1)] = (n_preds, step * np.arange(len(w)) * 1.0, w / w.sum())
    prec.append((n_preds + 1, [(n_preds, n_preds)]))
    E = n_preds + 2
    lo = float(bins // 3 * step)
    earliest = np.r_[np.zeros(n_preds), lo, lo]
    latest = earliest + (float(6 * bins * step) if window is None else window)
    return AO.flatten(earliest, latest, acts, prec, step, rule, rule), E


def check(ctx, E):
    ref = AO.run(ctx)
    compare(run_flat(ctx), np.array([r[0] for r in ref]), np.array([len(r[1]) for r in ref]),
            np.concatenate([r[1] for r in ref]), np.array([r[2] for r in ref]), np.array([r[3] for r in ref]))


@pytest.mark.parametrize("n_preds", [1, 2, 4, 5, 9, 130])
@pytest.mark.parametrize("bins", [1, 2, 33, 300])
def test_predecessor_counts_and_grid_sizes(cuda, n_preds, bins):
    check(*star(n_preds * 1000 + bins, n_preds, bins))


@pytest.mark.parametrize("bins", [4100, 12001])
def test_segments_at_and_past_shared_memory(cuda, bins):
    check(*star(bins, 3, bins))


@pytest.mark.parametrize("rule", [1, 2, 3])
@pytest.mark.parametrize("window", [0.0, 40.0, 333.0])
def test_rules_on_narrow_windows(cuda, rule, window):
    ctx, E = star(7 + rule, 5, 120, rule=rule, window=window)
    try:
        AO.run(ctx)
    except ValueError:
        with pytest.raises(ValueError):
            run_flat(ctx)
        return
    check(ctx, E)


@pytest.mark.parametrize("step", [1, 7])
@pytest.mark.parametrize("sparse", [False, True])
def test_steps_and_sparse_activities(cuda, step, sparse):
    check(*star(step, 6, 250, step=step, sparse=sparse))


def test_starts_off_the_step_grid(cuda):
    # half a step between the predecessors' grids: starts rounded half to even, as the oracle does
    check(*star(3, 4, 60, step=2, offset=1.0))
