"""How far rounding takes the analytic engine from the same fold in extended precision
(every step of it, the probabilities passed from event to event included): relative
2-norms over networks of 20 levels, most of whose events keep much of their mass on
their earliest time.  In double precision with each probability divided by the kept
mass the mean of the four norms is 2.8e-17 (restated with numpy), with one rounded
factor for all of an event's probabilities 4.9e-17: the bound is between them."""
from __future__ import annotations

import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))

import analytic_oracle as AO  # noqa: E402
from test_gpu_analytic import run_flat  # noqa: E402

pytestmark = pytest.mark.gpu

X = np.longdouble


def extended(ctx):
    """Probabilities of every event; activity PMFs of mass one, mass outside an event's
    window put on its bounds, starts on the step grid of one."""
    E = len(ctx["earliest"])
    probs, first = [np.ones(1, X)] * E, [float(round(e)) for e in ctx["earliest"]]
    rows = {int(t): k for k, t in enumerate(ctx["target"])}
    for e in range(E):  # (numbered level by level)
        if e not in rows:
            continue
        parts = []
        for p in range(ctx["pred_off"][rows[e]], ctx["pred_off"][rows[e] + 1]):
            s, k = int(ctx["pred_src"][p]), int(ctx["pred_pmf"][p])
            q = ctx["pmf_probs"][ctx["pmf_off"][k]:ctx["pmf_off"][k + 1]].astype(X)
            parts.append((int(first[s] + ctx["pmf_first"][k]), np.convolve(probs[s], q / q.sum())))
        lo = min(f for f, _ in parts)
        n = max(f + len(c) for f, c in parts) - lo
        r = None
        for f, c in parts:
            x = np.zeros(n, X)
            x[f - lo:f - lo + len(c)] = c
            below = np.concatenate([np.zeros(1, X), np.cumsum(x)[:-1]])
            r, b = (x, below) if r is None else (r * (below + x) + x * b, b * below)
        a, z = int(round(ctx["earliest"][e])) - lo, int(round(ctx["latest"][e])) - lo + 1
        a, z = max(a, 0), min(z, n)
        if a >= n:  # all of it early
            first[e] = float(round(ctx["earliest"][e]))
            continue
        kept = r[a:z].copy()
        kept[0] += r[:a].sum()
        kept[-1] += r[z:].sum()
        probs[e], first[e] = kept / kept.sum(), float(lo + a)
    return first, probs


def network(seed, layers=20, width=8, bins=120):
    """Events every 60 s or so, activities of 30 to 300 s with exponential delays."""
    rng = np.random.default_rng(seed)
    E = layers * width
    earliest = np.repeat(60.0 * np.arange(layers), width) + rng.integers(0, 30, E)
    acts, prec = {}, []
    for t in range(width, E):
        k, preds = t // width, []
        for s in rng.choice(np.arange(max(0, k - 3) * width, k * width), size=int(rng.integers(1, 5)), replace=False):
            base = float(rng.integers(30, 300))
            w = np.exp(-np.arange(bins) / (rng.uniform(0.05, 0.15) * base))
            acts[(int(s), t)] = (len(acts), base + np.arange(bins), w / w.sum())
            preds.append((int(s), len(acts) - 1))
        prec.append((t, preds))
    return AO.flatten(earliest, earliest + 600.0, acts, prec, 1, 1, 1)


def test_no_common_rounding_of_an_events_probabilities(cuda):
    norms = []
    for seed in (1, 2, 3, 4):
        ctx = network(seed)
        first, probs = extended(ctx)
        got = run_flat(ctx)
        assert np.array_equal(got[0], first)
        want = np.concatenate(probs)
        off = np.concatenate(got[2]) - want
        norms.append(float(np.sqrt((off * off).sum() / (want * want).sum())))
    assert np.mean(norms) <= 3.7e-17, norms


def test_a_kept_mass_too_small_for_its_reciprocal(cuda):
    q = np.array([1.0, 0.0, 0.0, 1e-310])
    ctx = AO.flatten(np.array([0.0, 3.0]), np.array([0.0, 3.0]), {(0, 1): (0, np.arange(4.0), q)}, [(1, [(0, 0)])],
                     1, 3, 3)
    assert [r[1].tolist() for r in AO.run(ctx)] == [[1.0], [1.0]]
    assert [p.tolist() for p in run_flat(ctx)[2]] == [[1.0], [1.0]]
