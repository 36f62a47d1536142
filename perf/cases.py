"""The work a user of this framework has it do, as cases to be timed and compared.

A case is a dict of plain values; ``prepare`` makes from it (and a seed) what a
user's program holds before the call -- a compiled DAG, sample seeds, output
buffers -- and ``run`` makes one pass through a public entry point:

    run        MonteCarloPropagator.run / run_many_arrays: results on the host
    device     mcd_run_device: results in device memory (sample-minor rows)
    given      mcd_propagate_device: propagation of durations the caller has
    stats      MonteCarloPropagator.run_stats: per-event statistics
    batch      batching.BatchRunner: statistics of many DAGs at once
    gradient   MonteCarloPropagator.gradient: objective and both gradients
    analytic   AnalyticPropagator.run_arrays: PMF propagation
    inspect    inspection.delay_histograms: histograms of delays by type

The DAGs, delay generators and sizes are those of the package's workloads and
benchmark: layered DAGs of 100 to 200,000 events (layers of 20 to 200, one
ragged), two or five delay types, 1 to 100,000 samples.  The request server runs
the batch kernels on requests that arrive at random; its passes are not
repeatable in time, so ``batch`` stands for it here.
"""
from __future__ import annotations

import ctypes
import math
import os

import numpy as np
import torch

import mc_dagprop_gb300 as mcd
from mc_dagprop_gb300 import analytic, batching, inspection
from mc_dagprop_gb300 import workloads as W

P = ctypes.c_void_p
EDGES_MOST = 200_000 * 2.5 * 9_728  # sample-edges of the largest listed case


def listed() -> list:
    return [
        # one simulation by seed, the reference's `run(seed)`: the smallest call there is
        dict(name="run one seed", kind="run", events=1_000, width=20, back=3, types=2, samples=1),
        # the reference-sized job: 10,000 seeds of the 1,000-event DAG, every result row on the host
        dict(name="run_many 10,000 seeds", kind="run", events=1_000, width=20, back=3, types=2, samples=10_000),
        # the 200,000-event network with all outputs kept on the device, two full waves of 32-sample tiles
        dict(name="device 200k events", kind="device", events=200_000, width=100, back=5, types=5, samples=9_728),
        # a regional network, ragged in every size, a sample count that fills a part of the device
        dict(name="device 20k events ragged", kind="device", events=20_017, width=37, back=3, types=5, samples=3_001),
        # durations that the caller drew or measured, propagated through the large network
        dict(name="given durations 200k", kind="given", events=200_000, width=100, back=5, types=5, samples=4_864),
        # statistics of a small network: the low end of a batch or a dashboard call
        dict(name="statistics small", kind="stats", events=203, width=20, back=3, types=2, samples=1_000),
        # statistics of a large request (serving's upper end of samples)
        dict(name="statistics 10k events", kind="stats", events=10_000, width=100, back=3, types=5, samples=65_536),
        # a mixed batch of networks, events 100-50,000 and samples 1,000-100,000, both log-uniform
        dict(name="batch of 32 DAGs", kind="batch", dags=32, types=2),
        # one optimisation step's gradient (10,000 events, 65,536 samples)
        dict(name="gradient 10k events", kind="gradient", events=10_000, width=100, back=3, types=5, samples=65_536),
        # analytic propagation of a short line
        dict(name="analytic 60 events", kind="analytic", layers=10, width=6, rule=1, bins=300),
        # analytic propagation of the 1,000-event network
        dict(name="analytic 1,000 events", kind="analytic", layers=50, width=20, rule=1, bins=300),
        # delay inspection of the 1,000-event network with five delay types
        dict(name="inspect 1,000 events", kind="inspect", events=1_000, width=20, back=3, types=5, samples=10_000, bins=64),
    ]


def _log(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["run", "device", "given", "stats", "batch", "gradient", "analytic", "inspect"])
    if kind == "batch":
        return dict(kind=kind, dags=rng.randint(2, 10), types=rng.choice([2, 5]))
    if kind == "analytic":
        rule = rng.choice([1, 1, 2, 3])
        return dict(kind=kind, layers=rng.randint(3, 50 if rule == 1 else 8), width=rng.randint(2, 20), rule=rule,
                    bins=rng.randint(20, 300))
    types = rng.choice([2, 5])
    width = _log(rng, 20, 200)
    back = rng.choice([3, 5])
    hi_ev = {"run": 200_000, "device": 200_000, "given": 200_000, "stats": 50_000, "gradient": 20_000, "inspect": 5_000}[kind]
    events = max(2 * width, _log(rng, 100, hi_ev))
    if kind == "run":  # results on the host: at most those of 10,000 seeds of 1,000 events
        samples = _log(rng, 1, max(1.0, min(10_000.0, 1e7 / events)))
    elif kind in ("device", "given"):
        most = EDGES_MOST if kind == "device" else EDGES_MOST / 2
        samples = _log(rng, 32, min(50_000.0, most / (2.5 * events)))
    elif kind == "inspect":
        samples = _log(rng, 300, min(20_000.0, 1e7 / events + 300))
    else:
        samples = _log(rng, 1_000, min(100_000.0, 6.5e8 / events))
    case = dict(kind=kind, events=events, width=width, back=back, types=types, samples=samples)
    if kind == "inspect":
        case["bins"] = rng.randint(8, 200)
    return case


# ---------------------------------------------------------------- inputs


# A case's network (who follows whom, the types of its activities) is its own; the
# seed gives the times, the durations, the delay laws' weights and the samples.


def _flat(case, seed):
    """(flat DAG, delay generator) of a case; an odd event count leaves the last layer short."""
    rng = np.random.default_rng([int(seed), 7])
    width = case["width"]
    layers = max(2, -(-case["events"] // width))
    types = [1, 2] if case["types"] == 2 else [1, 2, 3, 4, 5]
    flat = W.layered_dag_fast(np.random.default_rng([case["events"], width, case["back"], case["types"]]), layers, width,
                              case["back"], types, 3600.0 if case["back"] == 5 else 1800.0)
    _retime(flat, rng)
    gen = list(W.GEN_TWO_TYPES) if case["types"] == 2 else W.gen_five_types(rng)
    E = max(width + 1, min(case["events"], layers * width))
    if E < layers * width:  # drop the events past E: they are the last targets
        keep = int(flat["pred_offsets"][E - width])
        for k in ("act_idx", "act_duration", "act_type", "act_src", "act_dst", "pred_src", "pred_act"):
            flat[k] = flat[k][:keep]
        flat["earliest"] = flat["earliest"][:E]
        flat["target"] = flat["target"][:E - width]
        flat["pred_offsets"] = flat["pred_offsets"][:E - width + 1]
    return flat, gen


def _retime(flat, rng):
    flat["earliest"] = np.floor(flat["earliest"] / 60.0) * 60.0 + rng.uniform(0.0, 30.0, len(flat["earliest"]))
    flat["act_duration"] = rng.uniform(30.0, 300.0, len(flat["act_duration"]))


_lib = None


def _api():
    global _lib
    if _lib is None:
        lib = ctypes.CDLL(os.path.join(os.path.dirname(mcd.__file__), "_lib", "libmcdagprop_gb300.so"))
        lib.mcd_last_error.restype = ctypes.c_char_p
        lib.mcd_run_device.argtypes = [P, P, ctypes.c_int64, P, P, P, ctypes.c_int64, P]
        lib.mcd_propagate_device.argtypes = [P, P, ctypes.c_int64, ctypes.c_int64, P, P, ctypes.c_int64, P]
        _lib = lib
    return _lib


_the_stream = None


def _stream():
    """The stream of the user's program: its passes run one after another."""
    global _the_stream
    if _the_stream is None:
        _the_stream = torch.cuda.Stream()
    return _the_stream


def _analytic_context(case, seed):
    """A layered analytic network: exponential, gamma, empirical and constant
    activity PMFs of up to `bins` bins on a 1 s grid.  Rule 1 keeps the mass beyond an
    event's window (600 s) on its bound; the rules that take it off the bound run on
    short lines with wide windows, where every event keeps some mass inside."""
    laws = np.random.default_rng([int(seed), 11])
    layers, width, bins = case["layers"], case["width"], case["bins"]
    rng = np.random.default_rng([layers, width, bins, case["rule"]])
    headway, jitter, longest, window = (60, 30, 300, 600.0) if case["rule"] == 1 else (40, 5, 80, 1200.0)
    E = layers * width
    earliest = np.repeat(np.arange(layers) * headway, width) + rng.integers(0, jitter, E) * 1.0
    events = tuple(mcd.Event(str(i), mcd.EventTimestamp(e, e + window, e)) for i, e in enumerate(earliest))
    acts, precedence = {}, []
    for t in range(width, E):
        k = t // width
        pool = np.arange(max(0, k - 3) * width, k * width)
        preds = []
        sources = list(rng.choice(pool, size=min(len(pool), int(rng.integers(1, 5))), replace=False))
        if case["rule"] != 1 and all(s < (k - 1) * width for s in sources):
            sources[0] = int(rng.integers((k - 1) * width, k * width))
        for s in sources:
            base, law = int(rng.integers(30, longest)), int(rng.integers(0, 4))
            if law == 0:
                pmf = analytic.exponential_pmf(scale=laws.uniform(0.05, 0.15) * base, step=1, start=0, stop=bins)
            elif law == 1:
                pmf = analytic.gamma_pmf(shape=2.0, scale=laws.uniform(0.03, 0.07) * base, step=1, start=0.0, stop=float(bins))
            elif law == 2:
                w = np.zeros(bins + 1)
                w[:: max(1, bins // 15)] = 1.0
                w[w > 0] = laws.dirichlet(np.ones(int((w > 0).sum())))
                pmf = analytic.empirical_pmf(np.arange(bins + 1.0), w, step=1)
            else:
                pmf = analytic.constant_pmf(float(base // 2), step=1)
            acts[(int(s), t)] = (len(acts), analytic.AnalyticActivity(len(acts), pmf.shift(float(base))))
            preds.append((int(s), len(acts) - 1))
        precedence.append((t, preds))
    rule = case["rule"]
    return analytic.AnalyticContext(events, acts, tuple(precedence), 1, analytic.UnderflowRule(rule),
                                    analytic.OverflowRule(rule), 1800.0)


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng([int(seed), 3])
    state = {"case": case}
    if kind == "analytic":
        state["prop"] = analytic.create_analytic_propagator(_analytic_context(case, seed))
        return state
    if kind == "batch":
        items = []
        for flat, gen, n, _ in W.mixed_dags(case["dags"] * 10 + case["types"], case["dags"], 100, 50_000, 1_000, 100_000,
                                            case["types"] == 5, fast=True):
            _retime(flat, rng)
            items.append((flat, gen, n, int(rng.integers(0, 2**31))))
        state["runner"] = batching.BatchRunner(items, tune=False)
        return state
    flat, gen = _flat(case, seed)
    prop = batching.compile_dag(flat, gen)
    n, E, L = case["samples"], prop.node_count(), prop.activity_count()
    state.update(prop=prop, n=n, seed0=int(rng.integers(0, 2**31 - n)))
    if kind in ("run", "inspect"):
        state["seeds"] = rng.integers(0, 2**31, n)
        state["flat"] = flat
    if kind in ("device", "given"):
        _stream()
        f64 = dict(dtype=torch.float64, device="cuda")
        state["realized"] = torch.empty((E, n), **f64)
        state["cause"] = torch.empty((E, n), dtype=torch.int32, device="cuda")
        if kind == "device":
            state["seeds"] = torch.from_numpy(rng.integers(0, 2**31, n)).cuda()
            state["durations"] = torch.empty((L, n), **f64)
        else:
            state["durations"] = _durations(flat, n, seed)
    return state


def _durations(flat, n, seed):
    """Given durations [link][sample]: each link's minimal duration and an exponential delay."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    base = torch.from_numpy(np.ascontiguousarray(flat["act_duration"])).cuda()
    d = torch.empty((len(base), n), dtype=torch.float64, device="cuda").exponential_(10.0, generator=g)
    return d.add_(1.0).mul_(base[:, None])


# ---------------------------------------------------------------- one pass


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "analytic":
        first, _, length, probs, under, over = state["prop"].run_arrays()
        return {"first": first, "length": length, "probs": probs, "under": under, "over": over}
    if kind == "batch":
        runner = state["runner"]
        runner.run()
        st = [runner.stats(i) for i in range(case["dags"])]
        return {k: np.concatenate([s[k] for s in st]) for k in ("mean", "p50", "p90", "p99", "p_on_time")}
    prop = state["prop"]
    if kind == "run":
        if case["samples"] == 1:
            r = prop.run(int(state["seeds"][0]))
            return {"realized": r.realized, "durations": r.durations, "cause": r.cause_event}
        realized, durations, cause = prop.run_many_arrays(state["seeds"])
        return {"realized": realized, "durations": durations, "cause": cause}
    if kind == "stats":
        s = prop.run_stats(n=state["n"], seed0=state["seed0"])
        return {k: s[k] for k in ("mean", "p50", "p90", "p99", "p_on_time")}
    if kind == "gradient":
        g = prop.gradient(state["n"], state["seed0"])
        return {k: g[k] for k in ("objective", "grad_earliest", "grad_base")}
    if kind == "inspect":
        h = inspection.delay_histograms(prop, state["flat"], state["seeds"], bins=case["bins"])
        # (type 1 adds a constant factor: the variance of its delays relative to the base is rounding alone)
        return {t: [[v["counts"], v["under"], v["over"], v["count"], v["mean"]] + ([v["var"]] if t != 1 else [])
                    for v in d.values()] for t, d in h.items()}
    n, real, dur, cause = state["n"], state["realized"], state["durations"], state["cause"]
    h, stream = P(prop._handle()), P(_stream().cuda_stream)
    if kind == "device":
        rc = _api().mcd_run_device(h, state["seeds"].data_ptr(), n, real.data_ptr(), dur.data_ptr(), cause.data_ptr(), n, stream)
        out = {"realized": real, "durations": dur, "cause": cause}
    else:
        rc = _api().mcd_propagate_device(h, dur.data_ptr(), n, n, real.data_ptr(), cause.data_ptr(), n, stream)
        out = {"realized": real, "cause": cause}
    if rc != 0:
        raise RuntimeError(_api().mcd_last_error().decode())
    return out


# ---------------------------------------------------------------- what a pass cannot do without


def work(case) -> dict:
    """Bytes: each input read once, each output written once.  Operations: an
    addition and a maximum for each edge and sample (twice that with the backward
    half), a multiply-add for each pair of bins of a convolution."""
    kind = case["kind"]
    if kind == "analytic":
        edges = 2.5 * (case["layers"] - 1) * case["width"]
        events = case["layers"] * case["width"]
        pmf = 0.75 * case["bins"] + 0.25  # a quarter of the activities are constants of one bin
        return {"bytes": 8.0 * (edges * pmf + 600.0 * events), "flops": 2.0 * edges * 500.0 * pmf}
    if kind == "batch":  # means of the log-uniform laws
        ev = (50_000 - 100) / math.log(500.0)
        n = (100_000 - 1_000) / math.log(100.0)
        return {"bytes": case["dags"] * ev * (48 + 2.5 * 32 + 40), "flops": 2.0 * case["dags"] * 2.5 * ev * n}
    E = float(case["events"])
    L = 2.5 * (E - case["width"])
    n = float(case["samples"])
    dag = 48.0 * E + 32.0 * L
    if kind in ("run", "device"):
        return {"bytes": n * (12.0 * E + 8.0 * L) + dag, "flops": 2.0 * n * L}
    if kind == "given":
        return {"bytes": n * (12.0 * E + 8.0 * L) + dag, "flops": 2.0 * n * L}
    if kind == "stats":
        return {"bytes": dag + 40.0 * E, "flops": 2.0 * n * L}
    if kind == "gradient":
        return {"bytes": dag + 8.0 * (E + L), "flops": 4.0 * n * L}
    return {"bytes": dag + 8.0 * n, "flops": 2.0 * n * L}  # inspect


# ---------------------------------------------------------------- the same in 64 bits


def exact(case, seed):
    """Where the result follows from the inputs by arithmetic: the propagation of
    given durations and the analytic engine.  The other cases draw their delays
    from the framework's own random streams, which no other program defines."""
    if case["kind"] == "given":
        return _exact_given(case, seed)
    if case["kind"] == "analytic":
        return _exact_analytic(_analytic_context(case, seed))
    return None


def _exact_given(case, seed):
    """realized = min(max(earliest, min(realized[src] + duration, earliest + max_delay)), ...),
    predecessors in order and the last of equal ones named as the cause, level by level."""
    flat, _ = _flat(case, seed)
    dur = _durations(flat, case["samples"], seed)
    E = len(flat["earliest"])
    off, src = flat["pred_offsets"], flat["pred_src"]
    level, begin, count = np.zeros(E, np.int64), np.zeros(E, np.int64), np.zeros(E, np.int64)
    for k, t in enumerate(flat["target"]):
        begin[t], count[t] = off[k], off[k + 1] - off[k]
        if count[t]:
            level[t] = level[src[off[k]:off[k + 1]]].max() + 1
    order = np.argsort(level, kind="stable")
    bounds = np.searchsorted(level[order], np.arange(level.max() + 2))
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    early = dev(flat["earliest"])
    cap = early + flat["max_delay"]
    real = torch.empty((E, case["samples"]), dtype=torch.float64, device="cuda")
    cause = torch.full((E, case["samples"]), -1, dtype=torch.int32, device="cuda")
    for b, e in zip(bounds[:-1], bounds[1:]):
        ids = order[b:e]
        d_ids = dev(ids)
        best = early[d_ids][:, None].expand(-1, case["samples"]).clone()
        who = torch.full(best.shape, -1, dtype=torch.int32, device="cuda")
        for j in range(int(count[ids].max(initial=0))):
            has = np.flatnonzero(count[ids] > j)
            at = dev(has)
            p = begin[ids[has]] + j
            t = torch.minimum(real[dev(src[p].astype(np.int64))] + dur[dev(flat["pred_act"][p].astype(np.int64))],
                              cap[d_ids[at]][:, None])
            wins = t >= best[at]
            best[at] = torch.where(wins, t, best[at])
            who[at] = torch.where(wins, dev(src[p].astype(np.int32))[:, None], who[at])
        real[d_ids] = torch.minimum(best, cap[d_ids][:, None])
        cause[d_ids] = who
    return {"realized": real, "cause": cause}


def _near(a, b):
    return abs(a - b) <= 1e-15 + 1e-12 * abs(b)


def _scaled(p, mass):
    total = p.sum()
    return p * (mass / total) if total > 0 and not _near(total, mass) else p


def _joint(a, b):
    return 1.0 if _near(a.sum(), 1.0) and _near(b.sum(), 1.0) else a.sum() * b.sum()


def _clip(first, p, lo, hi, rule):
    """(first, probabilities, mass below, mass above) of a PMF on the integers within
    [lo, hi]: mass outside put on the bound (1), removed (2), or spread over the rest (3)."""
    v = first + np.arange(len(p))
    under, over = float(p[v < lo].sum()), float(p[v > hi].sum())
    inside = (v >= lo) & (v <= hi)
    v, p = v[inside], p[inside].copy()
    spread = 0.0
    if rule == 1:
        for mass, bound, at in ((under, lo, 0), (over, hi, -1)):
            if mass > 0.0 and not len(v):
                v, p = np.array([float(bound)]), np.array([mass])
            elif mass > 0.0:
                p[at] += mass
        under = over = 0.0
    elif rule == 3:
        spread, under, over = under + over, 0.0, 0.0
    if spread > 0.0:
        if p.sum() == 0.0:
            v, p = np.array([float(lo)]), np.array([spread])
        else:
            p = p + spread * (p / p.sum())
    target = max(0.0, 1.0 - (under + over))
    if p.sum() > 0.0:
        p = p / p.sum() * target
    elif target > 0.0:
        v, p = np.array([float(lo)]), np.array([target])
    total = p.sum() + under + over
    return float(v[0]), (p if _near(total, 1.0) else p / total), under, over


def _exact_analytic(ctx):
    """Every event's PMF: the maximum over its predecessors of their PMF convolved with
    the activity's, clipped to the event's window.  Laid out as run_arrays lays its
    arrays out: events in topological order, each with room for the bins that its
    window or its predecessors' ranges allow."""
    E = len(ctx.events)
    preds = {t: p for t, p in ctx.precedence_list}
    after = [[] for _ in range(E)]
    for e in range(E):
        for s, _ in preds.get(e, ()):
            after[s].append(e)
    left = [len(preds.get(e, ())) for e in range(E)]
    queue = [e for e in range(E) if not left[e]]
    pmf, room = [None] * E, [1] * E
    span = [None] * E
    under, over = np.zeros(E), np.zeros(E)
    for e in queue:
        for t in after[e]:
            left[t] -= 1
            if not left[t]:
                queue.append(t)
        ts = ctx.events[e].timestamp
        if e not in preds:
            pmf[e] = (float(round(ts.earliest)), np.ones(1))
            span[e] = (pmf[e][0], pmf[e][0])
            continue
        lo, hi = round(ts.earliest), round(min(ts.latest, ts.earliest + ctx.max_delay))
        best, ends = None, []
        for s, _ in preds[e]:
            act = ctx.activities[(s, e)][1].pmf
            q = act.probabilities
            ends.append((span[s][0] + act.values[0], span[s][1] + act.values[0] + len(q) - 1))
            f, p = pmf[s][0] + act.values[0], _scaled(np.convolve(pmf[s][1], q), _joint(pmf[s][1], q))
            if best is None:
                best = (f, p)
                continue
            g, r = best
            start, end = min(f, g), max(f + len(p), g + len(r))
            x, y = np.zeros(int(end - start)), np.zeros(int(end - start))
            x[int(g - start):int(g - start) + len(r)] = r
            y[int(f - start):int(f - start) + len(p)] = p
            cx, cy = np.cumsum(x), np.cumsum(y)
            best = (start, _scaled(x * cy + y * np.concatenate(([0.0], cx[:-1])), _joint(r, p)))
        first, p, under[e], over[e] = _clip(best[0], best[1], lo, hi, int(ctx.underflow_rule))
        pmf[e] = (first, p)
        span[e] = (float(lo), float(hi))
        room[e] = int(min(hi - lo + 1, math.floor(max(b for _, b in ends) - min(a for a, _ in ends)) + 3))
    probs = np.zeros(sum(room))
    at = 0
    for e in queue:
        probs[at:at + len(pmf[e][1])] = pmf[e][1]
        at += room[e]
    return {"first": np.array([p[0] for p in pmf]), "length": np.array([len(p[1]) for p in pmf], np.int64),
            "probs": probs, "under": under, "over": over}
