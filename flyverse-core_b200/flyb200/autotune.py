"""Launch-parameter autotuner for the native steps, cached per (graph, batch, activity bucket).

The best launch shape depends on the graph, the batch and how many cells spike per step. Calls of
many steps mostly go by delay windows: one cooperative launch or two launches per window, the spikes
scattered or pulled. Engines that step by single launches stream the state from HBM every step:
there the register and the bulk-copy kernels, block sizes and deliveries differ. `tune_lif` times
each distinct candidate (launch mode x block size x items per thread x spike delivery) for a few steps on a
copy of the live state, restores the state, installs the fastest and caches it under the key;
`tune_optic` does the same for the optic substep's launch mode and kernel shape.
"""
from __future__ import annotations

import hashlib
import math

import numpy as np
import torch

from .optic import long_row_entries

CACHE: dict = {}
# (launch, block, items per thread, delivery): "fused" delivers spikes inside the update kernel,
# "staged" runs per-step launches through the bulk-copy kernel, "defer" lists the spikers and
# delivers them from a second, load-balanced kernel, "staged-defer" does both
LIF_CANDIDATES = (("step", 256, 4, "fused"), ("step", 256, 2, "fused"), ("step", 256, 1, "fused"),
                  ("step", 256, 2, "staged"), ("step", 512, 2, "staged"), ("step", 256, 4, "staged"),
                  ("step", 256, 2, "defer"), ("step", 256, 1, "defer"), ("step", 128, 2, "defer"),
                  ("step", 256, 4, "defer"), ("step", 256, 2, "staged-defer"), ("step", 512, 2, "staged-defer"),
                  ("step", 256, 4, "staged-defer"), ("persistent", 256, 4, "fused"), ("persistent", 512, 2, "fused"),
                  ("step", 256, 2, "pull"), ("step", 256, 1, "pull"), ("step", 256, 2, "staged-pull"),
                  ("step", 512, 2, "staged-pull"), ("step", 128, 2, "staged"), ("step", 128, 2, "staged-defer"),
                  ("step", 128, 2, "staged-pull"))


def graph_key(brain) -> str:
    h = hashlib.sha1()
    h.update(brain._out_ptr.cpu().numpy().tobytes())
    h.update(str((brain.n, brain.nnz, brain.ring_mode)).encode())
    return h.hexdigest()[:16]


def activity_bucket(brain, steps: int = 20) -> int:
    """log2 bucket of the fraction of (neuron, fly) pairs spiking per step, measured on a copy."""
    saved = brain.state_dict()
    before = float(brain.spike_counts.sum())
    rec = brain.record_activity
    brain.record_activity = True
    brain.step(steps)
    rate = (float(brain.spike_counts.sum()) - before) / (steps * brain.n * brain.B)
    brain.record_activity = rec
    brain.load_state_dict(saved)
    return int(math.floor(math.log2(max(rate, 1e-7))))


def _time(fn, reps: int) -> float:
    torch.cuda.synchronize()
    s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    s.record()
    for _ in range(reps):
        fn()
    e.record()
    e.synchronize()
    return s.elapsed_time(e) / reps


def one_by_one(brain, steps: int) -> None:
    """`steps` steps by single-step launches. A plain brain takes them whole; one that is stepped beside
    other work (`single_steps`) as WholeFly takes them: the update by two ranges of neurons (one over
    all of them would pull by itself), the clock, and under pull delivery a pull per complete group."""
    if not getattr(brain, "single_steps", False):
        for _ in range(steps):
            brain.step(1)
        return
    head = brain.n * 15 // 16 // 32 * 32
    for _ in range(steps):
        for first, count in ((0, head), (head, brain.n - head)):
            if count:
                brain.step_range(first, count)
        brain.advance(1, pull=False)
        if brain._pull_active() and brain.step_count % brain.pull_group == 0:
            brain.deliver()
    brain.deliver()


def _time_one_by_one(brain, steps: int) -> float:
    """Milliseconds per step of `one_by_one`, replayed from a CUDA graph: the host's time per launch is
    not what the candidates differ in. The graph holds whole delivery groups from a group's start
    on, as a caller's graph should: a pull across a group end walks the input tables twice."""
    L = brain.pull_group if brain._pull_active() else 1
    steps = -(-steps // L) * L
    one_by_one(brain, 2 + (-(brain.step_count + 2)) % L)
    stream, graph = torch.cuda.Stream(brain.device), torch.cuda.CUDAGraph()
    stream.wait_stream(torch.cuda.current_stream(brain.device))
    # (thread_local: other threads may allocate, copy and step their own brains meanwhile)
    with torch.cuda.stream(stream), torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        one_by_one(brain, steps)
    torch.cuda.current_stream(brain.device).wait_stream(stream)
    graph.replay()
    return _time(graph.replay, 1) / steps


def _time_run(brain, steps: int) -> float:
    """Milliseconds per step of a call of `steps` steps."""
    brain.step(2)
    return _time(lambda: brain.step(steps), 1) / steps


def _route(brain, candidate: tuple, steps: int) -> tuple:
    """What tells the kernels of a call of `steps` steps under the installed candidate from another's:
    by delay windows the launch mode and whether spikes are pulled, else the whole candidate."""
    launch, _, _, delivery = candidate
    return (launch, "pull" in delivery) if brain.window_steps(steps) else candidate


def tune_lif(brain, steps: int = 10, candidates=LIF_CANDIDATES) -> dict:
    """Install and return the fastest LIF launch choice for this brain; state is left unchanged.
    A brain with per-neuron clocks or the slow receptor tone has one launch shape (the extended
    kernel): nothing to tune. Calls of several steps mostly run by delay windows, where candidates
    that differ in the launch mode and the delivery alone are the same kernels: each such route is
    timed once, and among the candidates of the fastest the one with the fastest single steps is
    installed, since the brain's calls of one step run its shape. A brain that is stepped one step
    per launch (`single_steps`, set by WholeFly) is timed that way only."""
    if getattr(brain, "_kvec", None) is not None or getattr(brain, "slow", None) is not None:
        return {"launch": "step", "block": 256, "items_per_thread": 1, "delivery": "extended", "ms_per_step": None}
    single = bool(getattr(brain, "single_steps", False))
    key = ("lif", graph_key(brain), brain.B, activity_bucket(brain), single)
    if key in CACHE:
        _apply(brain, CACHE[key])
        return CACHE[key]
    saved = brain.state_dict()
    if not brain.can_pull():             # pull delivery: count ring and 32-fly groups only
        candidates = [c for c in candidates if "pull" not in c[3]]

    def timed(candidate, fn) -> float:
        _apply(brain, dict(zip(("launch", "block", "items_per_thread", "delivery"), candidate)))
        ms = fn(brain, steps)
        brain.load_state_dict(saved)
        return ms

    if single:
        results = {c: timed(c, _time_one_by_one) for c in candidates}
        best = min(results, key=results.get)
    else:
        runs, route_of = {}, {}
        for c in candidates:
            _apply(brain, dict(zip(("launch", "block", "items_per_thread", "delivery"), c)))
            route_of[c] = _route(brain, c, steps)
            if route_of[c] not in runs:
                runs[route_of[c]] = timed(c, _time_run)
        results = {c: runs[route_of[c]] for c in candidates}
        fastest = min(runs, key=runs.get)
        alike = [c for c in candidates if route_of[c] == fastest]
        ones = {c: timed(c, _time_one_by_one) for c in alike} if len(alike) > 1 else {alike[0]: 0.0}
        best = min(ones, key=ones.get)
    choice = {"launch": best[0], "block": best[1], "items_per_thread": best[2], "delivery": best[3],
              "ms_per_step": results[best],
              "all": {f"{k[0]}-{k[3]}/{k[1]}/{k[2]}": v for k, v in results.items()}}
    CACHE[key] = choice
    _apply(brain, choice)
    return choice


def _apply(brain, choice: dict) -> None:
    brain.launch, brain.block = choice["launch"], choice["block"]
    brain.items_per_thread = choice.get("items_per_thread", 0)
    delivery = choice.get("delivery", "fused")
    brain.staged = delivery in ("staged", "staged-defer", "staged-pull")
    brain.defer = delivery in ("defer", "staged-defer")
    brain.pull = delivery in ("pull", "staged-pull")
    brain._make_args()


# Row lengths above which a row is shared by a whole block (OpticCore.set_long_rows), tried beside the
# lobe's own default: the split pays at many flies per row gather and in small lobes; at one fly a
# row of a few hundred entries of a large lobe is better left to its warp slot.
OPTIC_LONG_ROWS = (96, 192, 384, 512, 768, 1024, 2048)


def optic_variants(batch: int, width: int) -> tuple:
    """The flyb_optic_args.variant values that are kernels of their own at a batch whose flies lie in
    vectors of `width` (4, 2 or 1); the others are refused or run as variant 0."""
    if batch == 1:
        return 0, 1, 2, 3, 4
    if batch <= 32 or width == 1:
        return (0,)
    if batch <= 64:
        return (0, 1, 2, 3, 4, 5) if width == 4 else (0, 4)
    if width == 2:
        return (0,)
    return (0, 1, 3) if batch <= 128 else (0, 1, 3, 5)


def _vector_width(core) -> int:
    arrays = (core.v_s, core.adapt_s, *core._bufs, core.pr_in, core.spk_in)
    return next(w for w in (4, 2, 1) if core.B % w == 0 and all(x.data_ptr() % (4 * w) == 0 for x in arrays))


def tune_optic(core, steps: int = 10) -> dict:
    """Pick the optic substep's launch mode, kernel shape (fly lanes x flies per lane x lanes per
    row, flyb_optic_args.variant) and long-row threshold by timing each on a copy of the state. A
    lobe advanced one substep per call beside other work (`single_steps`, set by WholeFly) keeps
    per-substep launches: a persistent kernel holds every SM until its last item, and the update
    that should run beside it waits (whole fly, 64 flies, end to end: 0.277 against 0.307 ms)."""
    single = bool(getattr(core, "single_steps", False))
    key = ("optic", core.m, core.W.nnz, core.B, single)
    if key in CACHE:
        core.launch, core.variant = CACHE[key]["launch"], CACHE[key]["variant"]
        core.set_long_rows(CACHE[key]["long_row"])
        return CACHE[key]
    v, a = core.v_s.clone(), core.adapt_s.clone()
    results = {}
    for long_row in sorted({*OPTIC_LONG_ROWS, long_row_entries(core.W.nnz, core.B)}):
        core.set_long_rows(long_row)
        for launch in ("step",) if single else ("step", "persistent"):
            for variant in optic_variants(core.B, _vector_width(core)):
                core.launch, core.variant = launch, variant
                core.substeps(2)
                # five calls: shapes 1 % apart alone may be 10 % apart beside other work (256 flies: variants 0
                # and 5 at 460 and 457 us per substep, the whole fly 1.176 and 1.062 ms)
                results[(launch, variant, long_row)] = _time(lambda: core.substeps(steps, carry=True), 5) / steps
                core.v_s.copy_(v)
                core.adapt_s.copy_(a)
    best = min(results, key=results.get)
    CACHE[key] = {"launch": best[0], "variant": best[1], "long_row": best[2], "ms_per_step": results[best],
                  "all": {f"{k[0]}/{k[1]}/{k[2]}": t for k, t in results.items()}}
    core.launch, core.variant = best[0], best[1]
    core.set_long_rows(best[2])
    return CACHE[key]


def summary() -> list:
    return [{"key": list(map(str, k)), **{kk: vv for kk, vv in v.items() if kk != "all"}} for k, v in CACHE.items()]
