"""The per-step LIF kernels against the oracle, bit for bit. A run of several steps with a raster goes by delay
windows, so these take one step per call, the state carried over, or run without a raster."""
import numpy as np
import pytest
import torch

import oracle
from flyb200 import _abi, autotune
from gpu_helpers import LIF_ARRAYS, native_lif_run
from test_gpu_lif import PERS, STEP, case_19cell, case_random
from test_gpu_windows import brain

pytestmark = pytest.mark.gpu


def compare(case, launch, block=256, raster=True, **kw):
    ref, gpu = case["state"].copy(), case["state"].copy()
    counters = [None if case.get("fly_steps") is None else case["fly_steps"].copy() for _ in range(2)]
    common = dict(n_delay=case["n_delay"], flags=case["flags"], seed=case.get("seed", 0), raster=raster,
                  adapt_jump=case.get("adapt_jump"))
    steps, uniforms = case["nsteps"], case["uniforms"]
    r_ref, ev_ref = oracle.lif_run(ref, case["ptr"], case["edges"], case["P"], nsteps=steps, uniforms=uniforms,
                                   fly_steps=counters[0], **common)
    per_call = 1 if raster else steps
    rows, events = [], 0
    for s in range(0, steps, per_call):
        r, ev = native_lif_run(gpu, case["ptr"], case["edges"], case["P"], nsteps=per_call, launch=launch, block=block,
                               uniforms=None if uniforms is None else uniforms[s:s + per_call], fly_steps=counters[1],
                               **common, **kw)
        rows.append(r)
        events += ev
    if raster:
        assert r_ref.any()
        np.testing.assert_array_equal(np.concatenate(rows), r_ref)
    for name in LIF_ARRAYS:
        np.testing.assert_array_equal(getattr(gpu, name), getattr(ref, name), err_msg=name)
    np.testing.assert_array_equal(gpu.ring, ref.ring)
    assert events == ev_ref > 0
    if counters[0] is not None:
        np.testing.assert_array_equal(*counters)


@pytest.mark.parametrize("ipt", [1, 2, 4])
@pytest.mark.parametrize("launch,block,batch", [(STEP, 256, 64), (PERS, 256, 64), (STEP, 128, 3), (PERS, 512, 5)])
def test_items_per_thread(ipt, launch, block, batch):
    compare(case_random(batch=batch, n=2999, steps=40), launch, block, items_per_thread=ipt)


@pytest.mark.parametrize("kind", ["count", "fixed", "episodes", "depression"])
@pytest.mark.parametrize("staged,defer", [(1, False), (0, True), (1, True)])
@pytest.mark.parametrize("block,ipt", [(256, 2), (256, 4), (128, 2), (512, 2), (256, 1)])
def test_staged_and_deferred_launches(kind, staged, defer, block, ipt):
    case = case_random(batch=20, n=2999, steps=30, fixed=kind == "fixed", episodes=kind == "episodes",
                       std=kind == "depression", ext_uniform=kind == "depression")
    compare(case, STEP, block, items_per_thread=ipt, staged=staged, defer=defer)


@pytest.mark.parametrize("staged,defer", [(1, False), (1, True), (0, True)])
@pytest.mark.parametrize("n,batch", [(2999, 3), (1001, 1), (63, 2)])
def test_staged_request_falls_back_where_items_do_not_align(n, batch, staged, defer):
    compare(case_random(batch=batch, n=n, edges=20 * n, steps=40), STEP, staged=staged, defer=defer)


@pytest.mark.parametrize("staged", [0, 1])
@pytest.mark.parametrize("extra", [1023, 1024, 5000])
def test_deferred_lists_split_hubs(staged, extra):
    """A hub with more out-edges than one list entry covers, and one with exactly a whole number of entries."""
    case = case_random(batch=4, n=3000, edges=60_000, steps=40)
    rng = np.random.default_rng(11)
    ptr, e = case["ptr"], case["edges"]
    more = extra + 1 - int(ptr[1])                     # neuron 0's out-degree becomes extra + 1
    hub = np.stack([rng.integers(0, 3000, more), np.ones(more, np.int64)], 1)
    case["edges"] = np.concatenate([e[: ptr[1]], hub, e[ptr[1]:]]).astype(np.int32)
    case["ptr"] = np.concatenate([[0], ptr[1:] + more]).astype(np.int32)
    case["state"].poisson_p[0, :] = 0.5
    compare(case, STEP, items_per_thread=2, staged=staged, defer=True)


@pytest.mark.parametrize("launch,block", [(STEP, 128), (PERS, 256), (PERS, 512)])
@pytest.mark.parametrize("fixture", ["lif_19cell", "lif_19cell_adapt_by_type"])
def test_depression_and_adaptation(launch, block, fixture):
    compare(case_19cell(fixture), launch, block)


@pytest.mark.parametrize("launch", [STEP, PERS])
@pytest.mark.parametrize("kind", ["count", "fixed", "episodes", "depression"])
def test_runs_without_a_raster(launch, kind):
    """Several steps per launch: one grid barrier per step in the persistent kernel."""
    case = case_random(batch=5, n=2999, steps=50, fixed=kind == "fixed", episodes=kind == "episodes",
                       std=kind == "depression", ext_uniform=kind == "depression")
    compare(case, launch, raster=False)


@pytest.mark.parametrize("batch", [32, 64, 128, 256])
def test_every_launch_of_the_tuner_takes_the_same_single_steps(batch):
    """One step per call through every launch choice of the tuner, pulls among them."""
    states = []
    for launch, block, ipt, delivery in autotune.LIF_CANDIDATES:
        b = brain(batch, launch, "pull" in delivery)
        autotune._apply(b, {"launch": launch, "block": block, "items_per_thread": ipt, "delivery": delivery})
        for _ in range(21):
            b.step(1)
        b.check()
        states.append((b.v.clone(), b.ring.clone(), b.spike_counts.clone(), b.synaptic_events))
    assert float(states[0][2].sum()) > 0
    for v, ring, counts, events in states[1:]:
        assert torch.equal(v, states[0][0]) and torch.equal(ring, states[0][1]) and torch.equal(counts, states[0][2])
        assert events == states[0][3]
