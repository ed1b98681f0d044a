"""Delay windows (runs of more than one LIF step): bit for bit the oracle's per-step run, and a
Brain advanced by windows bit for bit the same Brain advanced one step per call."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

import oracle
from flyb200 import _abi, synthetic
from flyb200.brain import Brain, LIFParams, lif_coefficients, out_edges
from gpu_helpers import LIF_ARRAYS, native_lif_run

pytestmark = pytest.mark.gpu

STEP, PERS = _abi.LAUNCH_STEP, _abi.LAUNCH_PERSISTENT


def problem(batch, delay, slots, kind, n=1500, seed=0):
    """A random graph with a hub, whole warps of frozen cells at rest, a few frozen cells elsewhere and,
    on the fixed ring, cells of fractional `active` (they transmit that amount)."""
    rng = np.random.default_rng(seed)
    pre, post = rng.integers(0, n, 20 * n), rng.integers(0, n, 20 * n)
    pre = np.concatenate([pre, np.full(n, 700)])                       # the hub reaches every cell
    post = np.concatenate([post, np.arange(n)])
    quiet = (post >= 300) & (post < 500)                               # no input to the frozen block
    pre, post = pre[~quiet], post[~quiet]
    sign = np.where(rng.random(n) < 0.65, 1.0, -1.0).astype(np.float32)
    W = sp.csr_matrix((rng.geometric(0.25, pre.size).astype(np.float32) * sign[pre] * np.float32(0.275), (post, pre)),
                      shape=(n, n), dtype=np.float32)
    p = LIFParams(conn_cap=0.0, input_norm_alpha=0.0, path_gain=[], type_path_gain=[], same_type_gain=1.0,
                  adapt_jump=1.5, receptor_model=None, dt=0.1)
    std = kind == "depression"
    ptr, edges, mode = out_edges(W, p.w_syn, "auto" if kind == "count" else "fixed", std_on=std)
    st = oracle.LifState(n, batch, slots, mode, p.v_rest)
    st.v[:] = rng.uniform(-52.0, -45.2, st.v.shape)
    st.poisson_p[rng.choice(n, n // 10, replace=False)] = 0.02
    st.poisson_p[1200:1264] = 0.01                                     # warps of driven cells
    st.poisson_p[700] = 0.3
    st.drive[:] = rng.uniform(5.0, 8.0, st.drive.shape)
    st.active[rng.choice(n, n // 20, replace=False)] = 0.0
    st.active[300:500], st.drive[300:500], st.poisson_p[300:500], st.v[300:500] = 0.0, 0.0, 0.0, p.v_rest
    flags = _abi.LIF_POISSON | _abi.LIF_COUNTS | _abi.LIF_ADAPT | _abi.LIF_SKIP_FROZEN
    if kind != "count":
        st.active[rng.choice(np.arange(600, n), 40, replace=False)] = 0.5
    if std:
        flags |= _abi.LIF_STD
        st.std_u[:] = rng.uniform(0.0, 0.5, n).astype(np.float32)
        st.res[:] = rng.uniform(0.5, 1.0, st.res.shape)
    return st, ptr, edges, lif_coefficients(p, std), flags


@pytest.mark.parametrize("launch", [STEP, PERS])
@pytest.mark.parametrize("kind", ["count", "fixed", "depression"])
@pytest.mark.parametrize("batch,delay,extra,steps", [
    (1, 2, 0, 7),         # the shortest window, an odd end
    (7, 5, 0, 13),        # an item count that ends mid-word
    (3, 18, 3, 37),       # more ring slots than the delay needs
    (2, 45, 0, 70),       # a delay longer than a window may be
    (1, 18, 0, 2),        # a run shorter than the delay
])
def test_windows_equal_oracle(launch, kind, batch, delay, extra, steps):
    st, ptr, edges, P, flags = problem(batch, delay, delay + 1 + extra, kind)
    kw = dict(n_delay=delay, flags=flags, nsteps=steps, seed=77)
    ref, gpu = st.copy(), st.copy()
    for uniforms in (None, np.random.default_rng(1).random((steps, st.n, batch), dtype=np.float32)):
        kw["flags"] = flags | (0 if uniforms is None else _abi.LIF_EXT_UNIFORM)
        r_ref, ev_ref = oracle.lif_run(ref, ptr, edges, P, raster=True, uniforms=uniforms, **kw)
        r_gpu, ev_gpu = native_lif_run(gpu, ptr, edges, P, raster=True, uniforms=uniforms, launch=launch, **kw)
        assert r_ref.any()
        np.testing.assert_array_equal(r_gpu, r_ref)
        for name in LIF_ARRAYS:
            np.testing.assert_array_equal(getattr(gpu, name), getattr(ref, name), err_msg=name)
        np.testing.assert_array_equal(gpu.ring, ref.ring)
        assert ev_gpu == ev_ref


def brain(batch, launch, pull, std_u=0.0, delay=1.8):
    cfg = synthetic.lif_config1(seed=2, n=1500, edges=30_000)
    b = Brain(cfg.c, LIFParams(**{**cfg.params, "std_u": std_u, "delay": delay}), device="cuda", seed=9, batch=batch,
              launch=launch)
    b.record_activity = True
    b.set_poisson(cfg.poisson_idx, 400.0)
    b.set_drive(np.arange(cfg.c.n), 6.9)
    b.pull = pull
    b._make_args()
    return b


@pytest.mark.parametrize("batch,launch,pull,std_u", [(1, "persistent", False, 0.0), (6, "step", False, 0.3),
                                                     (6, "persistent", False, 0.3), (32, "step", True, 0.0),
                                                     (64, "step", True, 0.0), (128, "step", True, 0.0),
                                                     (256, "step", True, 0.0)])
def test_brain_by_windows_equals_one_step_per_call(batch, launch, pull, std_u):
    """Runs of 3, 50 and 9 steps from one call each (windows that start and end inside delivery groups
    and wrap the spike history) against the same steps one per call."""
    a, b = brain(batch, launch, pull, std_u), brain(batch, launch, pull, std_u)
    assert a._pull_active() == pull
    for steps in (3, 50, 9):
        a.step(steps)
        for _ in range(steps):
            b.step(1)
        for name in ("v", "g", "refrac", "rate", "adapt", "res", "spikes", "spike_counts"):
            assert torch.equal(getattr(a, name), getattr(b, name)), name
        assert torch.equal(a.ring, b.ring) and torch.equal(a._hist, b._hist) and torch.equal(a._clock, b._clock)
        assert a.synaptic_events == b.synaptic_events
    assert float(a.spike_counts.sum()) > 0
    a.check()


@pytest.mark.parametrize("batch", [32, 64, 128])
@pytest.mark.parametrize("counts", [1, 300])            # packed entries, and counts that need the plane table
def test_pulls_of_parts_of_groups_equal_the_scatter(batch, counts):
    """Calls of 1, 2, 3, ... steps, which pull parts of groups and across group ends, against the scatter."""
    cfg = synthetic.lif_config1(seed=2, n=1500, edges=30_000)
    cfg.c.W.data[::7] *= counts
    both = []
    for pull in (False, True):
        b = Brain(cfg.c, LIFParams(**cfg.params), device="cuda", seed=9, batch=batch, launch="step")
        b.record_activity, b.pull = True, pull
        b.set_poisson(cfg.poisson_idx, 400.0)
        b.set_drive(np.arange(cfg.c.n), 6.9)
        b._make_args()
        for steps in (1, 1, 2, 3, 1, 2, 2, 5, 1, 6, 20):
            b.step(steps)
        b.check()
        both.append(b)
    a, b = both
    assert b._pull_active() and b._pull_planes_n == (0 if counts == 1 else 16) and float(a.spike_counts.sum()) > 0
    assert torch.equal(a.ring, b.ring) and torch.equal(a.v, b.v) and a.synaptic_events == b.synaptic_events
