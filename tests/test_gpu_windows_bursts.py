"""Bursts that fill the rounds of a delay window's delivery, against the oracle."""
import numpy as np
import pytest

import oracle
from flyb200 import _abi
from flyb200.brain import LIFParams, lif_coefficients
from gpu_helpers import LIF_ARRAYS, native_lif_run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("launch", [_abi.LAUNCH_STEP, _abi.LAUNCH_PERSISTENT])
@pytest.mark.parametrize("fixed", [False, True])
@pytest.mark.parametrize("batch,first,firing", [(1, 0, 1023), (1, 0, 1024), (1, 7, 1025), (1, 0, 8192), (1, 33, 8260),
                                                (32, 0, 256), (256, 3, 9), (5, 100, 1700)])
def test_bursts(launch, fixed, batch, first, firing):
    """`firing` cells in a row spike together (more or fewer than a delivery round holds), some of them without
    targets, then fall silent until the burst returns through its synapses."""
    n, delay, steps = max(firing + first, 40) + 40, 6, 15
    rng = np.random.default_rng(firing)
    deg = rng.integers(0, 4, n)
    deg[first + 1] = 2000                                        # a hub among them
    ptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    post = rng.integers(0, n, ptr[-1])
    w = rng.integers(1, 9, ptr[-1]).astype(np.int32)
    edges = np.stack([post, w if not fixed else w.astype(np.float32).view(np.int32)], 1).astype(np.int32)
    p = LIFParams(receptor_model=None, dt=0.1)
    st = oracle.LifState(n, batch, delay + 1, _abi.RING_FIXED if fixed else _abi.RING_COUNT, p.v_rest)
    st.v[first:first + firing] = -30.0
    ref, gpu = st.copy(), st.copy()
    kw = dict(n_delay=delay, flags=_abi.LIF_COUNTS, nsteps=steps, seed=1, raster=True)
    r_ref, ev_ref = oracle.lif_run(ref, ptr, edges, lif_coefficients(p, False), **kw)
    r_gpu, ev_gpu = native_lif_run(gpu, ptr, edges, lif_coefficients(p, False), launch=launch, **kw)
    assert int(np.bitwise_count(r_ref[0]).sum()) == firing * batch
    np.testing.assert_array_equal(r_gpu, r_ref)
    for name in LIF_ARRAYS:
        np.testing.assert_array_equal(getattr(gpu, name), getattr(ref, name), err_msg=name)
    np.testing.assert_array_equal(gpu.ring, ref.ring)
    assert ev_gpu == ev_ref
