"""Frozen cells at rest are left untouched in every delay window of a run, not in the first alone. Their
refractory time is given as -0: an update would make it +0, an untouched cell keeps its sign bit."""
import numpy as np
import pytest

from flyb200 import _abi
from gpu_helpers import native_lif_run
from test_gpu_windows import problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("launch", [_abi.LAUNCH_STEP, _abi.LAUNCH_PERSISTENT])
@pytest.mark.parametrize("kind", ["count", "fixed", "depression"])
@pytest.mark.parametrize("batch,delay,steps", [(32, 5, 17), (1, 18, 56)])
def test_frozen_cells_at_rest_stay_untouched(launch, kind, batch, delay, steps):
    st, ptr, edges, P, flags = problem(batch, delay, delay + 1, kind)
    quiet = slice(320, 480)                       # whole warps of frozen cells without input
    st.res[quiet] = 1.0
    st.refrac[quiet] = -0.0
    native_lif_run(st, ptr, edges, P, raster=True, n_delay=delay, flags=flags, nsteps=steps, seed=77, launch=launch)
    assert np.signbit(st.refrac[quiet]).all()
    assert not st.spikes[quiet].any() and (st.res[quiet] == 1.0).all() and st.spikes.any()
