"""A run of several steps over a range of neurons goes by delay windows too: bit for bit the same steps taken
one launch at a time over that range."""
import ctypes as ct

import pytest
import torch

from flyb200 import _abi
from test_gpu_windows import brain

pytestmark = pytest.mark.gpu


def run_range(b, first, count, steps):
    a = b._args
    a.flags, a.nsteps, a.uniforms = b._flags(False) | _abi.LIF_NO_ADVANCE, steps, None
    b._set_delivery(a, first, count)
    b._set_pull(a)
    a.n_first, a.n_count = first, count
    rc = b._lib.flyb_lif_run(ct.byref(a), torch.cuda.current_stream().cuda_stream)
    a.n_first, a.n_count = 0, 0
    assert rc == 0
    b.advance(steps)


@pytest.mark.parametrize("first,count", [(0, 480), (480, 1020), (0, 1500), (96, 33)])
@pytest.mark.parametrize("batch,launch,pull,std_u,steps", [(1, "step", False, 0.0, 40), (1, "persistent", False, 0.0, 40),
                                                           (6, "step", False, 0.3, 25), (7, "persistent", False, 0.3, 25),
                                                           (64, "step", True, 0.0, 3), (128, "step", True, 0.0, 2)])
def test_range_runs_equal_single_steps(batch, launch, pull, std_u, steps, first, count):
    if pull and count == 1500:            # a launch over all neurons would pull by itself
        count = 1408
    a, b = brain(batch, launch, pull, std_u), brain(batch, launch, pull, std_u)
    for x in (a, b):
        x.step(21)
    run_range(a, first, count, steps)
    for _ in range(steps):
        b.step_range(first, count)
        b.advance(1)
    for name in ("v", "g", "refrac", "rate", "adapt", "res", "spikes", "spike_counts"):
        assert torch.equal(getattr(a, name), getattr(b, name)), name
    assert torch.equal(a.ring, b.ring) and torch.equal(a._hist, b._hist) and torch.equal(a._clock, b._clock)
    assert a.synaptic_events == b.synaptic_events and float(a.spike_counts.sum()) > 0
