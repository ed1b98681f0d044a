"""Which multi-step runs go by delay windows."""
import pytest
import torch

from flyb200 import synthetic
from flyb200.brain import Brain, LIFParams

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("staged", [False, True])
@pytest.mark.parametrize("n,batch,ring,delay,lists", [(300, 4, "auto", 1.8, False), (300, 4, "auto", 0.2, True),
                                                      (21_000, 256, "auto", 1.8, True), (20_000, 256, "auto", 1.8, False),
                                                      (21_000, 128, "fixed", 0.5, True)])
def test_deferred_runs_keep_their_kernels_where_windows_are_slower(n, batch, ring, delay, lists, staged):
    """The deferred kernel leaves its entry count in the list's counter; windows do not touch the list."""
    cfg = synthetic.lif_config1(seed=2, n=n, edges=10 * n)
    runs = []
    for defer in (False, True):
        b = Brain(cfg.c, LIFParams(**{**cfg.params, "delay": delay}), device="cuda", seed=9, batch=batch, launch="step",
                  ring=ring)
        b.record_activity, b.defer, b.staged = True, defer, defer and staged
        b.set_poisson(cfg.poisson_idx, 3000.0)
        b._make_args()
        b.step(5)
        runs.append(b)
    a, b = runs
    assert torch.equal(a.v, b.v) and torch.equal(a.ring, b.ring) and a.synaptic_events == b.synaptic_events > 0
    assert (int(b._lists[0, 0][1]) > 0) == lists
