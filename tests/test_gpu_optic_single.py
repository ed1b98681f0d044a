"""One substep per call on a carried dr, persistent launch: it needs no scratch words, so calls on other
streams that use the same ones are left alone, and equals per-substep launches."""
import numpy as np
import pytest
import torch

from flyb200 import synthetic
from flyb200.optic import OpticCore

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [300, 1200, 9500])
@pytest.mark.parametrize("batch", [1, 3, 12, 64])
def test_single_carried_substeps_leave_the_scratch_words(m, batch):
    cfg = synthetic.optic_config3(seed=1, m=m, nnz=30 * m, n_pr=30, n_types=20, n_spk=40)
    cores = []
    for launch in ("persistent", "step"):
        core = OpticCore(cfg.W_rr(), cfg.a, cfg.b, batch=batch, device="cuda", gain_rr=cfg.gain_rr, adapt_gain=cfg.adapt_gain,
                         aad=cfg.aad, launch=launch)
        core.set_long_rows(40)
        core.v_s.copy_(torch.from_numpy(np.random.default_rng(2).standard_normal((m, batch)).astype(np.float32) * 0.3))
        core.substeps(2)
        core._sync.fill_(7)
        for _ in range(3):
            core.substeps(1, carry=True)
        core.check()
        assert bool((core._sync == 7).all())
        cores.append(core)
    a, b = cores
    assert torch.equal(a.v_s, b.v_s) and torch.equal(a.adapt_s, b.adapt_s) and torch.equal(a.dr_out, b.dr_out)
