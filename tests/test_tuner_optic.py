"""The optic tuner times the threshold it would replace, and each kernel once (host logic; the shapes on a GPU)."""
import numpy as np
import pytest
import torch

from flyb200 import autotune, synthetic
from flyb200.optic import OpticCore, long_row_entries


class FakeCore:
    m, launch, variant, long_row = 3000, "persistent", 0, 0

    def __init__(self, nnz, batch):
        self.W, self.B = type("W", (), {"nnz": nnz}), batch
        self.v_s, self.adapt_s, self.pr_in, self.spk_in = (torch.zeros(16, batch) for _ in range(4))
        self._bufs = (torch.zeros(16, batch), torch.zeros(16, batch))

    def set_long_rows(self, long_row):
        self.long_row = long_row

    def substeps(self, steps, carry=False):
        if self.variant and self.B == 20:
            raise RuntimeError("no such shape")


@pytest.mark.parametrize("nnz,batch", [(100_000, 64), (1_340_000, 4), (600_000, 20), (6_000_000, 12)])
def test_the_lobes_own_threshold_is_among_those_timed(monkeypatch, nnz, batch):
    core, own = FakeCore(nnz, batch), long_row_entries(nnz, batch)
    monkeypatch.setattr(autotune, "CACHE", {})
    monkeypatch.setattr(autotune, "_time", lambda fn, reps: 1.0 if core.long_row == own else 2.0)
    assert autotune.tune_optic(core)["long_row"] == own == core.long_row


@pytest.mark.parametrize("batch,kernels", [(1, 5), (20, 1), (64, 6), (62, 2), (63, 1), (128, 3), (130, 1), (256, 4)])
def test_every_timing_is_of_another_kernel(monkeypatch, batch, kernels):
    core, taken = FakeCore(600_000, batch), []
    monkeypatch.setattr(autotune, "CACHE", {})
    monkeypatch.setattr(autotune, "_time", lambda fn, reps: taken.append((core.launch, core.variant, core.long_row)) or 1.0)
    autotune.tune_optic(core)
    own = {*autotune.OPTIC_LONG_ROWS, long_row_entries(600_000, batch)}
    assert len(taken) == len(set(taken)) == 2 * kernels * len(own)


@pytest.mark.gpu
@pytest.mark.parametrize("batch", [1, 3, 12, 33, 62, 64, 66, 127, 128, 130, 252, 255])
def test_every_variant_the_tuner_tries_is_accepted(batch):
    cfg = synthetic.optic_config3(seed=1, m=1200, nnz=36_000, n_pr=30, n_types=20, n_spk=40)
    core = OpticCore(cfg.W_rr(), cfg.a, cfg.b, batch=batch, device="cuda", gain_rr=cfg.gain_rr, adapt_gain=cfg.adapt_gain,
                     aad=cfg.aad)
    core.v_s.copy_(torch.from_numpy(np.random.default_rng(2).standard_normal((1200, batch)).astype(np.float32) * 0.3))
    start, ends = core.v_s.clone(), []
    for variant in autotune.optic_variants(batch, autotune._vector_width(core)):
        core.variant = variant
        core.v_s.copy_(start)
        core.adapt_s.zero_()
        core.substeps(3)
        core.check()
        ends.append(core.v_s.clone())
    for v in ends[1:]:
        torch.testing.assert_close(v, ends[0], rtol=1e-5, atol=1e-6)
