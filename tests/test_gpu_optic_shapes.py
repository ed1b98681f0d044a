"""The optic substep's kernel shapes over the batch widths: every vector width (the batch a multiple of
4, of 2, odd), one and several vectors per lane, lobes of few and of many rows, and arrays that are
not aligned for the batch's vectors, each against the FP32 oracle."""
import numpy as np
import pytest
import torch

import oracle
from flyb200 import synthetic
from flyb200.optic import OpticCore, long_row_entries

pytestmark = pytest.mark.gpu

RTOL, ATOL = 1e-5, 1e-6        # the FP32 oracle sums a row's entries in another order


def check(m, batch, launch="persistent", offset=0, history=False):
    cfg = synthetic.optic_config3(seed=batch, m=m, nnz=30 * m, n_pr=300, n_types=40, n_spk=400)
    W, T = cfg.W_rr(), 6
    rng = np.random.default_rng(batch)
    v, ad, pr, spk = ((rng.standard_normal((m, batch)) * s).astype(np.float32) for s in (0.3, 0.05, 0.3, 0.1))
    core = OpticCore(W, cfg.a, cfg.b, batch=batch, device="cuda", gain_rr=cfg.gain_rr, adapt_gain=cfg.adapt_gain, aad=cfg.aad,
                     launch=launch)
    if offset:                 # state that starts `offset` floats into its allocation
        for name in ("v_s", "adapt_s", "pr_in", "spk_in"):
            setattr(core, name, torch.zeros(m * batch + offset, device="cuda")[offset:].view(m, batch))
    for to, x in zip((core.v_s, core.adapt_s, core.pr_in, core.spk_in), (v, ad, pr, spk)):
        to.copy_(torch.from_numpy(x))
    hist = [torch.zeros(T, m, batch, device="cuda") for _ in range(2)] if history else [None, None]
    core.substeps(T, *hist)
    torch.cuda.synchronize()
    core.check()
    want = oracle.optic_run(v, ad, W.indptr, W.indices, W.data, pr, spk, cfg.a, cfg.b, cfg.gain_rr, cfg.adapt_gain, cfg.aad, T,
                            history=history)
    np.testing.assert_allclose(core.v_s.cpu().numpy(), v, rtol=RTOL, atol=ATOL)
    np.testing.assert_allclose(core.adapt_s.cpu().numpy(), ad, rtol=RTOL, atol=ATOL)
    np.testing.assert_allclose(core.dr_out.cpu().numpy(), core.dr().cpu().numpy(), rtol=0, atol=0)
    if history:
        for got, x in zip(hist, want):
            np.testing.assert_allclose(got.cpu().numpy(), x, rtol=RTOL, atol=ATOL)


@pytest.mark.parametrize("batch", [1, 2, 3, 4, 5, 6, 8, 9, 10, 12, 17, 18, 20, 33, 34, 40, 62, 63, 66, 100, 127, 130, 132, 252,
                                   254, 255, 256])
def test_every_batch_shape_matches_oracle(batch):
    check(1200, batch, history=batch in (3, 6, 12, 33, 130, 252))


@pytest.mark.parametrize("batch", [1, 2, 4, 8])
def test_lobes_of_many_rows_match_oracle(batch):
    for m in (9472, 9473):                # a warp per row, and rows sharing a warp
        check(m, batch)
    check(9473, batch, launch="step")


@pytest.mark.parametrize("batch,offset", [(2, 1), (4, 1), (4, 2), (12, 1), (24, 2), (64, 1), (64, 2), (128, 3), (256, 1)])
def test_unaligned_state_matches_oracle(batch, offset):
    check(1200, batch, offset=offset)


def test_long_row_threshold_follows_the_lobe_and_the_batch():
    cases = {(0, 1): 192, (100_000, 64): 96, (1_340_000, 4): 212, (6_000_000, 1): 512, (6_000_000, 12): 512}
    assert {k: long_row_entries(*k) for k in cases} == cases
