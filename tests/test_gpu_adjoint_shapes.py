"""The adjoint's kernel shapes over the batch widths (vectors of 4, 2 and 1 flies, one and several per
lane), lobes of many rows (rows sharing a warp) and transposed rows wide enough to take a whole warp,
each against FP64 autograd."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

from flyb200 import synthetic
from oracle import optic64
from test_gpu_adjoint import fp64, gpu_grads

pytestmark = pytest.mark.gpu


def problem(batch, m=400, nnz=9000, hubs=0, steps=25):
    cfg = synthetic.optic_config3(seed=7, m=m, nnz=nnz, n_pr=40, n_types=16, n_spk=50)
    if hubs:                              # unit 5 projects to `hubs` units: a transposed row that long
        rng = np.random.default_rng(0)
        post = rng.choice(m, hubs, replace=False)
        extra = sp.csr_matrix((rng.uniform(-0.05, 0.05, hubs).astype(np.float32), (post, np.full(hubs, 5))), shape=(m, m))
        cfg.W0 = (cfg.W0 + extra).tocsr().astype(np.float32)
        cfg.W0.sort_indices()
        rows = np.repeat(np.arange(m), np.diff(cfg.W0.indptr))
        uniq, pair = np.unique(cfg.type_of[cfg.W0.indices].astype(np.int64) * 16 + cfg.type_of[rows], return_inverse=True)
        cfg.pair_id, cfg.gain0 = pair.astype(np.int32), np.ones(len(uniq), np.float32)
    rng = np.random.default_rng(batch)
    v0, ad0, pr, spk = ((rng.standard_normal((m, batch)) * s).astype(np.float32) for s in (0.25, 0.02, 0.2, 0.05))
    w = rng.standard_normal(m) / np.sqrt(m)
    gains = cfg.gain0 * rng.uniform(0.8, 1.2, len(cfg.gain0))
    tau = cfg.tau_of_type * rng.uniform(0.9, 1.1, cfg.n_types)
    return cfg, v0, ad0, pr, spk, w, gains.astype(np.float64), tau.astype(np.float64), steps


def check(prob, launch):
    (g64, t64, L64), _ = fp64(*prob)
    g32, t32, L32 = gpu_grads(*prob, checkpoint=20, launch=launch)
    # the tolerances of the adjoint's FP64 check: FP32 sums of ~10^4 terms, relative to the gradient's norm
    assert abs(L32 - L64) <= 1e-5 * max(1.0, abs(L64))
    assert np.linalg.norm(g32 - g64) <= 1e-4 * np.linalg.norm(g64)
    assert np.linalg.norm(t32 - t64) <= 1e-4 * np.linalg.norm(t64)


@pytest.mark.parametrize("batch", [3, 4, 5, 6, 8, 10, 12, 17, 20, 33, 34, 40, 63, 64, 66, 100, 130, 255, 256])
def test_every_batch_shape_matches_fp64(batch):
    check(problem(batch), "persistent")


@pytest.mark.parametrize("launch", ["step", "persistent"])
@pytest.mark.parametrize("batch", [1, 2, 4, 8])
def test_rows_sharing_a_warp_and_wide_rows_match_fp64(batch, launch):
    check(problem(batch, m=9473, nnz=60_000, hubs=1500, steps=22), launch)
