"""The row pass's two forms of the iteration, packed (rows whose threshold has one
weight) and scalar (rows with a weight per element), do the same arithmetic: with
weights of one given either way a solve's maps agree bit for bit (rho fixed, as the
residual sums are in another order).  At the widths of every row kernel, with and
without the correction form (a mask writes whole row spectra)."""

import numpy as np
import pytest

import sporco_cuda.cbpdn as cb


@pytest.mark.gpu
@pytest.mark.parametrize("W", [64, 96, 128, 256, 512, 1024, 1536, 2048, 33, 75, 320])
@pytest.mark.parametrize("relax", [1.8, 1.0])
def test_weights_given_either_way(W, relax):
    rng = np.random.default_rng(W)
    H, M, K = 64, 4, 7
    D = rng.standard_normal((K, K, M))
    D = (D / np.sqrt(np.sum(D * D, axis=(0, 1), keepdims=True))).astype(np.float32)
    S = rng.standard_normal((H, W)).astype(np.float32)
    mask = (rng.random((H, W)) < 0.6).astype(np.float32)
    opt = {"MaxMainIter": 12, "RelStopTol": 0.0, "RelaxParam": relax, "AutoRho": {"Enabled": False}}
    full = dict(opt, L1Weight=np.ones((H, W, M), dtype=np.float32))
    X = cb.cbpdn(D, S, 0.05, opt)
    assert np.count_nonzero(X) > 100
    assert np.array_equal(X, cb.cbpdn(D, S, 0.05, full))
    assert np.array_equal(cb.cbpdnmsk(D, S * mask, mask, 0.05, opt),
                          cb.cbpdnmsk(D, S * mask, mask, 0.05, full))
