"""The convolution column pass's one transform pair per tile of four columns: its
errors are in every map at once, where a transform per map averages them.  X after
two iterations, at the column lengths with the longest transforms, against the
FP64 oracle, mean over three problems at one cluster size: no larger than with the
column pass before it, which took the sums over the maps in the same way but formed
its twiddles' powers and Psum together from one transform of the filters (3.457e-7
and 3.770e-7 at 1024 rows, 3.386e-7 and 3.755e-7 at 2048, plain and masked; with
the powers as products and Psum from the lags 3.489e-7 and 3.861e-7, 3.419e-7 and
3.853e-7)."""

import numpy as np
import pytest

import sporco_cuda.cbpdn as cb
from oracle import cbpdn_oracle as O


def _problem(H, W, M, K, seed):
    rng = np.random.default_rng(seed)
    D = rng.standard_normal((K, K, M))
    D = (D / np.sqrt(np.sum(D * D, axis=(0, 1), keepdims=True))).astype(np.float32)
    x = rng.standard_normal((H, W, M)) * (rng.random((H, W, M)) < .01)
    Df = np.fft.rfft2(D, s=(H, W), axes=(0, 1))
    S = np.fft.irfft2(np.sum(Df * np.fft.rfft2(x, axes=(0, 1)), axis=2), s=(H, W))
    S = (S + .01 * rng.standard_normal((H, W))).astype(np.float32)
    return D, S, (rng.random((H, W)) < .7).astype(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("H,M,plain,masked", [(1024, 64, 3.457e-7, 3.770e-7),
                                              (2048, 48, 3.386e-7, 3.755e-7)])
def test_error_of_long_columns(H, M, plain, masked, monkeypatch):
    monkeypatch.setenv("SPORCO_B200_COL_CLUSTER", "4")
    opt = {"MaxMainIter": 2, "RelStopTol": 0.0, "RelaxParam": 1.8, "AutoRho": {"Enabled": False}}
    err = np.zeros((3, 2))
    for seed in (1, 2, 3):
        D, S, mask = _problem(H, 64, M, 16, seed)
        for i, (X, R) in enumerate((
                (cb.cbpdn(D, S, .05, opt), O.cbpdn(D, S, .05, opt)),
                (cb.cbpdnmsk(D, S * mask, mask, .05, opt),
                 O.cbpdnmsk(D, S * mask, mask, .05, opt)))):
            err[seed - 1, i] = np.linalg.norm(X.astype(np.float64) - R) / np.linalg.norm(R)
    m = err.mean(axis=0)
    assert m[0] <= plain and m[1] <= masked, m
