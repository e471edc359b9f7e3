"""The convolution column pass's variants that the autotuner chooses between: 8 or 16
rows per thread at 512, 768 and 1024 rows, and the cluster size.  Rows per thread
change only how a column is split over threads: at one cluster size every output
sums maps and taps in the same order, so plain and masked solves agree bit for bit;
the gradient term's recursion is cut into other blocks.  Every variant against the
FP64 oracle with the parity bound of the coefficient maps (1e-4 relative)."""

import numpy as np
import pytest

import sporco_cuda.cbpdn as cb
from oracle import cbpdn_oracle as O

OPT = {"MaxMainIter": 6, "RelStopTol": 0.0, "AutoRho": {"Enabled": False}}


@pytest.mark.gpu
@pytest.mark.parametrize("H", [512, 768, 1024])
@pytest.mark.parametrize("K", [7, 12, 16])
@pytest.mark.parametrize("solver", ["cbpdn", "cbpdnmsk", "cbpdngrd", "cbpdngrdmsk"])
def test_rows_per_thread_and_cluster(H, K, solver, monkeypatch):
    rng = np.random.default_rng(H + K)
    M, W = 9, 44
    D = rng.standard_normal((K, K, M))
    D = (D / np.sqrt(np.sum(D * D, axis=(0, 1), keepdims=True))).astype(np.float32)
    S = rng.standard_normal((H, W)).astype(np.float32)
    mask = (rng.random((H, W)) < 0.6).astype(np.float32)
    args = (D, S * mask, mask, 0.1) if "msk" in solver else (D, S, 0.1)
    if "grd" in solver:
        args += (0.2,)
    ref = getattr(O, solver)(*args, OPT)
    for G in (1, 2, 3, 8):
        monkeypatch.setenv("SPORCO_B200_COL_CLUSTER", str(G))
        X = {}
        for rows in (8, 16):
            monkeypatch.setenv("SPORCO_B200_COL_RADIX", str(rows))
            X[rows] = getattr(cb, solver)(*args, OPT)
            err = np.linalg.norm(X[rows].astype(np.float64) - ref) / np.linalg.norm(ref)
            assert err < 1e-4, (G, rows, err)
        if "grd" not in solver:
            assert np.array_equal(X[8], X[16]), G
