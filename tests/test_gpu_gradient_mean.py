"""The gradient term with a weight far above rho: the maps' means, whose d is rho,
are nearly all of the solution (the other frequencies' part is below 1 % of it,
and off by some 1e-4 of itself at most, d being held in 32 bits), so X's relative
error is that of the column pass's response to a constant.  It is exact but for a few roundings
of the pass and of the recursion, a few 1e-7 and at most 4e-6 in a 32-bit
emulation of columns of 64 to 2048 rows: bound 2e-5 (a gain not of the rounded
ratio is off by 1e-4 and more)."""

import numpy as np
import pytest

import sporco_cuda.cbpdn as cb
from oracle import cbpdn_oracle as O


@pytest.mark.gpu
@pytest.mark.parametrize("H,W", [(64, 64), (75, 33), (512, 36), (2048, 20)])
@pytest.mark.parametrize("mu", [1e7, 1e8, 1e9])
def test_weight_far_above_rho(H, W, mu):
    rng = np.random.default_rng(H)
    D = rng.standard_normal((6, 5, 4)).astype(np.float32)
    D += np.float32(0.5)  # (filters with a mean)
    S = (3.0 + rng.standard_normal((H, W))).astype(np.float32)
    opt = {"MaxMainIter": 8, "RelStopTol": 0.0, "AutoRho": {"Enabled": False}}
    ref = O.cbpdngrd(D, S, 0.01, mu, opt)
    X = cb.cbpdngrd(D, S, 0.01, mu, opt)
    err = np.linalg.norm(X.astype(np.float64) - ref) / np.linalg.norm(ref)
    assert err < 2e-5, err
