"""The gradient term with a map of its own (a zero weight for map 0) at the longest
compiled columns, where the convolution pass's fourth tile does not fit (2048
rows) or just does (1536).  Against the FP64 oracle with the parity bound of the
coefficient maps (1e-4 relative)."""

import numpy as np
import pytest

import sporco_cuda.cbpdn as cb
from oracle import cbpdn_oracle as O


@pytest.mark.gpu
@pytest.mark.parametrize("H", [1024, 1536, 2048])
@pytest.mark.parametrize("K", [5, 12, 16])
def test_map_of_its_own_at_long_columns(H, K):
    rng = np.random.default_rng(H + K)
    M, W = 3, 36
    D = rng.standard_normal((K, K, M))
    D = (D / np.sqrt(np.sum(D * D, axis=(0, 1), keepdims=True))).astype(np.float32)
    S = rng.standard_normal((H, W)).astype(np.float32)
    mask = (rng.random((H, W)) < 0.6).astype(np.float32)
    opt = {"MaxMainIter": 8, "RelStopTol": 0.0, "AutoRho": {"Enabled": True}}
    own = dict(opt, GradWeight=np.array([0, 2, 2], dtype=np.float32))
    for X, ref in (
            (cb.cbpdngrdmsk(D, S * mask, mask, 0.1, 0.2, opt),
             O.cbpdngrdmsk(D, S * mask, mask, 0.1, 0.2, opt)),
            (cb.cbpdngrd(D, S, 0.1, 0.2, own), O.cbpdngrd(D, S, 0.1, 0.2, own))):
        err = np.linalg.norm(X.astype(np.float64) - ref) / np.linalg.norm(ref)
        assert err < 1e-4, err


def test_every_other_length_fits():
    """conv_fits from the header's own formulas (no GPU): only 2048 rows with a
    map of its own is past 227 KB."""
    def smem(H, L, KR, NT, two, grad=True):
        slots = H if L % 2 else H + H // L
        tile = max(4 * slots, KR * 8) * 8
        return 3 * tile + 3 * KR * 64 + (NT * (4 * 16 + (16 if L % 2 else 8)) if grad else 0) + (tile if two else 0)

    rows = {16: 4, 32: 4, 48: 6, 64: 4, 96: 4, 128: 4, 192: 8, 256: 8, 384: 8, 512: 8, 768: 8,
            1024: 8, 1536: 16, 2048: 16}
    for KR in (8, 12, 16):
        for H, L in rows.items():
            for two in (False, True):
                assert (smem(H, L, KR, 2 * H // L, two) <= 227 * 1024) == (not (two and H == 2048))
        assert smem(1024, 9, KR, 256, True) <= 227 * 1024  # the longest without a compiled plan
