"""Warm solves that reuse the spectra of D and S (run(warm="same")) and need
something of the dictionary that the solve before them did not: its 2-D spectrum
for the statistics or for another column solve, and the sums over the maps for
another class of gradient weights.  Against the same continuation with D and S
transformed again (run(warm=True)): the same arithmetic but for the order of the
double-precision sums of Psum, so to float32 rounding (1e-5 relative; the wrong
sums are off by parts of one)."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import sporco_cuda.cbpdn as cb

OPT = {"MaxMainIter": 6, "RelStopTol": 0.0, "AutoRho": {"Enabled": True, "Period": 2}}


def _prepare(H, W, K, gw=None, record=False, M=36):
    g = torch.Generator(device="cuda").manual_seed(H + K)
    D = torch.randn((M, K, K), generator=g, device="cuda")
    S = torch.randn((1, H, W), generator=g, device="cuda")
    kw = {} if gw is None else dict(grd=True, mu=0.5, gw=np.asarray(gw, np.float32))
    return cb.prepare_device(D, S, 0.05, OPT, record_itstat=record, **kw)


def _close(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    assert np.all(np.isfinite(a)) and np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b)


@pytest.mark.gpu
@pytest.mark.parametrize("H,W", [(16, 20), (64, 48), (75, 33), (512, 40)])
@pytest.mark.parametrize("K", [5, 16])
def test_statistics_switched_on(H, W, K):
    """Also on, off and on again: the 2-D spectrum stays."""
    stats = []
    for warm in ("same", True):
        ds = _prepare(H, W, K, record=True)
        ds.opts.record_itstat = 0
        ds.run()
        ds.opts.record_itstat = 1
        ds.run(warm=warm)
        first = ds.state()["itstat"]
        ds.opts.record_itstat = 0
        ds.run(warm=warm)
        ds.opts.record_itstat = 1
        Y = ds.run(warm=warm).clone()
        stats.append((first, ds.state()["itstat"], Y.cpu().numpy()))
    for a, b in zip(*stats):
        _close(a, b)


M = 36
ONE, SPLIT, OWN = [2] * M, [0] + [2] * (M - 1), [1, 2, 0] + [3] * (M - 3)


@pytest.mark.gpu
@pytest.mark.parametrize("H,W", [(64, 48), (75, 33)])
@pytest.mark.parametrize("first,then", [(ONE, SPLIT), (SPLIT, ONE), (ONE, OWN), (OWN, ONE),
                                        (OWN, SPLIT), (SPLIT, OWN)])
def test_sums_of_another_weight_class(H, W, first, then):
    """The weights' class changes with no iteration in between (F is zero then, in
    any layout)."""
    out = []
    for warm in ("same", True):
        ds = _prepare(H, W, 6, first)
        ds.run(iters=0)
        ds.keep["gw"].copy_(torch.tensor(then, dtype=torch.float32))
        ds.prob.wgrd_uniform = cb._weight_class(then, M)
        out.append(ds.run(warm=warm).cpu().numpy())
    ref = _prepare(H, W, 6, then).run().cpu().numpy()
    _close(out[0], out[1])
    _close(out[0], ref)


@pytest.mark.gpu
@pytest.mark.parametrize("H,W", [(64, 64), (64, 33), (64, 48), (75, 33)])
@pytest.mark.parametrize("warm", ["same", True])
@pytest.mark.parametrize("given", [False, True])
def test_column_pass_of_another_layout(H, W, warm, given):
    """The same problem with another class named for its (equal) weights: the
    other column pass wants the row spectra of Y - U in another layout.  Against
    the continuation that keeps the class.  given: from given iterates (Y and U
    kept apart).  Period 2 changes rho after the sixth iteration, not the fifth."""
    for first in (5, 6):
        out = []
        for classes in ((2, 2, 2), (2, 0, 2)):
            ds = _prepare(H, W, 6, ONE)
            if given:
                u0 = torch.full_like(ds.keep["Y"], 0.01)
                ds.keep["Y"].fill_(0.02)
                ds.prob.U0 = u0.data_ptr()
            for n, c in enumerate(classes):
                ds.prob.wgrd_uniform = c
                Y = ds.run(warm=warm if n else False, iters=(first, 2, 3)[n])
            out.append(Y.cpu().numpy())
        _close(out[1], out[0])
