"""What the column-pass autotuner remembers a measurement for: a gradient solve
and a masked gradient solve of the same image size and number of maps share one
kernel, but the second has a map of its own (one more tile of shared memory, two
more transforms), so each is measured; a third solve of either shape is not.  And what
it tries: clusters of two CTAs and more, since a lone CTA sums all maps in one
32-bit chain (1024 x 1024, 256 maps: error of X 6.9e-7 instead of 5.8e-7)."""

import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import sys
import numpy as np
sys.path[:0] = [{root!r}, {pkg!r}]
import sporco_cuda.cbpdn as cb
rng = np.random.default_rng(0)
D = rng.standard_normal((8, 8, 12)).astype(np.float32)
S = rng.standard_normal((64, 48)).astype(np.float32)
m = np.ones_like(S)
opt = {{"MaxMainIter": 2, "RelStopTol": 0.0}}
solves = {{"one": lambda: cb.cbpdngrd(D, S, 0.1, 0.2, opt),
          "own": lambda: cb.cbpdngrdmsk(D[..., 1:], S, m, 0.1, 0.2, opt)}}
for k in {order!r}:
    solves[k]()
"""


@pytest.mark.gpu
@pytest.mark.parametrize("order", [("one", "own", "one", "own"), ("own", "one")])
def test_map_of_its_own_is_measured_for_itself(order):
    code = CHILD.format(root=ROOT, pkg=os.path.join(ROOT, "sporco-cuda_b200"), order=order)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, SPORCO_B200_AUTOTUNE="verbose"))
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stderr.count("autotune: column pass 64x48 M=12:") == 2, r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("H,M", [(64, 12), (100, 5), (1024, 4)])
def test_no_lone_cta_is_tried(H, M):
    code = CHILD.format(root=ROOT, pkg=os.path.join(ROOT, "sporco-cuda_b200"), order=())
    code += f"""
D, S = D[..., :{M}], rng.standard_normal(({H}, 40)).astype(np.float32)
cb.cbpdn(D, S, 0.1, opt)
cb.cbpdngrd(D, S, 0.1, 0.2, opt)
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, SPORCO_B200_AUTOTUNE="verbose"))
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stderr.count(f"autotune: column pass {H}x40 M={M}:") == 2, r.stderr
    assert "/G=2 " in r.stderr and "/G=1 " not in r.stderr, r.stderr
