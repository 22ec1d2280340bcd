"""Gradients of the network at the row counts where the slices of the weight and
bias sums change (csrc/mlp.cu: slices of 128 rows, of 256 and more from 16385
rows on, the last one partial), and predictions over a part of the upload, whole
parts and a remainder, against the CPU restatement with BF16 rounding at the
same points.  Bounds: those of the network's other gradient and inference tests
(BF16's 2^-8 through two hidden layers)."""
import numpy as np
import pytest

from oracle import mlp_oracle as M
from test_gpu_warmstart import GRAD_TOL, _batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 2, 127, 128, 129, 256, 300, 16384, 16385, 33000])
def test_gradient_by_slices(pdgb, rows):
    p = pdgb.mlp_init(4)
    p[-3:] = [0.05, -0.02, 0.01]
    X, T = _batch(rows, rows)
    loss, g = pdgb.mlp_loss_grad(X, T, p)
    lo, go = M.loss_grad(X, T, p)
    assert abs(loss - lo) / lo < 2e-2
    at = 0
    for a, b in ((64, 128), (128, 128), (128, 3)):
        for size in (a * b, b):
            err = np.linalg.norm(g[at:at + size] - go[at:at + size]) / max(np.linalg.norm(go[at:at + size]), 1e-30)
            assert err < GRAD_TOL, (rows, at, err)
            at += size


@pytest.mark.parametrize("rows", [131071, 131072, 131073, 300000])
def test_prediction_by_parts(pdgb, rows):
    p = pdgb.mlp_init(9)
    X, _ = _batch(rows, 3)
    Y = pdgb.mlp_predict(X, p)
    at = np.r_[0:300, rows // 2:rows // 2 + 300, rows - 300:rows, 130900:min(rows, 131300)]
    Yo, _ = M.forward(X[at], p)
    assert Y.shape == (rows, 3) and np.isfinite(Y).all()
    assert np.linalg.norm(Y[at] - Yo) / np.linalg.norm(Yo) < 2e-2
