"""The training GEMMs' tile choices: one SGD step at row counts at the edges of
their tiles (64 and 32 rows of a tile, 64 rows of a weight-gradient stage, the
smallest batch and the sizes where the tile changes) equals the FP64 network's.

Bars: the step is w - lr g in FP32, so a weight's own rounding (2^-24 of at most 0.5)
is an absolute error of 3e-8 in g; the gradient's FP32 chains of n terms err by
about sqrt(n) 2^-24 of their terms' size, far below 2e-3 of the layer's largest."""
import numpy as np
import pytest

import tempestrenderer_b200 as svf
import test_gpu_mlp as mlp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 31, 33, 63, 64, 65, 449, 2303, 2369, 4097])
def test_sgd_step_matches_fp64_gradient(gpu_ctx, rows):
    lp = svf.directions_fibonacci(16)
    *stats, w = mlp._random_model(lp, 3)
    rng = np.random.default_rng(rows)
    X = rng.standard_normal((rows, mlp.INPUTS)).astype(np.float32)
    T = rng.standard_normal((rows, mlp.OUTPUTS)).astype(np.float32)
    loss64, g64 = mlp._loss_grad(w, X, T)
    m = svf.Mlp.load(gpu_ctx, mlp._blob(lp, *stats, w))
    assert m.step(X, T, lr=1.0, sgd=True) == pytest.approx(loss64, rel=1e-4)
    g = w.astype(np.float64) - mlp._weights_of(m.save())
    for a, b in ((mlp.W1, mlp.B1), (mlp.B1, mlp.W2), (mlp.W2, mlp.B2), (mlp.B2, mlp.W3), (mlp.W3, mlp.B3),
                 (mlp.B3, mlp.NPARAMS)):
        assert np.abs(g[a:b] - g64[a:b]).max() < 2e-3 * np.abs(g64[a:b]).max() + 6e-8, (a, b)
    m.close()
