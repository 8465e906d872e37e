"""The pooled LM kernel (RGB fits, and luminance fits summed in 7 shares): which
warp computes a share, how many slots and warps a launch has and which texels
share an SM must not show in a texel's result.

* A batch's texels equal, bit for bit, their fits one by one: layouts at both ends
  of the ranges that take 7 shares (even and odd direction counts, one to seven
  slots an SM), texel counts of one slot, of one more than the SMs and of several
  rounds of the counter.
* The residual at given parameters equals the oracle's evaluator's to 1e-4
  relative (the bar of the other pair passes: FP32 terms, FP64 sums).
"""
import numpy as np
import pytest

import tempestrenderer_b200 as svf

pytestmark = pytest.mark.gpu


def _samples(ctx, lp, T, seed):
    import torch

    s = torch.empty((T, lp.shape[0] ** 2, 3), dtype=torch.float32, device="cuda")
    ctx.synth_btf(seed, 1, lp, 0, T, s)
    torch.cuda.synchronize()
    return s


@pytest.mark.parametrize("L,rgb,T", [(90, False, 149), (111, False, 40), (113, False, 450), (130, False, 3),
                                     (132, False, 149), (151, False, 310), (160, False, 5), (16, True, 600),
                                     (49, True, 149), (62, True, 40), (81, True, 320), (134, True, 149),
                                     (160, True, 3)])
def test_batch_equals_single_texels(gpu_ctx, L, rgb, T):
    lp = svf.directions_ring81() if L == 81 else svf.directions_fibonacci(L)
    s = _samples(gpu_ctx, lp, T, 7000 + L)
    lay = svf.Layout(lp)
    opts = svf.options(max_iterations=60, rgb=rgb)
    want = ("params", "rmse", "stats", "init")
    got, _ = gpu_ctx.fit_texels(lay, s, T, 1, opts=opts, want=want, check=False)
    for t in sorted({0, 1, T // 2, T - 1}):
        one, _ = gpu_ctx.fit_texels(lay, s[t:t + 1], 1, 1, opts=opts, want=want, check=False)
        for k in want:
            assert one[k][0].tobytes() == got[k][t].tobytes(), (t, k, one[k][0], got[k][t])


@pytest.mark.parametrize("L", [90, 132, 160])
def test_residual_against_the_oracle(gpu_ctx, oracle_lib, L):
    lp = svf.directions_fibonacci(L)
    rng = np.random.default_rng(L)
    lum = rng.random((2, L * L)).astype(np.float32)
    p = np.array([[0.21, 0.4, 0.6, 0.3, 0.1, -0.2, 0.4], [0.7, 0.08, 0.3, 0.0, -0.3, 0.2, 1.1]], np.float32)
    _, rmse, _ = gpu_ctx.lsq_fit_batch(lp, lum, p, svf.options(max_iterations=0))
    for t in range(2):
        f32, _ = oracle_lib.brdf_all(p[t].astype(np.float64), lp)
        np.testing.assert_allclose(rmse[t], np.sqrt(np.mean((lum[t].astype(np.float64) - f32) ** 2)), rtol=1e-4)
