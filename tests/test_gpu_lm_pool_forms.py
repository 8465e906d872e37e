"""The forms of the pooled LM kernel that the other tests do not run: luminance fits with
a Fresnel factor, layouts with directions below the horizon, the batch call whose BTFs'
layouts differ within a launch, and the call without allocations.

* The residual at given parameters equals the oracle's evaluator's to 1e-4 relative
  (the bar of every pair pass).
* One LM step equals the one that the other kernel makes of the same sums in 4 parts
  (SVF_LM_KERNEL pins it): J^T J and J^T r are FP32 sums of at most 60 terms a lane, so
  their entries differ by about 60 x 6e-8 of the sum of their terms' magnitudes; the step
  solves with J^T J + 0.75 max(J^T J), whose condition is below 3.  The bar, 1e-3 of the
  step, leaves a factor for cancellation in J^T r; a term in the wrong sum moves the step
  by its own size.
* The batch and the call without allocations equal single calls bit for bit.
"""
import ctypes as C

import numpy as np
import pytest

import tempestrenderer_b200 as svf

pytestmark = pytest.mark.gpu


def _layout(L, low):
    lp = svf.directions_fibonacci(L).copy()
    if low:
        lp[[3, 17, L // 2, L - 1]] = [[1.0, 0.02], [0.0, 1.05], [0.7, -0.8], [-0.8, -0.8]]
    return lp


@pytest.mark.parametrize("fresnel", [1.0, 1.5])
@pytest.mark.parametrize("low", [False, True])
@pytest.mark.parametrize("L", [113, 134])
def test_residual_and_step(gpu_ctx, oracle_lib, monkeypatch, L, low, fresnel):
    lp = _layout(L, low)
    rng = np.random.default_rng(L)
    p = np.array([[0.21, 0.4, 0.6, 0.3, 0.1, -0.2, 0.4], [0.7, 0.3, 0.3, 0.1, -0.3, 0.2, 1.1],
                  [0.1, 0.5, 1.2, 0.4, 0.2, 0.1, -0.7]], np.float32)
    model = np.stack([oracle_lib.brdf_all(q.astype(np.float64), lp, fresnel)[0] for q in p])
    lum = rng.random(model.shape).astype(np.float32)
    opts = svf.options(max_iterations=0, fresnel=fresnel)
    _, rmse, _ = gpu_ctx.lsq_fit_batch(lp, lum, p, opts)
    expect = np.sqrt(np.mean((lum.astype(np.float64) - model) ** 2, axis=1))
    np.testing.assert_allclose(rmse, expect, rtol=1e-4)

    start = (p * (1 + 0.1 * rng.random(p.shape))).astype(np.float32)
    one = svf.options(max_iterations=1, fresnel=fresnel, restarts=0)
    pooled, _, st = gpu_ctx.lsq_fit_batch(lp, model, start, one)
    monkeypatch.setenv("SVF_LM_KERNEL", "160,2,0")
    other, _, st2 = gpu_ctx.lsq_fit_batch(lp, model, start, one)
    assert (st["effective"] == 1).all() and (st2["effective"] == 1).all()
    step = np.abs(other - start).max(axis=1, keepdims=True)
    assert (step > 1e-4).all()
    assert (np.abs(pooled - other) <= 1e-3 * step).all(), np.abs(pooled - other) / step


def test_batch_of_layouts_in_one_launch(gpu_ctx):
    import torch

    btfs, opts = [], svf.options(max_iterations=40)
    for L, T in ((132, 30), (160, 9), (151, 200), (132, 1)):
        lp = svf.directions_fibonacci(L)
        s = torch.empty((T, L * L, 3), dtype=torch.float32, device="cuda")
        gpu_ctx.synth_btf(60 + L, 1, lp, 0, T, s)
        init = np.tile(np.array([0.3, 0.2, 0.5, 0.2, 0.1, -0.2, 0.3], np.float32), (T, 1))
        btfs.append(dict(layout=svf.Layout(lp), samples=s, width=T, height=1, init=init))
    torch.cuda.synchronize()
    maps, _, _ = gpu_ctx.fit_btfs(btfs, opts, want=("params", "rmse", "stats"))
    for b, m in zip(btfs, maps):
        one, _ = gpu_ctx.fit_texels(b["layout"], b["samples"], b["width"], 1, opts=opts, init=b["init"],
                                    want=("params", "rmse", "stats"))
        for k in one:
            assert m[k].tobytes() == one[k].tobytes(), (b["layout"].light_count, k)


@pytest.mark.parametrize("L,T", [(113, 41), (160, 20)])
def test_call_without_allocations(gpu_ctx, L, T):
    import torch

    assert T == svf.SVF_NOALLOC_MAX_SLAB_FLOATS // ((L * L + 7) // 8 * 8)   # the most the scratch holds
    lp = svf.directions_fibonacci(L)
    lum = np.random.default_rng(L).random((T, L * L)).astype(np.float32)
    init = np.tile(np.array([0.3, 0.2, 0.5, 0.2, 0.1, -0.2, 0.3], np.float32), (T, 1))
    opts = svf.options(max_iterations=40)
    out_ref, rmse_ref, _ = gpu_ctx.lsq_fit_batch(lp, lum, init, opts)
    d = [torch.from_numpy(x).cuda() for x in (lp, lum, init)]
    out, rmse = torch.full((T, 7), float("nan"), device="cuda"), torch.full((T,), float("nan"), device="cuda")
    lib = svf.load()
    assert lib.svf_lsq_fit_batch_noalloc(d[0].data_ptr(), L, d[1].data_ptr(), L * L, T, C.byref(opts), d[2].data_ptr(),
                                         out.data_ptr(), rmse.data_ptr(), None, None) == svf.SVF_OK, lib.svf_last_error()
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), out_ref) and np.array_equal(rmse.cpu().numpy(), rmse_ref)
