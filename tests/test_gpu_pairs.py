"""The pair kernels of the renderer and the pair-wise error (svf_error.cu) over the
layouts they can go wrong at: an odd and an even number of views (the views go by in
twos), one to many groups of lights to a block, outputs at any offset.

Against the oracle's FP64 BRDF.  The renderer's bound is that of the rendered BTF at
Fresnel 1.5: 1e-5 of the texel's RMS.  The error maps' residuals are 30 % of the BRDF, so a BRDF
within 1e-5 moves an RMSE by less than 1e-4 of it, and a PSNR by 20 log10(1 + 1e-4) =
8.7e-4 dB."""
import numpy as np
import pytest

import tempestrenderer_b200 as svf

pytestmark = pytest.mark.gpu

T = 5


def _case(oracle, L):
    rng = np.random.default_rng(L)
    tp = np.stack([np.sort(np.radians(75.0) * np.sqrt(rng.random(L))), 2 * np.pi * rng.random(L)], 1)
    tp = tp.astype(np.float32)
    lp = oracle.angles_to_parabolic(tp)
    truths = [oracle.synth_truth(L, 1, x) for x in range(T)]
    maps = [np.array([getattr(t, k)[:] for t in truths], np.float32) for k in ("kd", "ks", "sigma", "quat")]
    f = np.empty((T, L * L, 3))
    for x, t in enumerate(truths):
        for c in range(3):
            p = np.array([maps[2][x, 0], maps[2][x, 1], maps[1][x, c], maps[0][x, c], *t.euler[:]])
            f[x, :, c] = oracle.brdf_all(p, lp, 1.0)[1]
    return tp, lp, maps, f


@pytest.mark.parametrize("L", [3, 4, 7, 33, 81, 129, 160])
def test_pair_kernels(gpu_ctx, oracle_lib, L):
    import torch

    tp, lp, maps, f = _case(oracle_lib, L)
    out = gpu_ctx.render_btf(lp, *maps)
    rms = np.sqrt((f ** 2).mean(axis=(1, 2)))
    assert np.all(np.sqrt(((out - f) ** 2).mean(axis=(1, 2))) < 1e-5 * rms)
    # halves, and device memory that begins 1 to 3 values past 16 bytes
    for typ, dt in ((svf.SVF_SAMPLES_F32, torch.float32), (svf.SVF_SAMPLES_F16, torch.float16)):
        want = torch.from_numpy(out).to(dt)
        for off in range(4):
            buf = torch.full((T * L * L * 3 + 8,), -1.0, dtype=dt, device="cuda")
            gpu_ctx.render_btf(lp, *maps, sample_type=typ, out=buf[off:off + T * L * L * 3].view(T, L * L, 3))
            got = buf.cpu()
            assert torch.equal(got[off:off + T * L * L * 3].view(T, L * L, 3), want)
            assert (got[:off] == -1).all() and (got[off + T * L * L * 3:] == -1).all()
    # a file whose samples are the BRDF with 30 % noise: U the samples, SxV the identity
    rng = np.random.default_rng(1)
    v = (f * (1 + 0.3 * rng.standard_normal(f.shape))).astype(np.float32)
    planes = [(v[:, :, c].T.copy(), np.eye(T, dtype=np.float32)) for c in range(3)]
    b = svf.Btf(gpu_ctx, oracle_lib.btf_file_bytes(tp, T, 1, planes, data_size=4))
    w = np.array([0.2126, 0.7152, 0.0722])
    for color in (False, True):
        res = v.astype(np.float64) - f
        val = v.astype(np.float64)
        if not color:
            res, val = (res @ w)[..., None], (val @ w)[..., None]
        ref = np.sqrt((res ** 2).mean(axis=1))
        rmse, psnr = b.error_maps(*(m[None] for m in maps), color=color)
        np.testing.assert_allclose(np.reshape(rmse, ref.shape), ref, rtol=1e-4)
        np.testing.assert_allclose(np.reshape(psnr, ref.shape), 20 * np.log10(val.max(axis=1) / ref), atol=8.7e-4)
    b.close()
