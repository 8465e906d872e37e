"""The pooled LM kernel's bounded waits, made to run out on purpose (RGB fits and
luminance fits summed in 7 shares; tests/test_gpu_timeout.py has the other kernel's).

The library's fault injection, read from the environment at each launch, leaves
one texel's slab copy unissued (SVF_FAULT_SKIP_SLAB_COPY: the wait of the warp
that starts the texel runs out) or that texel's passes unopened
(SVF_FAULT_HOLD_PASS: the wait of the warps that find nothing to do runs out).  The
call must return SVF_ETIMEOUT, the texel's status must carry SVF_TEXEL_TIMEOUT, every
other texel must be fitted as without the fault, and the context must stay usable.
No GPU fault is involved: the waits are counted, on a barrier that nothing completes
and on a word that nothing sets.

The texel counts give one texel an SM (a slot each), several slots an SM, and
several rounds of the slots; the texel at fault is dealt at the start or taken later.
"""
import numpy as np
import pytest

import tempestrenderer_b200 as svf

pytestmark = pytest.mark.gpu

SKIP, HOLD = "SVF_FAULT_SKIP_SLAB_COPY", "SVF_FAULT_HOLD_PASS"


def _fit(ctx, lp, s, rgb):
    T = s.shape[0]
    opts = svf.options(max_iterations=30, rgb=rgb)
    if rgb:
        out = {k: np.full((T, n), np.nan, np.float32) for k, n in (("params", 12), ("rmse", 1))}
        init = np.tile(np.array([.2, .2, .2, .5, .5, .5, .3, .3, 0, 0, 0, 1], np.float32), (T, 1))
        call = lambda: ctx.fit_texels(svf.Layout(lp), s, T, 1, opts=opts, init=init, want=("params", "rmse"),
                                      out=out)
        return out["params"], out["rmse"], None, call
    lum = (s @ s.new_tensor([0.2126, 0.7152, 0.0722])).cpu().numpy()
    init = np.tile(np.array([.3, .3, .4, .2, .1, -.1, .1], np.float32), (T, 1))
    out, rmse = np.full((T, 7), np.nan, np.float32), np.full(T, np.nan, np.float32)
    stats = np.zeros(T, svf.STATS_DTYPE)
    return out, rmse, stats, lambda: ctx.lsq_fit_batch(lp, lum, init, opts, out=out, rmse=rmse, stats=stats)


@pytest.mark.parametrize("fault", [SKIP, HOLD])
@pytest.mark.parametrize("L,rgb,T,texel", [(151, False, 1, 0), (151, False, 140, 3), (113, False, 700, 2),
                                           (113, False, 700, 690), (81, True, 60, 59), (62, True, 400, 300)])
def test_expired_wait_reports_timeout(oracle_lib, L, rgb, T, texel, fault, monkeypatch):
    import torch

    lp = svf.directions_ring81() if L == 81 else svf.directions_fibonacci(L)
    s = torch.empty((T, L * L, 3), dtype=torch.float32, device="cuda")
    with svf.Context(0) as ctx:
        ctx.synth_btf(900 + L, 1, lp, 0, T, s)
        torch.cuda.synchronize()
        ref_out, ref_rmse, ref_stats, call = _fit(ctx, lp, s, rgb)
        call()
    with svf.Context(0) as ctx:   # (of its own: no recorded launch)
        out, rmse, stats, call = _fit(ctx, lp, s, rgb)
        monkeypatch.setenv(fault, str(texel))
        monkeypatch.setenv("SVF_FAULT_WAIT_SPINS", "4096")
        with pytest.raises(svf.SvfError) as e:
            call()
        assert e.value.status == svf.SVF_ETIMEOUT, e.value
        others = np.arange(T) != texel
        assert np.array_equal(out[others], ref_out[others])
        assert np.array_equal(rmse[others], ref_rmse[others])
        if stats is not None:
            assert np.array_equal(stats["status"] & svf.SVF_TEXEL_TIMEOUT != 0, ~others)
        monkeypatch.delenv(fault)
        monkeypatch.delenv("SVF_FAULT_WAIT_SPINS")
        call()
        assert np.array_equal(out, ref_out) and np.array_equal(rmse, ref_rmse)
        if stats is not None:
            assert np.array_equal(stats, ref_stats)
