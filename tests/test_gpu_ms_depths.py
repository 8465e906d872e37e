"""The pseudo-volume model at the depths around the end of the table of draws (7 events
at 256 walks): the fit's evaluator against the oracle's, and the renderer's shared walks,
whose lost pairs go on in other blocks from 6 events on, against every pair's own."""
import numpy as np
import pytest

import oracle
import tempestrenderer_b200 as svf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth", [6, 7, 8, 9, 17])
def test_evaluator_against_the_oracle(gpu_ctx, depth):
    """The RMSE of a zero-iteration fit against the oracle's values is the evaluation
    difference; the bar of the other depths (2e-3 of the values' RMS).  Albedos above
    and below 1: walks that go on to the depth and walks that die before it."""
    lp = svf.directions_fibonacci(16)
    p = np.array([[0.3, 0.2, 1.3, 0.1, 0.1, -0.2, 0.4], [0.1, 0.4, 0.2, 0.3, 0.3, 0.2, -0.5],
                  [0.5, 0.5, 0.02, 0.2, 0.0, 0.1, 0.0]], np.float32)
    ref = np.stack([oracle.brdf_all_ms(q.astype(np.float64), lp, depth) for q in p]).astype(np.float32)
    _, rmse, _ = gpu_ctx.lsq_fit_batch(lp, ref, p, svf.options(max_iterations=0, multi_scattering=depth))
    assert (rmse <= 2e-3 * np.sqrt(np.mean(ref.astype(np.float64) ** 2, axis=1))).all(), rmse


@pytest.mark.parametrize("depth", [4, 5, 6, 7])
def test_shared_walks_equal_own_walks_anywhere(gpu_ctx, depth):
    """Orientations all over the sphere: most pairs lose sight of an event.  A call of 160
    texels shares the views' walks, calls of 40 do not (at most 1024 pairs an SM)."""
    lp = svf.directions_fibonacci(32)
    rng = np.random.default_rng(depth)
    q = rng.standard_normal((160, 4)).astype(np.float32)
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    maps = (rng.random((160, 3)).astype(np.float32), (0.5 + rng.random((160, 3))).astype(np.float32),
            (0.02 * 40.0 ** rng.random((160, 2))).astype(np.float32), q)
    got = gpu_ctx.render_btf_ms(lp, *maps, depth)
    own = np.concatenate([gpu_ctx.render_btf_ms(lp, *(m[t:t + 40] for m in maps), depth) for t in range(0, 160, 40)])
    np.testing.assert_array_equal(got.view(np.uint32), own.view(np.uint32))
