"""Calls on several threads, each with its own context, whose launches of one kernel
ask for different amounts of shared memory: the pooled LM kernel (one texel: one slot
an SM; 600: several), the other LM kernel and the luminance pass (layouts of different
slab sizes).  A kernel's shared-memory limit is the process's, so no launch may set it
below another's need."""
import ctypes as C
import threading

import pytest

import tempestrenderer_b200 as svf

pytestmark = pytest.mark.gpu


def _lsq(ctx, lib, L, T, keep):
    import torch

    lp = svf.directions_ring81() if L == 81 else svf.directions_fibonacci(L)
    lum = torch.rand((T, L * L), device="cuda")
    init = torch.tensor([[.3, .3, .4, .2, .1, -.1, .1]], device="cuda").repeat(T, 1)
    out, rmse = torch.empty((T, 7), device="cuda"), torch.empty(T, device="cuda")
    opts = svf.options(max_iterations=0)
    keep += [lp, lum, init, out, rmse, opts]
    args = (ctx.handle, lp.ctypes.data, L, lum.data_ptr(), L * L, T, C.byref(opts), init.data_ptr(), out.data_ptr(),
            rmse.data_ptr(), None)
    return lambda: lib.svf_lsq_fit_batch(*args)


def _fit(ctx, lib, L, T, keep):
    import torch

    lay = svf.Layout(svf.directions_fibonacci(L))
    init = torch.tensor([[.3, .3, .4, .2, .1, -.1, .1]], device="cuda").repeat(T, 1)
    v, fo, m = svf.BtfView(), svf.FitOptions(), svf.Maps()
    s = torch.rand((T, L * L, 3))   # (host samples: no call is recorded and replayed)
    out, rmse = torch.empty((T, 7)), torch.empty(T)
    keep += [lay, init, s, out, rmse]
    v.samples, v.sample_type, v.width, v.height, v.layout = s.data_ptr(), svf.SVF_SAMPLES_F32, T, 1, C.pointer(lay.desc)
    fo.lsq, fo.init_mode, fo.init_params = svf.options(max_iterations=0), svf.SVF_INIT_GIVEN, init.data_ptr()
    m.params, m.rmse = out.data_ptr(), rmse.data_ptr()
    keep += [v, fo, m]
    return lambda: lib.svf_fit_texels(ctx.handle, C.byref(v), C.byref(fo), C.byref(m), None)


@pytest.mark.parametrize("make,small,large", [(_lsq, (113, 1), (113, 600)), (_lsq, (78, 1), (81, 500)),
                                              (_fit, (115, 1), (160, 1))])
def test_launches_of_several_threads(make, small, large):
    import torch

    sizes = [small, large] * 4
    errors = []
    start = threading.Barrier(len(sizes))
    lib = svf.load()

    def loop(L, T):
        keep = []
        with svf.Context(0) as ctx:
            call = make(ctx, lib, L, T, keep)
            torch.cuda.synchronize()
            first = call()
            start.wait()
            for _ in range(2000):
                if first != svf.SVF_OK or call() != svf.SVF_OK:
                    errors.append((L, T, lib.svf_last_error()))
                    return

    threads = [threading.Thread(target=loop, args=a) for a in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
