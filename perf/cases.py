"""What a program that uses this library has it do, as cases that can be timed and compared.

Every case calls the Python package's public entry points on buffers such a program has at hand: a
BTF's samples in GPU memory, a factored BTF file that has been loaded, maps to render, luminance
slices to fit.  Texels are synthetic (``Context.synth_btf``: the uneven parameter mix, 20 %
near-diffuse and 10 % strongly anisotropic, 1 % noise); direction layouts are the 81-direction rings
and Fibonacci hemispheres.
"""
from __future__ import annotations

import math
import struct

import numpy as np
import torch

import tempestrenderer_b200 as svf

DEV = "cuda:0"
MIX = 1                 # synth_btf's uneven parameter mix
PI = float(np.float32(3.141592))      # the model's pi
LUM = (0.2126, 0.7152, 0.0722)
# multiply-add counts of the fit per ordered direction pair (FMA = 2): a Jacobian and a residual
FLOPS_PASS = 169 + 33
_kept: dict = {}


# ---- the cases -------------------------------------------------------------------------------

def listed():
    return [
        # one texel through the drop-in call, as a host program's own texel loop makes it
        {"name": "lsq_one_ring81", "kind": "lsq", "directions": 81, "texels": 1, "fresnel": 1.0},
        # a band of slices that is already on the GPU, at the refractive index svbrdffit defaults to
        {"name": "lsq_batch_ring81_n15", "kind": "lsq", "directions": 81, "texels": 2000, "fresnel": 1.5},
        # the plain LM workload: a small BTF, at most 100 iterations
        {"name": "fit_64x64_ring81", "kind": "fit", "directions": 81, "width": 64, "height": 64, "half": False,
         "rgb": False, "learned": False, "iterations": 100},
        # the benchmark's BTF
        {"name": "fit_400x400_ring81", "kind": "fit", "directions": 81, "width": 400, "height": 400, "half": False,
         "rgb": False, "learned": False, "iterations": 1024},
        # a dense layout in half precision, ragged sides
        {"name": "fit_97x89_fib151_half", "kind": "fit", "directions": 151, "width": 97, "height": 89, "half": True,
         "rgb": False, "learned": False, "iterations": 1024},
        # the 11-parameter colour fit
        {"name": "fit_rgb_201x149_ring81", "kind": "fit", "directions": 81, "width": 201, "height": 149,
         "half": False, "rgb": True, "learned": False, "iterations": 1024},
        # from the learned initial guess, half-precision samples
        {"name": "fit_learned_400x400_ring81_half", "kind": "fit", "directions": 81, "width": 400, "height": 400,
         "half": True, "rgb": False, "learned": True, "iterations": 1024},
        # a loaded factored file (half planes, 48 components per channel) to samples in GPU memory
        {"name": "decode_400x400_k48", "kind": "decode", "directions": 81, "width": 400, "height": 400,
         "components": 48, "plane_bytes": 2, "half": False},
        # the error tool over a whole file: fitted maps against the BTF, luminance, all pairs
        {"name": "error_128x128_k48", "kind": "error", "directions": 81, "width": 128, "height": 128,
         "components": 48, "plane_bytes": 2, "max_view": False, "color": False},
        # the BTF of SVBRDF maps
        {"name": "render_200x200_ring81", "kind": "render", "directions": 81, "width": 200, "height": 200,
         "half": False, "fresnel": 1.0},
        # the same with the multi-scattering model at its default depth
        {"name": "render_ms_16x16_ring81", "kind": "render_ms", "directions": 81, "width": 16, "height": 16,
         "bounces": 2, "half": False},
        # the learned initial guess trained for a layout (a quick training: fewer texels and epochs
        # than the default, the default's minibatch and step size)
        {"name": "train_16384_ring81", "kind": "train", "directions": 81, "texels": 16384, "epochs": 24,
         "batch": 4096},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, lo, hi):
    """Two sides of an image of about lo .. hi texels."""
    t = _log_int(rng, lo, hi)
    w = max(1, min(t, int(round(math.sqrt(t) * rng.uniform(0.7, 1.4)))))
    return w, max(1, t // w)


def draw(rng):
    kind = rng.choice(["lsq", "lsq", "fit", "fit", "fit", "decode", "error", "render", "render_ms", "train"])
    L = rng.choice([81, 81, 81, 151, rng.randint(24, 151)])
    pairs = (L / 81.0) ** 2
    if kind == "lsq":
        return {"kind": kind, "directions": L, "texels": _log_int(rng, 1, 8000 / pairs),
                "fresnel": rng.choice([1.0, 1.5])}
    if kind == "fit":
        rgb = rng.random() < 0.25
        learned = not rgb and rng.random() < 0.3
        if learned:
            L, pairs = 81, 1.0
        w, h = _sides(rng, 40, (30000 if rgb else 100000) / pairs)
        return {"kind": kind, "directions": L, "width": w, "height": h, "half": rng.random() < 0.5, "rgb": rgb,
                "learned": learned, "iterations": rng.choice([100, 1024])}
    if kind == "decode":
        w, h = _sides(rng, 100, 60000 / pairs)
        return {"kind": kind, "directions": L, "width": w, "height": h, "components": rng.randint(5, 60),
                "plane_bytes": rng.choice([2, 2, 2, 4]), "half": rng.random() < 0.5}
    if kind == "error":
        w, h = _sides(rng, 60, 10000 / pairs)
        return {"kind": kind, "directions": L, "width": w, "height": h, "components": rng.randint(5, 60),
                "plane_bytes": rng.choice([2, 2, 2, 4]), "max_view": rng.random() < 0.5, "color": rng.random() < 0.5}
    if kind == "render":
        w, h = _sides(rng, 40, 40000 / pairs)
        return {"kind": kind, "directions": L, "width": w, "height": h, "half": rng.random() < 0.5,
                "fresnel": rng.choice([1.0, 1.0, 1.5])}
    if kind == "render_ms":
        w, h = _sides(rng, 10, 256 / pairs)
        return {"kind": kind, "directions": L, "width": w, "height": h, "bounces": rng.randint(1, 3),
                "half": rng.random() < 0.5}
    return {"kind": kind, "directions": L if L <= 81 else 81, "texels": _log_int(rng, 3000, 16384),
            "epochs": rng.randint(3, 24), "batch": rng.choice([512, 1000, 4096])}


# ---- what a program has in hand --------------------------------------------------------------

def _context():
    """The program's one device context."""
    if "ctx" not in _kept:
        _kept["ctx"] = svf.Context(0)
    return _kept["ctx"]


def _lights(n):
    return svf.directions_ring81() if n == 81 else svf.directions_fibonacci(n)


def _model(n):
    """The trained model a program loads at its start (a short training: the weights are not measured)."""
    if ("mlp", n) not in _kept:
        opts = svf.mlp_train_options(texels=1 << 15, epochs=16, batch=2048)
        _kept["mlp", n] = svf.Mlp.train(_context(), _lights(n), opts)[0]
    return _kept["mlp", n]


def _generator(seed):
    g = torch.Generator(DEV)
    g.manual_seed(seed & 0x7fffffff)
    return g


def _rand(g, *shape):
    return torch.rand(shape, generator=g, device=DEV, dtype=torch.float32)


def _maps(g, T):
    """SVBRDF maps as a fit writes them (albedos, SGGX scales, orientations within 30 degrees of +z)."""
    kd, ks = 0.8 * _rand(g, T, 3), _rand(g, T, 3)
    sigma = torch.exp(math.log(0.02) + math.log(40.0) * _rand(g, T, 2))
    tilt, az, spin = 0.26 * torch.sqrt(_rand(g, T)), 2 * math.pi * _rand(g, T), math.pi * _rand(g, T)
    # tilt about an axis in the plane, after a spin about z (half angles)
    tx, ty, tw = torch.sin(tilt) * torch.cos(az), torch.sin(tilt) * torch.sin(az), torch.cos(tilt)
    sz, sw = torch.sin(spin), torch.cos(spin)
    quat = torch.stack([tx * sw + ty * sz, ty * sw - tx * sz, tw * sz, tw * sw], 1)
    return [m.cpu().numpy() for m in (kd, ks, sigma, quat)]


def _angles(n):
    """(theta, phi) of the layout's directions, as a BTF file stores them."""
    if n == 81:
        return np.array([(math.radians(15.0 * r), 2 * math.pi * k / c)
                         for r, c in enumerate((1, 6, 12, 18, 20, 24)) for k in range(c)], np.float32)
    p = _lights(n).astype(np.float64)
    q = (p ** 2).sum(1)
    return np.stack([np.arccos((1 - q) / (1 + q)), np.arctan2(p[:, 1], p[:, 0])], 1).astype(np.float32)


def _planes(case, seed):
    """U [3][pairs][K] (prototype texels) and SxV [texels][K] (each texel's weights of them), rounded
    to the file's element type."""
    n, K = case["directions"], case["components"]
    N, T = n * n, case["width"] * case["height"]
    dt = torch.float16 if case["plane_bytes"] == 2 else torch.float32
    proto = torch.empty((K, N, 3), dtype=torch.float32, device=DEV)
    _context().synth_btf(seed & 0x7fffffff, MIX, _lights(n), 0, K, proto)
    g = _generator(seed)
    w = (-torch.log(1.0 - _rand(g, T, K))) ** 3
    w /= w.sum(1, keepdim=True)
    return proto.permute(2, 1, 0).contiguous().to(dt), w.to(dt)


def _file(case, seed):
    """A DFMF file image of such a BTF (three channels, the same weights in each)."""
    U, S = (x.cpu().numpy() for x in _planes(case, seed))
    tp = _angles(case["directions"])
    L, K = len(tp), case["components"]
    parts = [b"!DFMF08FC", struct.pack("<II", 264, 1), b"\0" * 240, struct.pack("<f3f", 0.0, 1.0, 1.0, 1.0),
             struct.pack("<I", L)]
    for v in range(L):
        parts += [tp[v].tobytes(), struct.pack("<I", L), tp.tobytes()]
    parts += [struct.pack("<II", case["width"], case["height"]), struct.pack("<II", K, 0),
              struct.pack("<3f", 0, 0, 0), np.eye(3, dtype=np.float32).tobytes()]
    for c in range(3):
        parts += [struct.pack("<B", case["plane_bytes"]), struct.pack("<III", K, U.shape[1], S.shape[0]),
                  np.ones(K, U.dtype).tobytes(), U[c].tobytes(), S.tobytes()]
    return b"".join(parts)


def _slices(case, seed):
    """Luminance slices of synthetic texels and initial parameters near their truth, on the GPU."""
    n, T = case["directions"], case["texels"]
    lp = _lights(n)
    lum = torch.empty((T, n * n), dtype=torch.float32, device=DEV)
    truth = torch.empty((T, 16), dtype=torch.float32, device=DEV)
    w = torch.tensor(LUM, device=DEV)
    for t0 in range(0, T, 4096):
        t1 = min(T, t0 + 4096)
        s = torch.empty((t1 - t0, n * n, 3), dtype=torch.float32, device=DEV)
        _context().synth_btf(seed & 0x7fffffff, MIX, lp, t0, t1 - t0, s, truth=truth[t0:t1])
        lum[t0:t1] = s @ w
    g = _generator(seed)
    wob = 0.8 + 0.4 * _rand(g, T, 4)
    init = torch.cat([truth[:, 6:8] * wob[:, :2], (truth[:, 3:6] @ w)[:, None] * wob[:, 2:3],
                      (truth[:, 0:3] @ w)[:, None] * wob[:, 3:4], truth[:, 12:15] + 0.2 * (_rand(g, T, 3) - 0.5)], 1)
    return lp, lum, init.contiguous()


def _samples(T, N, half):
    return torch.empty((T, N, 3), dtype=torch.float16 if half else torch.float32, device=DEV)


def prepare(case, seed):
    kind, n = case["kind"], case["directions"]
    N = n * n
    st = dict(case=case, ctx=_context())
    if kind == "lsq":
        lp, lum, init = _slices(case, seed)
        T = case["texels"]
        st.update(lp=lp, opts=svf.options(fresnel=case["fresnel"]))
        if T == 1:   # the host call
            st.update(lum=lum[0].cpu().numpy(), init=init[0].cpu().numpy())
        else:
            st.update(lum=lum, init=init, out=torch.empty((T, 7), device=DEV), rmse=torch.empty(T, device=DEV),
                      stats=torch.empty((T, 5), dtype=torch.int32, device=DEV))
    elif kind == "fit":
        W, H = case["width"], case["height"]
        T, k = W * H, 12 if case["rgb"] else 7
        st["layout"] = svf.Layout(_lights(n))
        st["samples"] = _samples(T, N, case["half"])
        st["type"] = svf.SVF_SAMPLES_F16 if case["half"] else svf.SVF_SAMPLES_F32
        _context().synth_btf(seed & 0x7fffffff, MIX, _lights(n), 0, T, st["samples"], sample_type=st["type"])
        st["opts"] = svf.options(max_iterations=case["iterations"], rgb=case["rgb"])
        st["mlp"] = _model(n) if case["learned"] else None
        st["maps"] = {m: torch.empty((T, c), device=DEV) for m, c in
                      {"diffuse": 3, "specular": 3, "sigma": 2, "basis": 4, "rmse": 1, "params": k, "init": k}.items()}
        st["maps"]["stats"] = torch.empty((T, 5), dtype=torch.int32, device=DEV)
    elif kind in ("decode", "error"):
        st["btf"] = svf.Btf(_context(), _file(case, seed))
        W, H = case["width"], case["height"]
        if kind == "decode":
            st["out"] = _samples(W * H, N, case["half"])
            st["type"] = svf.SVF_SAMPLES_F16 if case["half"] else svf.SVF_SAMPLES_F32
        else:
            st["maps"] = [m.reshape(H, W, -1) for m in _maps(_generator(seed), W * H)]
    elif kind in ("render", "render_ms"):
        T = case["width"] * case["height"]
        st["lp"], st["maps"] = _lights(n), _maps(_generator(seed), T)
        st["out"] = _samples(T, N, case["half"])
        st["type"] = svf.SVF_SAMPLES_F16 if case["half"] else svf.SVF_SAMPLES_F32
    else:
        st["lp"] = _lights(n)
        st["opts"] = svf.mlp_train_options(texels=case["texels"], epochs=case["epochs"], batch=case["batch"],
                                           seed=seed & 0x7fffffff)
    return st


# ---- one pass --------------------------------------------------------------------------------

def run(st):
    case, ctx = st["case"], st["ctx"]
    kind = case["kind"]
    if kind == "lsq":
        if case["texels"] == 1:
            p, rmse, s = ctx.lsq_fit_sggx(st["lp"], st["lum"], st["init"], st["opts"])
            return {"params": p, "rmse": rmse, "iterations": int(s.iterations), "status": int(s.status)}
        p, rmse, s = ctx.lsq_fit_batch(st["lp"], st["lum"], st["init"], st["opts"], st["out"], st["rmse"], st["stats"])
        return {"params": p, "rmse": rmse, "stats": s}
    if kind == "fit":
        maps, _ = ctx.fit_texels(st["layout"], st["samples"], case["width"], case["height"], sample_type=st["type"],
                                 opts=st["opts"], want=tuple(st["maps"]), out=st["maps"], check=False, mlp=st["mlp"])
        return maps
    if kind == "decode":
        return st["btf"].decode(sample_type=st["type"], out=st["out"])
    if kind == "error":
        return st["btf"].error_maps(*st["maps"], color=case["color"],
                                    method=svf.SVF_ERROR_MAX_VIEW if case["max_view"] else svf.SVF_ERROR_PAIRWISE)
    if kind == "render":
        return ctx.render_btf(st["lp"], *st["maps"], fresnel=case["fresnel"], sample_type=st["type"], out=st["out"])
    if kind == "render_ms":
        return ctx.render_btf_ms(st["lp"], *st["maps"], case["bounces"], sample_type=st["type"], out=st["out"])
    model, loss = svf.Mlp.train(ctx, st["lp"], st["opts"])
    blob = model.save()
    # the file's tail: the weights and biases of the three layers
    n_w = 96 * 256 + 256 + 256 * 256 + 256 + 256 * 8 + 8
    return {"weights": np.frombuffer(blob, np.float32, n_w, len(blob) - 4 * n_w).copy(), "loss": loss}


def work(case):
    kind, N = case["kind"], case["directions"] ** 2
    T = case["texels"] if "texels" in case else case["width"] * case["height"]
    if kind == "lsq":
        return {"bytes": T * (4 * N + 4 * 20), "flops": T * N * FLOPS_PASS * 10}
    if kind == "fit":
        # LM iterations a texel: about 12 from the default guess, 4 from the learned one; the colour
        # fit follows the luminance fit
        passes = (4 if case["learned"] else 13) + (20 if case["rgb"] else 0)
        return {"bytes": T * (3 * N * (2 if case["half"] else 4) + 4 * (25 + (10 if case["rgb"] else 0) + 7)),
                "flops": T * N * FLOPS_PASS * passes}
    if kind in ("decode", "error"):
        K = case["components"]
        planes = 3 * K * (N + T) * case["plane_bytes"]
        flops = 2 * 3 * K * N * T
        if kind == "decode":
            return {"bytes": planes + T * N * 3 * (2 if case["half"] else 4), "flops": flops}
        return {"bytes": planes + 4 * T * (12 + 2 * (3 if case["color"] else 1)), "flops": flops + 50 * N * T}
    if kind == "render":
        return {"bytes": T * (N * 3 * (2 if case["half"] else 4) + 48), "flops": 40 * N * T}
    if kind == "render_ms":
        # about 200 flops a scattering event, 256 walks an evaluation
        return {"bytes": T * (N * 3 * (2 if case["half"] else 4) + 48), "flops": 256 * 200 * case["bounces"] * N * T}
    weights = 96 * 256 + 256 * 256 + 256 * 8
    return {"bytes": T * (case["epochs"] * 4 * (96 + 8)) + 4 * weights,
            "flops": 6 * weights * T * case["epochs"] + T * N * FLOPS_PASS * 13}


# ---- the same in 64 bits ---------------------------------------------------------------------

def _directions64(n, angles):
    """Cartesian directions [n][3]; angles: as derived from a file's (theta, phi)."""
    if angles:
        tp = torch.from_numpy(_angles(n)).to(DEV, torch.float64)
        t, p = tp[:, 0], tp[:, 1]
        return torch.stack([torch.sin(t) * torch.cos(p), torch.sin(t) * torch.sin(p), torch.cos(t)], 1)
    q = torch.from_numpy(_lights(n)).to(DEV, torch.float64)
    s = (q ** 2).sum(1, keepdim=True)
    return torch.cat([2 * q / (1 + s), (1 - s) / (1 + s)], 1)


def _brdf64(w, kd, ks, sigma, quat, fresnel=1.0):
    """The SGGX surface BRDF of texels [T] at all pairs (view, light): [T][n][n][3]."""
    q = quat / quat.norm(dim=1, keepdim=True)
    x, y, z, r = q.unbind(1)
    R = torch.stack([torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y + z * r), 2 * (x * z - y * r)], 1),
                     torch.stack([2 * (x * y - z * r), 1 - 2 * (x * x + z * z), 2 * (y * z + x * r)], 1),
                     torch.stack([2 * (x * z + y * r), 2 * (y * z - x * r), 1 - 2 * (x * x + y * y)], 1)], 1)
    a = torch.einsum("tij,dj->tdi", R, w)                         # R^T w
    sd = torch.cat([sigma, torch.ones_like(sigma[:, :1])], 1)
    c = w[:, 2]
    sp = (a * sd[:, None]).norm(dim=2) / c                        # sigma(w) / cos
    s = a[:, :, None] + a[:, None]                                # view, light
    g = (s ** 2).sum(3)
    Q = ((s / sd[:, None, None]) ** 2).sum(3)
    k = 1.0 / (4 * PI * sigma[:, 0] * sigma[:, 1])
    spec = k[:, None, None] / c[None, :, None] * g * g / (Q * Q * (sp[:, :, None] + sp[:, None]))
    if fresnel != 1.0:
        h = w[:, None] + w[None]
        cm = (h * w[None]).sum(2) / h.norm(dim=2)
        ct = torch.sqrt(1 - (1 - cm * cm) / fresnel ** 2)
        rp, rs = (fresnel * cm - ct) / (fresnel * cm + ct), (cm - fresnel * ct) / (cm + fresnel * ct)
        spec = spec * (0.5 * (rp * rp + rs * rs)).clamp(0, 1)
    return kd[:, None, None] * (c / PI)[None, None, :, None] + ks[:, None, None] * spec[..., None]


def _decoded64(case, U, S, t0, t1):
    """Samples [t1 - t0][pairs][3] of file texels (image rows are stored bottom up)."""
    W, H = case["width"], case["height"]
    t = torch.arange(t0, t1, device=DEV)
    rows = S[(H - 1 - t // W) * W + t % W].double()
    return torch.stack([rows @ U[c].double().T for c in range(3)], 2)


def exact(case, seed):
    kind, n = case["kind"], case["directions"]
    if kind not in ("decode", "error", "render"):
        return None     # a fit's end point, a random walk and trained weights have no 64-bit value of their own
    T = case["width"] * case["height"]
    step = max(1, 3_000_000 // (n * n))
    if kind == "decode":
        U, S = _planes(case, seed)
        return torch.cat([_decoded64(case, U, S, t, min(T, t + step)) for t in range(0, T, step)])
    kd, ks, sigma, quat = (torch.from_numpy(m).to(DEV, torch.float64) for m in _maps(_generator(seed), T))
    w = _directions64(n, kind == "error")
    if kind == "render":
        return torch.cat([_brdf64(w, *(m[t:t + step] for m in (kd, ks, sigma, quat)), case["fresnel"]).flatten(1, 2)
                          for t in range(0, T, step)])
    U, S = _planes(case, seed)
    lw = torch.tensor(LUM, device=DEV, dtype=torch.float64)
    rmse, psnr = [], []
    for t0 in range(0, T, step):
        t1 = min(T, t0 + step)
        b = _decoded64(case, U, S, t0, t1).unflatten(1, (n, n))
        f = _brdf64(w, *(m[t0:t1] for m in (kd, ks, sigma, quat)))
        if not case["color"]:
            b, f = (b @ lw)[..., None], (f @ lw)[..., None]
        sq = ((b - f) ** 2).sum(2)                                # per view: [T][n][C]
        peak = b.amax(2)
        if case["max_view"]:
            at = sq.argmax(1, keepdim=True)
            mse, top = sq.gather(1, at)[:, 0] / n, peak.gather(1, at)[:, 0]
        else:
            mse, top = sq.sum(1) / (n * n), peak.amax(1)
        rmse.append(mse.sqrt())
        psnr.append(20 * torch.log10(top / mse.sqrt()))
    shape = (case["height"], case["width"], 3) if case["color"] else (case["height"], case["width"])
    return torch.cat(rmse).reshape(shape), torch.cat(psnr).reshape(shape)
