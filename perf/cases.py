"""What hologram programs ask of this framework, as measurable cases.

Each case is one call (or the short chain of calls that a program makes for
one hologram) through the public entry points: depth-map frames, point-cloud
and point-light-source sums, wavefront-recording planes with their Fresnel
propagation, the encoders, and the learned surrogate's layers and network.
`listed()` names the cases, `draw()` gives more of the same ranges,
`prepare()` makes a case's inputs and parameters, `run()` is one pass and
`exact()` states the same result in 64 bits with plain torch.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from openholo_gb300 import _lib, depthmap, surrogate
from openholo_gb300.pls import PointLightSources

PITCH, LAM = 8e-6, 532e-9
ENC_PHASE_ONLY_U8, ENC_SSB_LEFT = 9, 5


def listed():
    return [
        # the benchmark frame: one 1080p RGB-D frame of a video or a display loop, inputs resident on the GPU
        dict(name="depthmap_1080p", kind="depthmap", nx=1920, ny=1080, layers=32, pad=2, fp64=False,
             phase="seeded", window=False, field=False, host=False),
        # a thumbnail or preview on the reference's own grid, where launches and latency count
        dict(name="depthmap_small", kind="depthmap", nx=256, ny=128, layers=16, pad=1, fp64=False,
             phase="reference", window=True, field=False, host=False),
        # an odd-sized SLM region with measured per-pixel phase, the complex field wanted too
        dict(name="depthmap_ragged", kind="depthmap", nx=1155, ny=819, layers=24, pad=2, fp64=False,
             phase="array", window=False, field=True, host=False),
        # HologramGenerator.GenerateHologram as the reference runs it: double precision, the reference's
        # grid and viewing-window transform, images and fringe in host memory
        dict(name="depthmap_fp64_host", kind="depthmap", nx=1920, ny=1080, layers=32, pad=1, fp64=True,
             phase="reference", window=True, field=False, host=True),
        # an offline job: frames of uneven size, depth and wavelength in one call
        dict(name="depthmap_batch", kind="batch", sides="512,2048,768,1024,1536,512,1024,768",
             layers="21,40,64,8,33,52,47,12", lams="450,532,633,532,450,633,450,532"),
        # a display-rate point cloud in single precision
        dict(name="pointcloud_fp32", kind="pointcloud", nx=1024, ny=1024, points=5000, fp64=False, tilt=0.0),
        # the point-cloud hologram in double precision, the reference result a user checks others against
        dict(name="pointcloud_fp64", kind="pointcloud", nx=1024, ny=1024, points=5000, fp64=True, tilt=0.0),
        # paraxial point-light-source sum (the tensor-core contraction)
        dict(name="pls_fresnel", kind="pls", nx=1024, ny=1024, points=5000, mode="fresnel", fp64=False),
        # a 4K hologram of a dense point set by way of a wavefront-recording plane
        dict(name="wrp_hologram_4k", kind="wrp", nx=3840, ny=2160, points=200000, window=32),
        # a complex field turned into a phase-only SLM image and a single-sideband amplitude image
        dict(name="encode_1080p", kind="encode", nx=1920, ny=1080, fp64=False),
        # one decoder layer of the surrogate in training: forward, input gradient, weight gradient
        dict(name="conv_layer_train", kind="conv", n=4, h=512, w=512, cin=192, cout=64),
        # the surrogate's inference on one RGB-D frame
        dict(name="unet_forward", kind="unet", n=1, h=1024, w=1024),
    ]


# ---- further cases of the same ranges ----------------------------------------

def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _smooth(n):
    """The nearest length at or below n whose prime factors are at most 13."""
    while True:
        m = n
        for p in (2, 3, 5, 7, 11, 13):
            while m % p == 0:
                m //= p
        if m == 1:
            return n
        n -= 1


def draw(rng):
    kind = rng.choice(["depthmap", "depthmap", "depthmap", "batch", "pointcloud", "pls", "wrp", "encode", "conv",
                       "unet"])
    if kind == "depthmap":
        fp64 = rng.random() < 0.3
        pad = rng.choice([1, 2])
        nx = rng.choice([1920, 1024, 960, 512, _smooth(_log_int(rng, 96, 1920)), _smooth(_log_int(rng, 96, 1920))])
        ny = rng.choice([1080, 1024, 540, 512, _smooth(_log_int(rng, 64, 1080)), _smooth(_log_int(rng, 64, 1080))])
        return dict(kind=kind, nx=nx, ny=ny, layers=rng.randint(4, 32), pad=pad, fp64=fp64,
                    phase=rng.choice(["reference", "seeded", "array"]), window=rng.random() < 0.5,
                    field=rng.random() < 0.3, host=rng.random() < 0.3)
    if kind == "batch":
        n = rng.randint(2, 8)
        return dict(kind=kind, sides=",".join(str(rng.choice([512, 768, 1024, 1536])) for _ in range(n)),
                    layers=",".join(str(rng.randint(8, 64)) for _ in range(n)),
                    lams=",".join(str(rng.choice([450, 532, 633])) for _ in range(n)))
    if kind == "pointcloud":
        return dict(kind=kind, nx=_log_int(rng, 100, 1024), ny=_log_int(rng, 100, 1024),
                    points=_log_int(rng, 30, 5000), fp64=rng.random() < 0.5, tilt=rng.choice([0.0, 0.0, 1.5]))
    if kind == "pls":
        return dict(kind=kind, nx=_log_int(rng, 100, 1536), ny=_log_int(rng, 100, 1536),
                    points=_log_int(rng, 30, 5000), mode=rng.choice(["fresnel", "fresnel", "cgh_fresnel", "huygens"]),
                    fp64=False)
    if kind == "wrp":
        nx, ny = rng.choice([(3840, 2160), (1920, 1080), (1024, 1024), (_smooth(_log_int(rng, 200, 2000)),
                                                                       _smooth(_log_int(rng, 200, 1500)))])
        return dict(kind=kind, nx=nx, ny=ny, points=_log_int(rng, 300, 200000), window=rng.choice([16, 24, 32, 32]))
    if kind == "encode":
        nx, ny = rng.choice([(3840, 2160), (1920, 1080), (1024, 1024), (_smooth(_log_int(rng, 100, 2000)),
                                                                       _smooth(_log_int(rng, 100, 2000)))])
        return dict(kind=kind, nx=nx, ny=ny, fp64=rng.random() < 0.25)
    if kind == "conv":
        return dict(kind=kind, n=rng.randint(1, 4), h=rng.randint(16, 512), w=rng.choice([32, 64, 128, 160, 256, 512]),
                    cin=32 * rng.randint(1, 12), cout=rng.choice([32, 64, 128, 256]))
    return dict(kind="unet", n=rng.randint(1, 2), h=8 * rng.randint(8, 96), w=rng.choice([128, 256, 512, 1024]))


# ---- inputs ----------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _rand(g, *shape):
    return torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)


def _gaussians(g, ny, nx, count, lo, hi):
    """Sum of `count` random 2-D Gaussians, sigmas lo..hi pixels."""
    u = _rand(g, count, 4)
    s = (lo + u[:, 2] * (hi - lo))[:, None]
    x = torch.arange(nx, device="cuda", dtype=torch.float64)[None]
    y = torch.arange(ny, device="cuda", dtype=torch.float64)[None]
    gx = torch.exp(-((x - u[:, :1] * nx) ** 2) / (2 * s * s))
    gy = torch.exp(-((y - u[:, 1:2] * ny) ** 2) / (2 * s * s))
    return gy.T @ (gx * (0.2 + 0.8 * u[:, 3:]))


def _bytes(v):
    return torch.clamp(torch.round(255.0 * v), 0, 255).to(torch.uint8)


def _scene(g, ny, nx):
    """uint8 intensity (20 Gaussians) and depth (8 broad ones over the full byte range)."""
    sc = min(ny, nx) / 1080.0
    inten = _gaussians(g, ny, nx, 20, 20 * sc, 200 * sc)
    dep = _gaussians(g, ny, nx, 8, 200 * sc, 600 * sc)
    dep = dep - dep.min()
    return _bytes(inten / inten.max()), _bytes(dep / dep.max())


def _dm_inputs(case, seed):
    g = _gen(seed)
    img, dep = _scene(g, case["ny"], case["nx"])
    phase = None
    if case["phase"] == "array":
        phase = (2 * math.pi * _rand(g, case["ny"], case["nx"])).float()
    return img, dep, phase


def _dm_params(nx, ny, layers, pad, window, phase, seed, lam=LAM):
    mode = dict(reference=_lib.OH_PHASE_REFERENCE, array=_lib.OH_PHASE_ARRAY, seeded=_lib.OH_PHASE_SEEDED)[phase]
    return depthmap.make_params(pnx=nx, pny=ny, num_of_depth=layers, pad=pad, lam=lam, phase_mode=mode,
                                transform_viewing_window=1 if window else 0, seed=int(seed))


def _batch_frames(case):
    return list(zip([int(v) for v in case["sides"].split(",")], [int(v) for v in case["layers"].split(",")],
                    [int(v) * 1e-9 for v in case["lams"].split(",")]))


def _pc_points(case, seed):
    """x, y in +-2 mm, z in 0.10-0.12 m, amplitude 0-1 (float4 records)."""
    u = _rand(_gen(seed), case["points"], 4)
    lo = torch.tensor([-2e-3, -2e-3, 0.10, 0.0], device="cuda", dtype=torch.float64)
    hi = torch.tensor([2e-3, 2e-3, 0.12, 1.0], device="cuda", dtype=torch.float64)
    return (lo + u * (hi - lo)).float()


def _pls_points(case, seed):
    """Unit-amplitude records (a_re, a_im, x, y, z) over the same box."""
    p = _pc_points(case, seed)
    out = torch.zeros((case["points"], 5), device="cuda")
    out[:, 0] = 1.0
    out[:, 2:] = p[:, :3]
    return out


WRP_PITCH, WRP_ZC, WRP_Z = 3.74e-6, 0.2, 0.194


def _wrp_points(case, seed):
    """Points of a box as wide as the plane (at most 10 mm), 2 mm deep, 5 mm behind the plane."""
    u = _rand(_gen(seed), case["points"], 3) - 0.5
    box = torch.tensor([min(10e-3, case["nx"] * WRP_PITCH), min(10e-3, case["ny"] * WRP_PITCH), 2e-3],
                       device="cuda", dtype=torch.float64)
    return (u * box + torch.tensor([0.0, 0.0, WRP_ZC], device="cuda", dtype=torch.float64)).contiguous()


def _field(case, seed):
    """A hologram-like field: a smooth amplitude under a random phase, band-limited by a small blur."""
    g = _gen(seed)
    ny, nx = case["ny"], case["nx"]
    amp = _gaussians(g, ny, nx, 12, 0.05 * min(nx, ny), 0.4 * min(nx, ny)) + 0.05
    u = torch.polar(amp, 2 * math.pi * _rand(g, ny, nx))
    u = u + torch.roll(u, 1, 0) + torch.roll(u, 1, 1)
    return u if case["fp64"] else u.to(torch.complex64)


def _conv_inputs(case, seed):
    """Activations after a ReLU, a sparse output gradient, He-scaled weights in both layouts, a bias."""
    g = _gen(seed)
    n, h, w, ci, co = (case[k] for k in ("n", "h", "w", "cin", "cout"))

    def normal(*s):
        return torch.randn(s, generator=g, device="cuda", dtype=torch.float32)

    x = torch.relu(normal(n, h, w, ci)).bfloat16()
    dz = (normal(n, h, w, co) * (normal(n, h, w, co) > 0)).bfloat16()
    wt = (normal(co, 9, ci) * math.sqrt(2.0 / (9 * ci))).bfloat16()
    return x, dz, wt, 0.1 * normal(co)


def _unet_inputs(case, seed):
    g = _gen(seed)
    n, h, w = case["n"], case["h"], case["w"]
    rgbd = torch.empty((n, h, w, 4), dtype=torch.uint8, device="cuda")
    for i in range(n):
        for c in (0, 2):
            rgbd[i, ..., c], _ = _scene(g, h, w)
        rgbd[i, ..., 1], rgbd[i, ..., 3] = _scene(g, h, w)
    parts = []
    for name, ci, co, taps in surrogate.layer_shapes():
        sd = math.sqrt(2.0 / (taps * ci)) * (0.1 if name == "head" else 1.0)
        parts += [torch.randn(co * taps * ci, generator=g, device="cuda") * sd,
                  torch.randn(co, generator=g, device="cuda") * 0.02]
    return rgbd, torch.cat(parts).cpu().numpy()


# ---- one pass --------------------------------------------------------------------

_CTX = []


def _ctx():
    """The context that a program keeps for its lifetime."""
    if not _CTX:
        _CTX.append(_lib.Context(0))
    return _CTX[0]


def _p(t):
    return C.c_void_p(t.data_ptr()) if t is not None else None


def _st():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def prepare(case, seed):
    ctx, k = _ctx(), case["kind"]
    s = dict(case=case, ctx=ctx)
    if k == "depthmap":
        img, dep, phase = _dm_inputs(case, seed)
        s["p"] = _dm_params(case["nx"], case["ny"], case["layers"], case["pad"], case["window"], case["phase"], seed)
        if case["host"]:
            img, dep, phase = (None if t is None else t.cpu().numpy() for t in (img, dep, phase))
        s.update(img=img, dep=dep, phase=phase)
    elif k == "batch":
        s["frames"] = []
        for i, (side, layers, lam) in enumerate(_batch_frames(case)):
            img, dep = _scene(_gen(seed * 64 + i), side, side)
            p = _dm_params(side, side, layers, 2, False, "seeded", seed * 64 + i, lam)
            s["frames"].append((p, img, dep, torch.empty((side, side), device="cuda")))
    elif k == "pointcloud":
        s["pts"] = _pc_points(case, seed)
        s["p"] = _lib.PcParams(1.0, 1.0, 1.0, 0.0, PITCH, PITCH, case["nx"], case["ny"], LAM, case["tilt"], 0.0)
    elif k == "pls":
        s["src"] = PointLightSources(ctx, case["nx"], case["ny"], pitch=(PITCH, PITCH), lam=LAM,
                                     precision="fp64" if case["fp64"] else "fp32")
        s["src"].set_points(_pls_points(case, seed))
    elif k == "wrp":
        s["pts"] = _wrp_points(case, seed)
        s["p"] = _lib.WrpParams(case["nx"], case["ny"], WRP_PITCH, LAM, WRP_Z, case["window"])
    elif k == "encode":
        s["u"] = _field(case, seed)
    elif k == "conv":
        x, dz, wt, b = _conv_inputs(case, seed)
        # the input gradient reads the weights transposed: [cin][taps * cout]
        s.update(x=x, dz=dz, w=wt.reshape(case["cout"], -1).contiguous(), b=b,
                 wd=wt.permute(2, 1, 0).reshape(case["cin"], -1).contiguous())
    else:
        s["rgbd"], flat = _unet_inputs(case, seed)
        s["net"] = surrogate.UNet(ctx, max_batch=case["n"], max_height=case["h"], max_width=case["w"])
        s["net"].set_params(flat)
    return s


def run(s):
    case, ctx = s["case"], s["ctx"]
    k = case["kind"]
    if k == "depthmap":
        prec = "fp64" if case["fp64"] else "fp32"
        if case["host"]:
            return depthmap.generate_host(ctx, s["p"], s["img"], s["dep"], s["phase"], precision=prec)
        field = None
        if case["field"]:
            field = torch.empty((case["ny"], case["nx"]), device="cuda",
                                dtype=torch.complex128 if case["fp64"] else torch.complex64)
        fringe = depthmap.generate(ctx, s["p"], s["img"], s["dep"], s["phase"], precision=prec, field=field)
        return dict(fringe=fringe) if field is None else dict(fringe=fringe, field=field)
    if k == "batch":
        depthmap.generate_batch(ctx, s["frames"])
        return [f[3] for f in s["frames"]]
    if k == "pointcloud":
        out = torch.empty((case["ny"], case["nx"]), device="cuda",
                          dtype=torch.complex128 if case["fp64"] else torch.complex64)
        _lib.call("oh_pointcloud", ctx.handle, 1 if case["fp64"] else 0, C.byref(s["p"]), _p(s["pts"]),
                  case["points"], _p(out), None, _st())
        return out
    if k == "pls":
        f = dict(fresnel=s["src"].Fresnel, cgh_fresnel=s["src"].CGHFresnel, huygens=s["src"].Huygens)[case["mode"]]
        return f(0.0)
    if k == "wrp":
        u = torch.zeros((case["ny"], case["nx"]), dtype=torch.complex64, device="cuda")
        _lib.call("oh_wrp_accumulate", ctx.handle, 0, C.byref(s["p"]), _p(s["pts"]), case["points"], _p(u), _st())
        _lib.call("oh_fresnel_propagate", ctx.handle, 0, case["nx"], case["ny"], WRP_PITCH, LAM, WRP_Z, _p(u), _st())
        return u
    if k == "encode":
        ny, nx = case["ny"], case["nx"]
        slm = torch.empty((ny, nx), dtype=torch.uint8, device="cuda")
        ssb = torch.empty((ny, nx), dtype=torch.float64 if case["fp64"] else torch.float32, device="cuda")
        for kind, out in ((ENC_PHASE_ONLY_U8, slm), (ENC_SSB_LEFT, ssb)):
            _lib.call("oh_encode", ctx.handle, 1 if case["fp64"] else 0, kind, nx, ny, _p(s["u"]), _p(out), _st())
        return dict(phase_only=slm, ssb=ssb)
    if k == "conv":
        n, h, w, ci, co = (case[q] for q in ("n", "h", "w", "cin", "cout"))
        y = torch.empty((n, h, w, co), dtype=torch.bfloat16, device="cuda")
        dx = torch.empty((n, h, w, ci), dtype=torch.bfloat16, device="cuda")
        dw = torch.zeros((9 * ci, co), device="cuda")
        _lib.call("oh_conv2d_bf16", ctx.handle, 9, 1, n, h, w, ci, co, _p(s["x"]), ci, _p(s["w"]), _p(s["b"]), 1,
                  None, 0, _p(y), co, _st())
        _lib.call("oh_conv2d_bf16", ctx.handle, 9, -1, n, h, w, co, ci, _p(s["dz"]), co, _p(s["wd"]), None, 0,
                  _p(s["x"]), ci, _p(dx), ci, _st())
        _lib.call("oh_conv2d_wgrad_bf16", ctx.handle, 9, n, h, w, ci, co, _p(s["x"]), ci, _p(s["dz"]), co, _p(dw),
                  _st())
        return dict(y=y, dx=dx, dw=dw)
    return s["net"].forward(s["rgbd"])


# ---- what a pass cannot do without ---------------------------------------------

def _fft(n):
    """Operations of one complex transform of length n."""
    return 5.0 * n * math.log2(max(n, 2))


def _dm_work(nx, ny, layers, pad, fp64, phase, field):
    px, py, r = pad * nx, pad * ny, 8 if fp64 else 4
    nbytes = nx * ny * (2 + r + (4 if phase == "array" else 0) + (2 * r if field else 0))
    # per layer: row transforms of the image rows, column transforms, transfer-function multiply-add;
    # once: the inverse transforms of the cropped spectrum
    flops = layers * (ny * _fft(px) + px * _fft(py) + 8.0 * px * py) + px * _fft(py) + ny * _fft(px)
    return nbytes, flops


def work(case):
    k = case["kind"]
    if k == "depthmap":
        b, f = _dm_work(case["nx"], case["ny"], case["layers"], case["pad"], case["fp64"], case["phase"],
                        case["field"])
    elif k == "batch":
        b = f = 0
        for side, layers, _ in _batch_frames(case):
            bi, fi = _dm_work(side, side, layers, 2, False, "seeded", False)
            b, f = b + bi, f + fi
    elif k == "pointcloud":
        n = case["nx"] * case["ny"]
        b = n * (16 if case["fp64"] else 8) + 16 * case["points"]
        f = 20.0 * n * case["points"]       # distance, phase, sine and cosine, two sums
    elif k == "pls":
        n = case["nx"] * case["ny"]
        b = n * (4 if case["mode"] == "cgh_fresnel" else 8) * (2 if case["fp64"] else 1) + 20 * case["points"]
        f = (20.0 if case["mode"] == "huygens" else 8.0) * n * case["points"]
    elif k == "wrp":
        nx, ny = case["nx"], case["ny"]
        b = 24 * case["points"] + 8 * nx * ny
        f = 8.0 * case["points"] * (2 * case["window"]) ** 2 + 2 * (ny * _fft(2 * nx) + nx * _fft(2 * ny))
    elif k == "encode":
        nx, ny, r = case["nx"], case["ny"], 8 if case["fp64"] else 4
        b = nx * ny * (2 * r + 1 + r)
        f = 2 * (ny * _fft(nx) + nx * _fft(ny)) + 20.0 * nx * ny
    elif k == "conv":
        n = case["n"] * case["h"] * case["w"]
        b = n * (2 * case["cin"] + 2 * case["cout"]) * 2 + 9 * case["cin"] * case["cout"] * 8
        f = 3 * 2.0 * n * 9 * case["cin"] * case["cout"]
    else:
        n = case["n"] * case["h"] * case["w"]
        b, f, level = 12 * n, 0.0, dict(enc0=0, enc1=1, enc2=2, enc3=3, dec2=2, dec1=1, dec0=0, head=0)
        for name, ci, co, taps in surrogate.layer_shapes():
            f += 2.0 * (n >> (2 * level[name[:4]])) * taps * ci * co
            b += 4 * taps * ci * co
    return dict(bytes=b, flops=f)


# ---- the same results in 64 bits ------------------------------------------------

def _ar(n):
    return torch.arange(n, device="cuda", dtype=torch.float64)


def _cis(ph):
    return torch.polar(torch.ones_like(ph), ph)


def _turns(t):
    """exp(2 pi i t), t reduced first."""
    return _cis(2 * math.pi * (t - torch.round(t)))


def _shift2(a):
    """Shift by floor(n/2) along both axes."""
    return torch.roll(a, (a.shape[0] // 2, a.shape[1] // 2), (0, 1))


def _exact_frame(nx, ny, layers, pad, window, lam, img, dep, src):
    """Layered angular-spectrum frame: levels over 0.30-0.35 m, binning, padded propagation, the upper
    sideband's crop window, centre region times the encoding's shift phase.  Returns the complex field."""
    near, far = 0.30, 0.35
    if layers > 1:
        step = (far - near) / (layers - 1)
        lev, val = [], near
        while len(lev) < layers:
            lev.append(val)
            val += step
    else:
        step, lev = (far + near) / 2, [far - near]
    lut = [0] * 256
    for b in range(256):
        d = (1 - b / 255.0) * (far - near) + near
        for i, t in enumerate(lev):
            above = d < t + step / 2.0 if i < layers - 1 else d <= t + step / 2.0
            lut[b] += (i + 1) * (d >= t - step / 2.0 and above)
    idx = torch.tensor(lut, device="cuda")[dep.long()] * (img > 0)
    px, py = pad * nx, pad * ny
    ox, oy = (px - nx) // 2, (py - ny) // 2
    fx = -1.0 / (2 * PITCH) + _ar(px) / (PITCH * px)
    fy = 1.0 / (2 * PITCH) - (1.0 + _ar(py)) / (PITCH * py)
    s = (lam * fx)[None] ** 2 + (lam * fy)[:, None] ** 2
    g = s / (1 + torch.sqrt(1 - s))                  # 1 - sqrt(1 - s): the carrier cancels the constant part
    spec = torch.zeros((py, px), dtype=torch.complex128, device="cuda")
    for i, t in enumerate(lev):
        m = idx == i + 1
        if not bool(m.any()):
            continue
        z = -t / (t - 1.0) if window else t
        u = torch.zeros((py, px), dtype=torch.complex128, device="cuda")
        u[oy:oy + ny, ox:ox + nx] = torch.where(m, src, torch.zeros_like(src))
        spec += _turns(g * (z / lam)) * _shift2(torch.fft.fft2(_shift2(u)))
    c1 = py // 2 - (py // 2) // 2 - 1
    keep = torch.zeros((py, 1), device="cuda", dtype=torch.float64)
    keep[c1:c1 + py // 2] = 1.0
    h = _shift2(torch.fft.ifft2(_shift2(spec * keep)))[oy:oy + ny, ox:ox + nx]
    yy = ny * PITCH / 2 - PITCH * _ar(ny) - PITCH
    return h * _turns(yy / (4 * PITCH))[:, None]


def _seeded_phase(seed, ny, nx, fp64):
    with np.errstate(over="ignore"):
        z = np.uint64(seed) + (np.arange(ny * nx, dtype=np.uint64) + np.uint64(1)) * np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        z = z ^ (z >> np.uint64(31))
    u = (z >> np.uint64(40)).astype(np.float32) * np.float32(2.0 ** -24)
    ph = u.astype(np.float64) * (2 * math.pi) if fp64 else u * np.float32(2 * math.pi)
    return torch.from_numpy(ph.astype(np.float64)).cuda().reshape(ny, nx)


def _exact_depthmap(case, seed):
    img, dep, phase = _dm_inputs(case, seed)
    src = (img.double() / 255.0).to(torch.complex128)
    if case["phase"] == "array":
        src = src * _cis(phase.double())
    elif case["phase"] == "seeded":
        src = src * _cis(_seeded_phase(seed, case["ny"], case["nx"], case["fp64"]))
    f = _exact_frame(case["nx"], case["ny"], case["layers"], case["pad"], case["window"], LAM, img, dep, src)
    if case["host"]:
        return f.real.contiguous()
    return dict(fringe=f.real.contiguous(), field=f) if case["field"] else dict(fringe=f.real.contiguous())


def _exact_batch(case, seed):
    out = []
    for i, (side, layers, lam) in enumerate(_batch_frames(case)):
        img, dep = _scene(_gen(seed * 64 + i), side, side)
        src = (img.double() / 255.0) * _cis(_seeded_phase(seed * 64 + i, side, side, False))
        out.append(_exact_frame(side, side, layers, 2, False, lam, img, dep, src).real.contiguous())
    return out


def _sum_points(X, Y, x, y, z, a, wave, tilt, spherical):
    """sum_j a_j exp(2 pi i t_j) [/ r_j]: t = r / lambda (wave "exact") or rho^2 / (2 z lambda) ("paraxial"),
    the distance split as z + rho^2 / (r + z) so that no digit of the phase is lost."""
    out = torch.zeros((Y.numel(), X.numel()), dtype=torch.complex128, device="cuda")
    per = max(1, int(3e7 // out.numel()))
    for j in range(0, x.numel(), per):
        xs, ys, zs, am = (v[j:j + per, None, None] for v in (x, y, z, a))
        rho2 = (X[None, None, :] - xs) ** 2 + (Y[None, :, None] - ys) ** 2
        r = torch.sqrt(rho2 + zs * zs)
        if wave == "exact":
            t0 = zs / LAM
            v = _turns((t0 - torch.round(t0)) + rho2 / (r + zs) / LAM - tilt[None, None, :])
        else:
            v = _turns(rho2 / (2 * zs * LAM))
        out += torch.sum(v * (am / r if spherical else am), 0)
    return out


def _exact_pointcloud(case, seed):
    p = _pc_points(case, seed).double()
    nx, ny = case["nx"], case["ny"]
    X = (_ar(nx) + 0.5) * PITCH - nx * PITCH / 2
    Y = ny * PITCH / 2 - (_ar(ny) + 0.5) * PITCH
    tilt = X * math.sin(math.radians(case["tilt"])) / LAM
    return _sum_points(X, Y, p[:, 0], p[:, 1], p[:, 2], p[:, 3], "exact", tilt, False)


def _exact_pls(case, seed):
    p = _pls_points(case, seed).double()
    X, Y = (_ar(case["nx"]) - case["nx"] // 2) * PITCH, (_ar(case["ny"]) - case["ny"] // 2) * PITCH
    x, y, z = p[:, 2], p[:, 3], p[:, 4]
    if case["mode"] == "huygens":
        return _sum_points(X, Y, x, y, z, torch.ones_like(x), "exact", 0 * X, True)
    ex = _turns((X[None] - x[:, None]) ** 2 / (2 * LAM * z[:, None]))
    ey = _turns((Y[None] - y[:, None]) ** 2 / (2 * LAM * z[:, None]))
    u = ey.T @ ex
    return u if case["mode"] == "fresnel" else u.real.contiguous()


def _exact_wrp(case, seed):
    p = _wrp_points(case, seed)
    nx, ny, w = case["nx"], case["ny"], case["window"]
    # the plane position, the pitch and the wave number are single-precision numbers there
    dp, zw, k = (float(np.float32(v)) for v in (WRP_PITCH, WRP_Z, 2 * math.pi / LAM))
    tx = torch.trunc(p[:, 0] / dp).long() + nx // 2
    ty = torch.trunc(p[:, 1] / dp).long() + ny // 2
    dz = zw - p[:, 2]
    o = torch.arange(-w, w, device="cuda")
    rho2 = ((o * dp) ** 2)[None, :] + ((o * dp) ** 2)[:, None]
    re = torch.zeros(nx * ny, dtype=torch.float64, device="cuda")
    im = torch.zeros_like(re)
    per = max(1, 16_000_000 // (4 * w * w))
    for j in range(0, p.shape[0], per):
        d = dz[j:j + per, None, None]
        r = torch.sign(d) * torch.sqrt(rho2 + d * d)
        X = tx[j:j + per, None, None] + o[None, None, :]
        Y = ty[j:j + per, None, None] + o[None, :, None]
        ok = (X >= 0) & (X < nx) & (Y >= 0) & (Y < ny)
        at = (Y * nx + X)[ok]
        re.index_add_(0, at, (torch.cos(k * r) / (r + 0.05))[ok])
        im.index_add_(0, at, (torch.sin(k * r) / (r + 0.05))[ok])
    u = torch.complex(re, im).reshape(ny, nx)
    # Fresnel convolution on the doubled grid
    px, py, ox, oy = 2 * nx, 2 * ny, nx // 2, ny // 2
    jx, jy = _ar(px), _ar(py)
    jx, jy = torch.where(jx < nx, jx, jx - px), torch.where(jy < ny, jy, jy - py)
    gx = torch.fft.fft(_turns((jx * WRP_PITCH) ** 2 / (2 * LAM * WRP_Z)))
    gy = torch.fft.fft(_turns((jy * WRP_PITCH) ** 2 / (2 * LAM * WRP_Z)))
    a = torch.zeros((py, px), dtype=torch.complex128, device="cuda")
    a[oy:oy + ny, ox:ox + nx] = u
    a = torch.fft.fft2(a)
    a *= gx[None, :]
    a *= gy[:, None]
    a = torch.fft.ifft2(a)[oy:oy + ny, ox:ox + nx]
    kz = 2 * math.pi * math.fmod(WRP_Z / LAM, 1.0)
    return a * (complex(math.cos(kz), math.sin(kz)) * WRP_PITCH ** 2 / (1j * LAM * WRP_Z))


def _exact_encode(case, seed):
    u = _field(case, seed).to(torch.complex128)
    ny, nx = u.shape
    spec = _shift2(torch.fft.fft2(_shift2(u)))
    spec[:, nx // 2 - 1:] = 0
    re = _shift2(torch.fft.ifft2(_shift2(spec))).real
    return dict(phase_only=None, ssb=((re - re.min()) / (re.max() - re.min())).contiguous())


def _taps(h, w):
    """(tap, output window, input window) of the nine shifts with zero padding."""
    for t in range(9):
        dy, dx = t // 3 - 1, t % 3 - 1
        yield (t, (slice(max(0, -dy), h - max(0, dy)), slice(max(0, -dx), w - max(0, dx))),
               (slice(max(0, dy), h + min(0, dy)), slice(max(0, dx), w + min(0, dx))))


def _conv64(x, wt, b):
    """x [n, h, w, cin], wt [cout, 9, cin] in 64 bits."""
    n, h, w, _ = x.shape
    y = torch.zeros((n, h, w, wt.shape[0]), dtype=torch.float64, device="cuda") + b
    for t, o, i in _taps(h, w):
        y[(slice(None), *o)] += x[(slice(None), *i)] @ wt[:, t].T
    return y


def _exact_conv(case, seed):
    x, dz, wt, b = (v.double() for v in _conv_inputs(case, seed))
    h, w = case["h"], case["w"]
    y = torch.relu(_conv64(x, wt, b))
    dx = torch.zeros_like(x)
    dw = torch.zeros((9, case["cin"], case["cout"]), dtype=torch.float64, device="cuda")
    for t, o, i in _taps(h, w):
        d = dz[(slice(None), *o)]
        dx[(slice(None), *i)] += d @ wt[:, t]
        dw[t] = x[(slice(None), *i)].reshape(-1, case["cin"]).T @ d.reshape(-1, case["cout"])
    return dict(y=y, dx=dx * (x > 0), dw=dw.reshape(-1, case["cout"]))


def _exact_unet(case, seed):
    rgbd, flat = _unet_inputs(case, seed)
    par = {k: (torch.from_numpy(w).cuda().double(), torch.from_numpy(b).cuda().double())
           for k, (w, b) in surrogate.unflatten(flat).items()}

    def block(v, name):
        return torch.relu(_conv64(torch.relu(_conv64(v, *par[name + "a"])), *par[name + "b"]))

    h, enc = rgbd.double() / 255.0, []
    for lv in range(4):
        e = block(h, "enc%d" % lv)
        enc.append(e)
        n, hh, ww, c = e.shape
        h = e.reshape(n, hh // 2, 2, ww // 2, 2, c).mean((2, 4)) if lv < 3 else e
    for lv in (2, 1, 0):
        up = h.repeat_interleave(2, 1).repeat_interleave(2, 2)
        h = block(torch.cat([enc[lv], up], 3), "dec%d" % lv)
    w, b = par["head"]
    return torch.view_as_complex((h @ w[:, 0].T + b).contiguous())


def exact(case, seed):
    f = dict(depthmap=_exact_depthmap, batch=_exact_batch, pointcloud=_exact_pointcloud, pls=_exact_pls,
             wrp=_exact_wrp, encode=_exact_encode, conv=_exact_conv, unet=_exact_unet)
    return f[case["kind"]](case, seed)
