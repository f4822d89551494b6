"""The plan-driven FFT engine and the depth-map passes on it, at the lengths
where they branch: every straight-line radix as the only, first and last stage,
primes that run the loop, padded (even last radix) and unpadded layouts, the
longest lines; frames with odd padded grids, single rows and columns, and the
column pass's many-samples variant.

Tolerances: an n-point FFT's rounding error grows like eps log2(n); 2 eps
log2(n) (at least four eps) relative L2 covers both precisions.  Frames: 1e-9 in
FP64, 1e-5 in FP32.  The reference cancels the carrier exp(i k z') against the
constant part of the transfer function analytically: the product of the two,
each rounded at 6e6 rad, is itself off by about 1e-9."""
import ctypes as C
import math

import numpy as np
import pytest
import torch

from openholo_gb300 import _lib, depthmap as dm, scenes
from oracle import depthmap as odm

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16, 17, 61, 34, 121, 128, 143, 196, 255, 256, 289, 512,
           819, 1000, 1155, 1638, 2310, 4096, 4320, 5632, 7680, 8192, 9216, 11024]


@pytest.mark.parametrize("n", LENGTHS)
def test_row_lines(ctx, n):
    rng = np.random.default_rng(n)
    rows = 5
    x = rng.standard_normal((rows, n)) + 1j * rng.standard_normal((rows, n))
    for prec, dt, eps in ((1, torch.complex128, 2.3e-16), (0, torch.complex64, 1.2e-7)):
        t = torch.from_numpy(x).to(dt).cuda()
        out = torch.empty_like(t)
        for direction, ref in ((-1, np.fft.fft(x)), (1, np.fft.ifft(x) * n)):
            _lib.call("oh_fft1d_rows", ctx.handle, prec, n, rows, C.c_void_p(t.data_ptr()), C.c_void_p(out.data_ptr()),
                      direction, 0, C.c_void_p(torch.cuda.current_stream().cuda_stream))
            torch.cuda.synchronize()
            err = np.linalg.norm(out.cpu().numpy() - ref) / np.linalg.norm(ref)
            assert err <= 2 * eps * max(math.log2(n), 2), (prec, direction, err)


def reference(img, depth, op, phase):
    """Oracle frame with U_e = FFT(layer) exp(2 pi i (z'/lambda) s / (1 + sqrt(1 - s)))."""
    ny, nx = img.shape
    Px, Py = op.pad * nx, op.pad * ny
    ox, oy = (Px - nx) // 2, (Py - ny) // 2
    idx, src, zt = odm.depth_lut(op)[depth], odm.source_field(img, phase), odm.transformed_levels(op)
    fx = -1.0 / (2 * op.ppx) + np.arange(Px) / (Px * op.ppx)
    fy = 1.0 / (2 * op.ppy) - (1.0 + np.arange(Py)) / (Py * op.ppy)
    s = (op.lam * fx[None, :]) ** 2 + (op.lam * fy[:, None]) ** 2
    spec = np.zeros((Py, Px), np.complex128)
    for d in range(1, op.num_of_depth + 1):
        u = np.zeros((Py, Px), np.complex128)
        u[oy:oy + ny, ox:ox + nx] = np.where(idx == d, src, 0)
        t = zt[d - 1] / op.lam * s / (1 + np.sqrt(1 - s))
        spec += np.exp(2j * np.pi * (t - np.rint(t))) * odm.centred_fft2(u)
    return odm.encode_symmetrization(spec, op, return_field=True)[1], spec


FRAMES = [(1, 1, 1), (1, 9, 1), (9, 1, 2), (13, 7, 1), (121, 77, 1), (63, 55, 2), (34, 61, 2), (16, 4116, 2),
          (8, 1400, 2), (1400, 8, 2), (256, 128, 1)]


@pytest.mark.parametrize("nx,ny,pad", FRAMES)
@pytest.mark.parametrize("window,sig", [(0, (0, 1)), (1, (1, 0))])
def test_frames(ctx, dev, nx, ny, pad, window, sig):
    layers = 5
    rng = np.random.default_rng(nx * 10000 + ny)
    img = rng.integers(0, 256, (ny, nx), dtype=np.uint8)
    depth = rng.integers(0, 256, (ny, nx), dtype=np.uint8)
    depth[(depth > 100) & (depth < 160)] = 0            # a level without pixels
    phase = scenes.seeded_phase(3, ny, nx)
    p = dm.make_params(pnx=nx, pny=ny, num_of_depth=layers, pad=pad, phase_mode=dm.OH_PHASE_ARRAY,
                       transform_viewing_window=window, sig_location=sig)
    op = odm.DMParams(pnx=nx, pny=ny, num_of_depth=layers, pad=pad, transform_viewing_window=window, sig_location=sig)
    field, spec = reference(img, depth, op, phase)
    ti, td, tp = (torch.from_numpy(v).to(dev) for v in (img, depth, phase))
    for prec, dt, tol in (("fp64", torch.complex128, 1e-9), ("fp32", torch.complex64, 1e-5)):
        # with and without the spectrum (which keeps every row of the columns)
        f = torch.empty((ny, nx), dtype=dt, device=dev)
        s = torch.empty((pad * ny, pad * nx), dtype=dt, device=dev)
        for spectrum in (None, s):
            dm.generate(ctx, p, ti, td, tp, precision=prec, field=f, spectrum=spectrum)
            torch.cuda.synchronize()
            scale = max(np.linalg.norm(field), 1e-3 * np.linalg.norm(spec) / math.sqrt(spec.size))
            assert np.linalg.norm(f.cpu().numpy() - field) <= tol * scale, prec
        assert np.linalg.norm(s.cpu().numpy() - spec) <= tol * np.linalg.norm(spec), prec
