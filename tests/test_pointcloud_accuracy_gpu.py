"""The point-cloud sum where its tensor-core forms are weakest, against a sum in
64 bits (r / lambda as z / lambda, reduced in extended precision, plus rho^2 / (r +
z) / lambda): the corners of planes whose cross phase is as large as the form
takes, sums that stay in phase over a whole chunk of points, clouds of uneven
amplitude, and small clouds, where the direct sum loses least.

Each tolerance is the form's own error, derived beside its test; none is larger
than the error of the direct sum at the same sizes."""
import ctypes as C

import numpy as np
import pytest
import torch

from openholo_gb300 import _lib

pytestmark = pytest.mark.gpu
LAM = 532e-9


def run(ctx, prec, pts, nx, ny, pitch=8e-6):
    p = _lib.PcParams(1.0, 1.0, 1.0, 0.0, pitch, pitch, nx, ny, LAM, 0.0, 0.0)
    t = torch.from_numpy(pts).cuda()
    out = torch.full((ny, nx), 9.0, dtype=torch.complex128 if prec else torch.complex64, device="cuda")
    _lib.call("oh_pointcloud", ctx.handle, prec, C.byref(p), C.c_void_p(t.data_ptr()), len(pts),
              C.c_void_p(out.data_ptr()), None, C.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    return out


def reference(pts, nx, ny, rows, pitch=8e-6):
    d = torch.float64
    z0 = pts[:, 2].astype(np.longdouble) / np.longdouble(LAM)
    t0 = torch.from_numpy((z0 - np.rint(z0)).astype(np.float64)).cuda()
    x, y, z, a = (torch.from_numpy(pts[:, i].astype(np.float64)).cuda() for i in range(4))
    X = (torch.arange(nx, device="cuda", dtype=d) + 0.5) * pitch - nx * pitch / 2
    Y = ny * pitch / 2 - (torch.tensor(rows, device="cuda", dtype=d) + 0.5) * pitch
    out = torch.zeros((len(rows), nx), dtype=torch.complex128, device="cuda")
    per = max(1, int(1e8 // out.numel()))
    for j in range(0, len(pts), per):
        s = slice(j, j + per)
        rho2 = (X[None, None, :] - x[s, None, None]) ** 2 + (Y[None, :, None] - y[s, None, None]) ** 2
        t = rho2 / (torch.sqrt(rho2 + (z * z)[s, None, None]) + z[s, None, None]) / LAM
        t = (t - torch.round(t)) + t0[s, None, None]
        t = 2 * np.pi * (t - torch.round(t))
        am = a[s, None, None]
        out += torch.complex((am * torch.cos(t)).sum(0), (am * torch.sin(t)).sum(0))
    return out


def cloud(n, seed, amp=None, scale=1.0):
    """x, y in +-2 mm, z in 0.10-0.12 m (times scale); amplitudes `amp`, or 0-1."""
    u = np.random.default_rng(seed).random((n, 4))
    return np.stack([(u[:, 0] - 0.5) * 4e-3 * scale, (u[:, 1] - 0.5) * 4e-3 * scale, (0.10 + 0.02 * u[:, 2]) * scale,
                     u[:, 3] if amp is None else amp], 1).astype(np.float32)


def off(got, ref):
    """Error of rows in the L2 norm, and the largest error over the largest value."""
    e = (got - ref).abs()
    return float(e.norm() / ref.abs().norm()), float(e.max() / ref.abs().max())


def rows_of(ny):
    return sorted({0, 1, ny // 5, ny // 3, ny // 2, ny - 2, ny - 1})


@pytest.mark.parametrize("nx,ny", [(1920, 1080), (1024, 1024), (1500, 700)])
def test_fp64_corners(ctx, nx, ny):
    """Per point at most 1.2e-10 of the six-term form, 1e-11 of two-float arithmetic;
    points beyond it go through the direct sum (3e-10 at these distances)."""
    n = 40
    pts = cloud(n, nx + ny, np.ones(n))
    rows = rows_of(ny)
    assert float((run(ctx, 1, pts, nx, ny)[rows] - reference(pts, nx, ny, rows)).abs().max()) <= n * 3e-10


@pytest.mark.parametrize("nx,ny,n", [(1920, 1080, 32768), (256, 256, 5000), (1024, 1024, 20000)])
def test_fp32_sums_in_phase(ctx, nx, ny, n):
    """One point n times over, whole chunks of it in one block where the plane fills the
    SMs.  One term is off by up to 2e-6 (operands 2^-21 each way, sine and cosine);
    the sum is taken in n / 224 FP32 additions of 2^-25 each on average."""
    pts = np.tile(cloud(1, 3, np.ones(1)), (n, 1))
    rows = rows_of(ny)
    rel, mx = off(run(ctx, 0, pts, nx, ny)[rows], reference(pts, nx, ny, rows))
    tol = 2e-6 + (n / 224 + 8) * 2.0 ** -25
    assert rel <= tol and mx <= 2 * tol


def uneven(kind, n):
    rng = np.random.default_rng(n)
    if kind == "bright":
        return np.where(np.arange(n) == n // 2, 1.0, 0.01)
    if kind == "two_levels":
        return np.where(np.arange(n) % 50 == 7, 1.0, 2e-3)
    return np.exp(2.0 * rng.standard_normal(n))


@pytest.mark.parametrize("kind,n,nx,ny", [("bright", 10001, 640, 480), ("bright", 2500, 300, 200),
                                          ("two_levels", 6000, 300, 200), ("lognormal", 5000, 640, 480),
                                          ("lognormal", 33000, 130, 129)])
def test_uneven_amplitudes(ctx, kind, n, nx, ny):
    """A point's operands are off by 2^-22 of its group's scale, and a group's scales add
    up to at most sqrt(8) of the sum's L2 norm: 6e-7, with the rest below 2e-6.  FP64: 1e-11."""
    pts = cloud(n, n, uneven(kind, n))
    rows = rows_of(ny)
    ref = reference(pts, nx, ny, rows)
    assert off(run(ctx, 0, pts, nx, ny)[rows], ref)[0] <= 2e-6
    assert off(run(ctx, 1, pts, nx, ny)[rows], ref)[0] <= 1e-11


@pytest.mark.parametrize("n,nx,ny,pitch,scale", [(200, 300, 300, 8e-6, 1.0), (200, 300, 300, 2e-6, 1.0), (40, 1024, 700, 8e-6, 1.0),
                                                 (1000, 257, 131, 8e-6, 1.0), (600, 300, 300, 8e-7, 0.1),
                                                 (500, 640, 480, 2e-5, 10.0)])
def test_fp32_small_clouds(ctx, n, nx, ny, pitch, scale):
    """The direct FP32 sum is 3e-7 off for a few hundred points.  Three-part operands
    (2^-25), phases of 2^-25 turns and a sine and cosine of 2^-23 leave 2e-7."""
    pts = cloud(n, n + nx, None, scale)
    rows = rows_of(ny)
    assert off(run(ctx, 0, pts, nx, ny, pitch)[rows], reference(pts, nx, ny, rows, pitch))[0] <= 3e-7
