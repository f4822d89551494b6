"""The FP64 point-cloud sum on the tensor cores: plane sizes that end inside a
region, splits, groups and chunks of the points, points the separable form
refuses beside the others, identical points (sums that stay in phase), tilt,
amplitude scales, the fringe, and the same bits on every run.

The reference sums exp(2 pi i r / lambda) in 64 bits with r / lambda as z / lambda
(reduced in extended precision) plus rho^2 / (r + z) / lambda, good to 1e-13; the
plain k r in 64 bits is itself off by 1e-10.  Tolerance: two-float operands and
exact products leave about 2e-12, the seventh term of the cross phase less on
average: 1e-11 of the L2 norm.  Refused points go through the plain form: 1e-9."""
import ctypes as C

import numpy as np
import pytest
import torch

from openholo_gb300 import _lib

pytestmark = pytest.mark.gpu
TOL, PITCH, LAM = 1e-11, 8e-6, 532e-9


def run(ctx, nx, ny, pts, tilt=(0.0, 0.0), fringe=None):
    p = _lib.PcParams(1.0, 1.0, 1.0, 0.0, PITCH, PITCH, nx, ny, LAM, *tilt)
    t = torch.from_numpy(pts).cuda()
    out = torch.full((ny, nx), 9.0, dtype=torch.complex128, device="cuda")
    _lib.call("oh_pointcloud", ctx.handle, 1, C.byref(p), C.c_void_p(t.data_ptr()), pts.shape[0],
              C.c_void_p(out.data_ptr()), C.c_void_p(fringe.data_ptr()) if fringe is not None else None,
              C.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    return out


def reference(nx, ny, pts, tilt=(0.0, 0.0)):
    """The whole plane on the GPU."""
    d = torch.float64
    z0 = pts[:, 2].astype(np.longdouble) / np.longdouble(LAM)
    t0 = torch.from_numpy((z0 - np.rint(z0)).astype(np.float64)).cuda()
    x, y, z, a = (torch.from_numpy(pts[:, i].astype(np.float64)).cuda() for i in range(4))
    X = (torch.arange(nx, device="cuda", dtype=d) + 0.5) * PITCH - nx * PITCH / 2
    Y = ny * PITCH / 2 - (torch.arange(ny, device="cuda", dtype=d) + 0.5) * PITCH
    ref = (X * np.sin(np.radians(tilt[0])))[None, :] / LAM + (Y * np.sin(np.radians(tilt[1])))[:, None] / LAM
    out = torch.zeros((ny, nx), dtype=torch.complex128, device="cuda")
    per = max(1, int(2e7 // out.numel()))
    for j in range(0, len(pts), per):
        s = slice(j, j + per)
        rho2 = (X[None, None, :] - x[s, None, None]) ** 2 + (Y[None, :, None] - y[s, None, None]) ** 2
        zz = z[s, None, None]
        t = rho2 / (torch.sqrt(rho2 + zz * zz) + zz) / LAM - ref
        t = (t - torch.round(t)) + t0[s, None, None]
        out += torch.sum(torch.polar(a[s, None, None].expand_as(t).contiguous(), 2 * np.pi * (t - torch.round(t))), 0)
    return out


def cloud(n, seed, amp=1.0):
    u = np.random.default_rng(seed).random((n, 4))
    return np.stack([(u[:, 0] - 0.5) * 4e-3, (u[:, 1] - 0.5) * 4e-3, 0.10 + 0.02 * u[:, 2], amp * u[:, 3]], 1).astype(
        np.float32)


def check(ctx, nx, ny, pts, tilt=(0.0, 0.0), tol=TOL):
    got, ref = run(ctx, nx, ny, pts, tilt), reference(nx, ny, pts, tilt)
    assert float((got - ref).norm()) <= tol * float(ref.norm())
    return got


@pytest.mark.parametrize("nx,ny,n", [(64, 128, 300), (65, 129, 97), (1, 700, 1000), (700, 1, 1000), (257, 131, 2007),
                                     (127, 300, 96), (127, 300, 101), (31, 40, 33000), (1024, 1024, 150),
                                     (1024, 1024, 20)])
def test_sizes(ctx, nx, ny, n):
    check(ctx, nx, ny, cloud(n, nx + ny))


def test_tilt_and_amplitude_scale(ctx):
    for amp, tilt in ((3e8, (1.5, -0.7)), (1e-12, (0.0, 2.0))):
        check(ctx, 200, 160, cloud(700, 5, amp), tilt)


def test_sums_in_phase(ctx):
    """One point 3000 times over: every product of a group has the same sign."""
    pts = np.tile(cloud(1, 3), (3000, 1))
    pts[:, 3] = 1.0
    check(ctx, 128, 128, pts)


def test_refused_points_are_summed_directly(ctx):
    pts = cloud(900, 9)
    pts[::7, 2] *= 0.02
    pts[3::11, 0] += 0.3
    check(ctx, 256, 128, pts, tol=1e-9)
    pts = cloud(900, 10)
    pts[:, 3] = 0.0
    assert not bool(run(ctx, 256, 128, pts).abs().any())
    pts[5, 0] = np.nan
    assert bool(torch.isnan(run(ctx, 256, 128, pts).real).all())


def test_fringe_accumulates_and_runs_repeat(ctx):
    pts = cloud(1500, 2)
    a = check(ctx, 320, 200, pts)
    fr = torch.full((200, 320), 2.5, dtype=torch.float64, device="cuda")
    b = run(ctx, 320, 200, pts, fringe=fr)
    assert torch.equal(a, b)
    assert bool(torch.allclose(fr, 2.5 + a.real, rtol=1e-14, atol=1e-12))
