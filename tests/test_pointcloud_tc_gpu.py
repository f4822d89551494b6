"""The point-cloud sum on the tensor cores against the FP64 oracle: plane sizes
that end inside a region, odd rows, splits and chunks of the points, points the
separable form refuses (near, off-axis, not finite) beside the others, the
fringe's accumulation, tilt, amplitudes of any scale, and the same bits on every
run.

Tolerance: operands carry 22 bits and the sines an absolute 5e-7, independent
from term to term, so the sum is off by less than 2e-6 of its L2 norm.  Refused
points go through the direct FP32 sum, whose contract is 1e-3."""
import ctypes as C

import numpy as np
import pytest
import torch

from openholo_gb300 import _lib
from oracle import pointcloud as opc

pytestmark = pytest.mark.gpu
TOL = 2e-6


def spec(nx, ny, tilt=(0.0, 0.0)):
    return dict(scale_x=1.0, scale_y=1.0, scale_z=1.0, offset_depth=0.0, pitch_x=8e-6, pitch_y=8e-6, nx=nx, ny=ny,
                tilt_x=tilt[0], tilt_y=tilt[1], **{"lambda": 532e-9})


def run(ctx, s, pts, fringe=None):
    p = _lib.PcParams(1.0, 1.0, 1.0, 0.0, s["pitch_x"], s["pitch_y"], s["nx"], s["ny"], s["lambda"], s["tilt_x"],
                      s["tilt_y"])
    t = torch.from_numpy(pts).cuda()
    out = torch.full((s["ny"], s["nx"]), 9.0, dtype=torch.complex64, device="cuda")
    _lib.call("oh_pointcloud", ctx.handle, 0, C.byref(p), C.c_void_p(t.data_ptr()), pts.shape[0],
              C.c_void_p(out.data_ptr()), C.c_void_p(fringe.data_ptr()) if fringe is not None else None,
              C.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    return out.cpu().numpy()


def cloud(n, seed, amp=1.0):
    rng = np.random.default_rng(seed)
    u = rng.random((n, 4))
    return np.stack([(u[:, 0] - 0.5) * 4e-3, (u[:, 1] - 0.5) * 4e-3, 0.10 + 0.02 * u[:, 2], amp * u[:, 3]], 1).astype(
        np.float32)


def check(ctx, s, pts, rows=24, tol=TOL):
    got = run(ctx, s, pts)
    for r0 in sorted({0, max(0, s["ny"] // 2 - rows // 2), max(0, s["ny"] - rows)}):
        n = min(rows, s["ny"] - r0)
        ref = opc.pc_f64(pts.astype(np.float64), s, r0, n)
        band = ref[r0:r0 + n] if ref.shape[0] == s["ny"] else ref[:n]
        assert np.linalg.norm(got[r0:r0 + n] - band) <= tol * np.linalg.norm(band)
    return got


@pytest.mark.parametrize("nx,ny,n", [(64, 128, 25000), (65, 129, 24001), (1, 2000, 100003), (2000, 1, 100003),
                                     (257, 131, 6007), (127, 300, 33000), (1024, 768, 257)])
def test_sizes(ctx, nx, ny, n):
    check(ctx, spec(nx, ny), cloud(n, nx + ny))


def test_tilt_and_amplitude_scale(ctx):
    for amp, tilt in ((3e8, (1.5, -0.7)), (1e-12, (0.0, 2.0))):
        check(ctx, spec(200, 160, tilt), cloud(7000, 5, amp))


def test_refused_points_are_summed_directly(ctx):
    s = spec(256, 128)
    pts = cloud(6500, 9)
    pts[::7, 2] *= 0.02                     # 2 mm away: not separable over a region
    pts[3::11, 0] += 0.3                    # far off axis
    check(ctx, s, pts, tol=1e-3)
    pts[:, 2] *= 0.02                       # all of them
    check(ctx, s, pts, tol=1e-3)
    pts = cloud(6500, 10)
    pts[:, 3] = 0.0                         # nothing to sum
    assert not run(ctx, s, pts).any()
    pts = cloud(6500, 11)
    pts[17, 3] = np.inf
    assert not np.isfinite(run(ctx, s, pts)).any()


def test_fringe_accumulates_and_runs_repeat(ctx):
    s = spec(320, 200)
    pts = cloud(5000, 2)
    a = check(ctx, s, pts)
    fr = torch.full((200, 320), 2.5, device="cuda")
    b = run(ctx, s, pts, fr)
    assert np.array_equal(a, b)
    assert np.allclose(fr.cpu().numpy(), 2.5 + a.real, rtol=1e-6, atol=1e-4)
