"""FP32 clouds about the size up to which one block forms and sorts the points: all
refused by the separable form (then the sum is the direct one, bit for bit), half
of them, none.

Tolerance of the mixed sum: each form is 3e-7 off at these counts, 1e-6 in all."""
import ctypes as C

import numpy as np
import pytest
import torch

from openholo_gb300 import _lib

pytestmark = pytest.mark.gpu
NX, NY = 256, 300
PAR = _lib.PcParams(1.0, 1.0, 1.0, 0.0, 8e-6, 8e-6, NX, NY, 532e-9, 0.0, 0.0)


def total(ctx, pts, direct=False):
    t = torch.from_numpy(np.ascontiguousarray(pts)).cuda()
    out = torch.full((NY, NX), 9.0, dtype=torch.complex64, device="cuda")
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    if direct:
        _lib.call("oh_pointcloud_noalloc", C.byref(PAR), C.c_void_p(t.data_ptr()), len(pts), C.c_void_p(out.data_ptr()),
                  None, st)
    else:
        _lib.call("oh_pointcloud", ctx.handle, 0, C.byref(PAR), C.c_void_p(t.data_ptr()), len(pts),
                  C.c_void_p(out.data_ptr()), None, st)
    torch.cuda.synchronize()
    return out


def cloud(n):
    u = np.random.default_rng(n).random((n, 4))
    return np.stack([(u[:, 0] - 0.5) * 4e-3, (u[:, 1] - 0.5) * 4e-3, 0.10 + 0.02 * u[:, 2], u[:, 3]], 1).astype(np.float32)


@pytest.mark.parametrize("n", [300, 1000, 1024, 1025, 2100])
def test_refused(ctx, n):
    pts = cloud(n)
    near = pts.copy()
    near[:, 2] *= 0.02                      # 2 mm away: not separable over a region
    assert torch.equal(total(ctx, near), total(ctx, near, direct=True))
    mixed = np.where(np.arange(n)[:, None] % 3 == 1, near, pts)
    want = total(ctx, near[1::3], direct=True).to(torch.complex128)
    for k in (0, 2):
        want += total(ctx, pts[k::3], direct=True)
    got = total(ctx, mixed)
    assert float((got - want).norm()) <= 1e-6 * float(want.norm())
