"""2-D transforms on the plan's engine whose blocks have few lines or are few: one
column a block (odd widths), a handful of blocks, rows much shorter than a block,
single rows and columns.

Tolerance: 2 eps log2(nx ny) relative L2 for a transform's rounding."""
import ctypes as C
import math

import numpy as np
import pytest
import torch

from openholo_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(1, 4000), (4000, 1), (3, 700), (6, 900), (100, 100), (121, 31), (31, 121), (625, 49),
                                   (37, 1763), (512, 640), (2187, 125), (300, 1080)])
@pytest.mark.parametrize("shift", [0, 1])
def test_fft2d(ctx, nx, ny, shift):
    rng = np.random.default_rng(nx * 7919 + ny)
    x = rng.standard_normal((ny, nx)) + 1j * rng.standard_normal((ny, nx))
    roll = lambda a: np.roll(a, (ny // 2, nx // 2), (0, 1)) if shift else a  # noqa: E731
    ref = roll(np.fft.fft2(roll(x)))
    for prec, dt, eps in ((1, torch.complex128, 2.3e-16), (0, torch.complex64, 1.2e-7)):
        t = torch.from_numpy(x).to(dt).cuda()
        _lib.call("oh_fft2d", ctx.handle, prec, nx, ny, C.c_void_p(t.data_ptr()), C.c_void_p(t.data_ptr()), -1, shift, 0,
                  C.c_void_p(torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        assert np.linalg.norm(t.cpu().numpy() - ref) <= 2 * eps * math.log2(nx * ny) * np.linalg.norm(ref)
