"""A field with an infinity encodes to NaN everywhere, as with a NaN, on lines of any length
(the two-dimensional transforms of the SSB encoding spread it over the image)."""
import ctypes as C

import pytest
import torch

from openholo_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("ny,nx", [(14, 2), (2, 14), (9, 1), (1, 9), (5, 4), (4, 5), (7, 3), (3, 8), (1, 1)])
def test_ssb_of_an_infinity(ctx, prec, ny, nx):
    u = torch.randn(ny, nx, dtype=torch.complex128, device="cuda").to(torch.complex128 if prec else torch.complex64)
    out = torch.empty((ny, nx), dtype=torch.float64 if prec else torch.float32, device="cuda")
    for at, v in ((0, complex(float("inf"), 0)), (nx * ny // 2, complex(float("-inf"), 1)), (nx * ny - 1, complex(0, float("inf")))):
        f = u.clone()
        f.view(-1)[at] = v
        for kind in (5, 6, 7, 8):
            _lib.call("oh_encode", ctx.handle, prec, kind, nx, ny, C.c_void_p(f.data_ptr()), C.c_void_p(out.data_ptr()),
                      C.c_void_p(torch.cuda.current_stream().cuda_stream))
            assert not bool(torch.isfinite(out).any()), (kind, at)
