"""SSB encodings along sides whose line fills a block's shared memory to within a few
hundred bytes."""
import ctypes as C

import numpy as np
import pytest
import torch

from openholo_gb300 import _lib

pytestmark = pytest.mark.gpu


def S():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("prec,n", [(1, 14500), (1, 14520), (0, 29036), (0, 29040), (1, 14400)])
@pytest.mark.parametrize("kind", [5, 8])
def test_ssb_of_the_longest_lines(ctx, prec, n, kind):
    """16 eps log2(n) of the scaled image, as at other lengths."""
    m = 3
    ny, nx = (m, n) if kind == 5 else (n, m)
    rng = np.random.default_rng(n)
    U = rng.standard_normal((ny, nx)) + 1j * rng.standard_normal((ny, nx))

    def shift(a):
        return np.roll(a, (a.shape[0] // 2, a.shape[1] // 2), (0, 1))

    A = shift(np.fft.fft2(shift(U)))
    zero = (np.arange(nx) >= nx // 2 - 1)[None, :] if kind == 5 else (np.arange(ny) <= ny // 2 - 1)[:, None]
    re = shift(np.fft.ifft2(shift(np.where(zero, 0, A)))).real
    ref = (re - re.min()) / (re.max() - re.min())
    u = torch.from_numpy(U).cuda().to(torch.complex128 if prec else torch.complex64)
    out = torch.empty((ny, nx), dtype=torch.float64 if prec else torch.float32, device="cuda")
    _lib.call("oh_encode", ctx.handle, prec, kind, nx, ny, C.c_void_p(u.data_ptr()), C.c_void_p(out.data_ptr()), S())
    torch.cuda.synchronize()
    assert np.abs(out.cpu().numpy() - ref).max() <= 16 * (2.3e-16 if prec else 1.2e-7) * np.log2(n)
