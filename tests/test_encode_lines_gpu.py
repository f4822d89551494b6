"""The one-axis SSB encoder and the two-pass phase-only encoder against the
centred 2-D transform form (shift by floor(n/2) on both sides of each
transform, as oh_fft2d's shift does), at odd and even sides, single rows and
columns, ragged strips, and an output written over the field.

Tolerance: the image is min..max scaled, so two FFT roundings of eps log2(n)
relative to the field's RMS show as at most 16 eps log2(n) absolute."""
import ctypes as C
import math

import numpy as np
import pytest
import torch

from openholo_gb300 import _lib

pytestmark = pytest.mark.gpu


def S():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def shift(a):
    return np.roll(a, (a.shape[0] // 2, a.shape[1] // 2), (0, 1))


def ssb(U, kind):
    ny, nx = U.shape
    A = shift(np.fft.fft2(shift(U)))
    c, r = np.arange(nx)[None, :], np.arange(ny)[:, None]
    zero = {5: c >= nx // 2 - 1, 6: c <= nx // 2 - 1, 7: r >= ny // 2 - 1, 8: r <= ny // 2 - 1}[kind]
    re = shift(np.fft.ifft2(shift(np.where(zero, 0, A)))).real
    return (re - re.min()) / (re.max() - re.min())


@pytest.mark.parametrize("ny,nx", [(7, 9), (8, 9), (9, 8), (48, 64), (121, 77), (5, 640), (640, 5), (1080, 1920), (613, 611)])
@pytest.mark.parametrize("kind", [5, 6, 7, 8])
def test_ssb(ctx, ny, nx, kind):
    rng = np.random.default_rng(ny * 1000 + nx)
    U = rng.standard_normal((ny, nx)) + 1j * rng.standard_normal((ny, nx))
    if max(ny, nx) == 613:
        t = torch.from_numpy(U).cuda()              # a prime side above 61 stays refused
        out = torch.empty((ny, nx), dtype=torch.float64, device="cuda")
        with pytest.raises(_lib.OhError):
            _lib.call("oh_encode", ctx.handle, 1, kind, nx, ny, C.c_void_p(t.data_ptr()), C.c_void_p(out.data_ptr()), S())
        return
    ref = ssb(U, kind)
    for prec, cdt, rdt, eps in ((1, torch.complex128, torch.float64, 2.3e-16), (0, torch.complex64, torch.float32, 1.2e-7)):
        tol = 16 * eps * math.log2(max(nx, ny))
        t = torch.from_numpy(U).to(cdt).cuda()
        out = torch.empty((ny, nx), dtype=rdt, device="cuda")
        _lib.call("oh_encode", ctx.handle, prec, kind, nx, ny, C.c_void_p(t.data_ptr()), C.c_void_p(out.data_ptr()), S())
        torch.cuda.synchronize()
        assert np.abs(out.cpu().numpy() - ref).max() <= tol
        _lib.call("oh_encode", ctx.handle, prec, kind, nx, ny, C.c_void_p(t.data_ptr()), C.c_void_p(t.data_ptr()), S())
        torch.cuda.synchronize()
        over = torch.view_as_real(t).reshape(-1)[:ny * nx].reshape(ny, nx)
        assert torch.equal(over, out)


def test_ssb_of_a_nan_is_nan(ctx):
    U = torch.randn(16, 24, dtype=torch.complex64, device="cuda")
    U[3, 5] = float("nan")
    out = torch.empty((16, 24), device="cuda")
    for kind in (5, 6, 7, 8):
        _lib.call("oh_encode", ctx.handle, 0, kind, 24, 16, C.c_void_p(U.data_ptr()), C.c_void_p(out.data_ptr()), S())
        assert bool(torch.isnan(out).all())


@pytest.mark.parametrize("n,offset", [(1, 0), (3, 1), (1021, 0), (4096, 3), (100003, 2)])
def test_phase_only_bytes(ctx, n, offset):
    """Any output alignment gives the same bytes: 255 (angle + pi) / max, halves away from zero."""
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    u = torch.randn(n, generator=g, dtype=torch.complex128, device="cuda")
    out = torch.zeros(n + 8, dtype=torch.uint8, device="cuda")
    _lib.call("oh_encode", ctx.handle, 1, 9, n, 1, C.c_void_p(u.data_ptr()), C.c_void_p(out.data_ptr() + offset), S())
    torch.cuda.synchronize()
    ph = np.angle(u.cpu().numpy()) + np.pi
    v = 255 * ph / ph.max()
    got = out.cpu().numpy()
    ref = np.clip(np.floor(v + 0.5), 0, 255)
    clear = np.abs(v + 0.5 - np.rint(v + 0.5)) > 1e-9
    assert np.array_equal(got[offset:offset + n][clear], ref[clear].astype(np.uint8))
    assert not got[:offset].any() and not got[offset + n:].any()
