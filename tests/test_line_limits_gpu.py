"""Lines that fill a block's shared memory to within the kernels' own few hundred
bytes: SSB encodings along such a side, and FP64 depth-map frames whose column
pass does (its step factors included)."""
import ctypes as C

import numpy as np
import pytest
import torch

from openholo_gb300 import _lib, depthmap, scenes
from oracle import depthmap as odm
from test_fft_generic_gpu import reference

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


@pytest.mark.parametrize("pny,layers,near,far", [(9120, 168, 0.30, 0.35), (9116, 216, 0.30, 0.35), (9212, 40, 1e-4, 2e-4),
                                                 (9204, 136, 1e-4, 2e-4)])
def test_fp64_column_at_the_limit(ctx, pny, layers, near, far):
    """Against the frame in 64 bits (itself good to 1e-11): the step between layers, 2e-13
    off in two floats, is taken once per layer."""
    pnx = 16
    kw = dict(pnx=pnx, pny=pny, num_of_depth=layers, pad=1, near=near, far=far, transform_viewing_window=0)
    rng = np.random.default_rng(pny)
    img = rng.integers(1, 256, (pny, pnx), dtype=np.uint8)
    dep = rng.integers(0, 256, (pny, pnx), dtype=np.uint8)
    phase = scenes.seeded_phase(3, pny, pnx).astype(np.float32)
    ref, _ = reference(img, dep, odm.DMParams(**kw), phase)
    p = depthmap.make_params(phase_mode=depthmap.OH_PHASE_ARRAY, **kw)
    f = torch.empty((pny, pnx), dtype=torch.complex128, device="cuda")
    depthmap.generate(ctx, p, *(torch.from_numpy(v).cuda() for v in (img, dep, phase)), precision="fp64", field=f)
    torch.cuda.synchronize()
    assert np.linalg.norm(f.cpu().numpy() - ref) <= (1e-11 + layers * 2e-13) * np.linalg.norm(ref)
