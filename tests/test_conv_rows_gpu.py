"""3x3 convolutions over whole 128-pixel rows in tiles of several output rows:
heights below, at and past a tile's rows, widths past one and two tiles, channel
counts with resident and with streamed weights, every channel tile; forward and,
with a mask, input gradient, against the float64 oracle on the same BF16 inputs.

Tolerance: products are exact, sums FP32, outputs rounded to BF16 (2^-9 relative
each): 6e-3 relative L2."""
import numpy as np
import pytest
import torch

from openholo_gb300 import _lib
from oracle import unet as U
from test_unet_conv_gpu import P, S, bf16, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,w,cin,cout", [(1, 1, 128, 32, 32), (2, 2, 137, 32, 64), (1, 37, 160, 64, 96),
                                            (2, 50, 128, 192, 64), (1, 40, 256, 320, 128), (1, 33, 128, 96, 192),
                                            (1, 70, 300, 32, 32), (1, 301, 128, 32, 32), (1, 5, 128, 512, 256),
                                            (3, 130, 256, 64, 32), (1, 19, 129, 256, 160)])
def test_rows(ctx, n, h, w, cin, cout):
    rng = np.random.default_rng(h * 1000 + cin + cout)
    x, dz = bf16(rng, (n, h, w, cin + 8)), bf16(rng, (n, h, w, cin))
    W = bf16(rng, (cout, 9 * cin), (2.0 / (9 * cin)) ** 0.5)
    b = torch.from_numpy(rng.standard_normal(cout).astype(np.float32) * 0.1).cuda()
    mask = bf16(rng, (n, h, w, cout))
    y = torch.full((n, h, w, cout + 8), 7.0, dtype=torch.bfloat16, device="cuda")
    dx = torch.empty((n, h, w, cout), dtype=torch.bfloat16, device="cuda")
    _lib.call("oh_conv2d_bf16", ctx.handle, 9, 1, n, h, w, cin, cout, P(x), cin + 8, P(W), P(b), 1, None, 0, P(y),
              cout + 8, S())
    _lib.call("oh_conv2d_bf16", ctx.handle, 9, -1, n, h, w, cin, cout, P(dz), cin, P(W), None, 0, P(mask), cout, P(dx),
              cout, S())
    torch.cuda.synchronize()
    Wn = W.float().cpu().numpy().astype(np.float64).reshape(cout, 9, cin)
    ref = U.conv(x.float().cpu().numpy()[..., :cin].astype(np.float64), Wn, b.cpu().numpy().astype(np.float64),
                 relu=True)
    got = y.float().cpu().numpy()
    assert rel(got[..., :cout], ref) < 6e-3
    assert np.all(got[..., cout:] == 7.0)
    ref = U.conv_dgrad(dz.float().cpu().numpy().astype(np.float64), Wn.transpose(2, 1, 0))
    assert rel(dx.float().cpu().numpy(), ref * (mask.float().cpu().numpy() > 0)) < 6e-3
