"""A point-cloud call whose tensor-core form finds no memory for its partial planes
runs the direct sum, which needs none of them."""
import ctypes as C

import numpy as np
import pytest
import torch

from openholo_gb300 import Context, _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1])
def test_no_room_for_partial_planes(lib_built, prec):
    nx = ny = 16384
    p = _lib.PcParams(1.0, 1.0, 1.0, 0.0, 2e-7, 2e-7, nx, ny, 532e-9, 0.0, 0.0)
    pts = torch.tensor([[0.0, 0.0, 0.1, 1.0], [1e-4, 2e-4, 0.11, 0.5]], device="cuda")
    torch.cuda.empty_cache()
    fringe = torch.zeros((ny, nx), dtype=torch.float64 if prec else torch.float32, device="cuda")
    part = nx * ny * (16 if prec else 8)
    ctx = Context(0)
    free, _ = torch.cuda.mem_get_info()
    filler = torch.empty(free - part // 2, dtype=torch.uint8, device="cuda")    # half a plane is left
    try:
        _lib.call("oh_pointcloud", ctx.handle, prec, C.byref(p), C.c_void_p(pts.data_ptr()), 2, None,
                  C.c_void_p(fringe.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
    finally:
        del filler
        ctx.close()
        torch.cuda.empty_cache()
    q = pts.cpu().numpy().astype(np.float64)
    for r, c in ((0, 0), (8000, 9000), (16383, 5)):
        X, Y = (c + 0.5) * 2e-7 - nx * 1e-7, ny * 1e-7 - (r + 0.5) * 2e-7
        ref = sum(a * np.cos(2 * np.pi / 532e-9 * np.sqrt((X - x) ** 2 + (Y - y) ** 2 + z * z)) for x, y, z, a in q)
        assert abs(float(fringe[r, c]) - ref) <= (1e-8 if prec else 1e-4)
