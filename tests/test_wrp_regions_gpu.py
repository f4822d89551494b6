"""The tensor-core form of the fixed-window WRP sum over its overlapping regions:
windows of one pixel up to half a region (one bin per point), wider ones (every
region they touch), planes of odd width (no vector reductions) and smaller than a
region, one point and several stages of points in a cell, centres off the plane.

Tolerance: the form's own bounds (cross terms of 3e-5 rad at a window's corner,
BF16 high and low parts without their low product), 5e-5 as a sum."""
import numpy as np
import pytest

from openholo_gb300 import scenes
from oracle import pointcloud as opc
from test_encode_wrp_gpu import _wrp_run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,gap", [(1, 5e-3), (16, 5e-3), (31, 8e-3), (32, -8e-3), (33, 8e-3), (64, 2e-2), (70, -3e-2)])
@pytest.mark.parametrize("nx,ny,npts", [(320, 200, 600), (255, 131, 1), (40, 301, 65)])
def test_regions(ctx, w, gap, nx, ny, npts):
    dp, lam = 3.74e-6, 532e-9
    pts = scenes.wrp_scene(7, npts, box=(nx * 4.2e-6, ny * 4.2e-6, 1e-3), zc=0.1)
    z = 0.1 - 0.5e-3 - gap if gap > 0 else 0.1 + 0.5e-3 - gap
    ran = set()
    got = _wrp_run(ctx, pts, nx, ny, dp, lam, z, w, kernels=ran)
    assert "wrp_tc" in ran
    ref = opc.wrp_f64(pts, nx, ny, dp, lam, z, w)
    assert np.linalg.norm(got - ref) <= 5e-5 * np.linalg.norm(ref)
