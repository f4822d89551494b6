"""The tensor-core form of the fixed-window WRP sum where several blocks share a
region's points (small planes, many points), and at the windows on both sides of
the change from one bin per point to every region touched.

Tolerance: the form's own bounds, 5e-5 as a sum (see test_wrp_regions_gpu.py)."""
import numpy as np
import pytest

from openholo_gb300 import scenes
from oracle import pointcloud as opc
from test_encode_wrp_gpu import _wrp_run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,gap", [(20, 5e-3), (34, 8e-3), (48, 1e-2), (49, 1e-2)])
@pytest.mark.parametrize("nx,ny,npts", [(120, 90, 3001), (255, 131, 127), (33, 300, 1100)])
def test_parts(ctx, w, gap, nx, ny, npts):
    dp, lam = 3.74e-6, 532e-9
    pts = scenes.wrp_scene(11, npts, box=(nx * 4.2e-6, ny * 4.2e-6, 1e-3), zc=0.1)
    z = 0.1 - 0.5e-3 - gap
    ran = set()
    got = _wrp_run(ctx, pts, nx, ny, dp, lam, z, w, kernels=ran)
    assert "wrp_tc" in ran
    ref = opc.wrp_f64(pts, nx, ny, dp, lam, z, w)
    assert np.linalg.norm(got - ref) <= 5e-5 * np.linalg.norm(ref)
