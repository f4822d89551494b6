"""FP64 depth-map frames on either side of the rule that takes them to two-float
arithmetic, over what its kernels branch on: short and wide columns, odd and even
grids, evenly spaced layers by the step and by the per-layer transfer function,
phases inside and beyond the short reduction, a distance below the rule's.

Tolerance: the reference and the tables round propagation phases of up to 3e3
turns in FP64, 2e4 rad x 2 eps = 5e-12; twice that."""
import math

import numpy as np
import pytest
import torch

from openholo_gb300 import depthmap as dm, scenes
from oracle import depthmap as odm
from test_fft_generic_gpu import reference

pytestmark = pytest.mark.gpu

CASES = [(1, 1, 1, 1.0, 1.0), (64, 48, 2, 1.0, 1.0), (121, 77, 1, 1.0, 1.0), (63, 55, 2, 1000.0, 1.0),
         (8, 1400, 2, 1.0, 1.0), (1400, 8, 1, 1.0, 1.0), (64, 48, 2, 1.0, 0.005), (360, 270, 1, 6.0, 0.1)]


@pytest.mark.parametrize("nx,ny,pad,pscale,zscale", CASES)
@pytest.mark.parametrize("step", ["1", "0"])
def test_fp64_frames(ctx, dev, monkeypatch, nx, ny, pad, pscale, zscale, step):
    monkeypatch.setenv("OH_DM_LAYER_STEP", step)
    rng = np.random.default_rng(nx * 10000 + ny)
    img = rng.integers(0, 256, (ny, nx), dtype=np.uint8)
    depth = rng.integers(0, 256, (ny, nx), dtype=np.uint8)
    depth[(depth > 100) & (depth < 160)] = 0
    phase = (scenes.seeded_phase(3, ny, nx) * np.float32(pscale)).astype(np.float32)
    kw = dict(pnx=nx, pny=ny, num_of_depth=6, pad=pad, near=0.8 * zscale, far=1.0 * zscale,
              transform_viewing_window=0)
    field, spec = reference(img, depth, odm.DMParams(**kw), phase)
    ti, td, tp = (torch.from_numpy(v).to(dev) for v in (img, depth, phase))
    f = torch.empty((ny, nx), dtype=torch.complex128, device=dev)
    s = torch.empty((pad * ny, pad * nx), dtype=torch.complex128, device=dev)
    p = dm.make_params(phase_mode=dm.OH_PHASE_ARRAY, **kw)
    for spectrum in (None, s):
        dm.generate(ctx, p, ti, td, tp, precision="fp64", field=f, spectrum=spectrum)
        torch.cuda.synchronize()
        scale = max(np.linalg.norm(field), 1e-3 * np.linalg.norm(spec) / math.sqrt(spec.size))
        assert np.linalg.norm(f.cpu().numpy() - field) <= 1e-11 * scale
    assert np.linalg.norm(s.cpu().numpy() - spec) <= 1e-11 * np.linalg.norm(spec)
