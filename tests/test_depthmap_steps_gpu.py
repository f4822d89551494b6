"""FP64 frames of many evenly spaced layers: the step from layer to layer against the
transfer function of every layer.

Tolerance: a step rounds by 2^-46 in two floats, a random walk over the layers, and its
factor is off by 1e-14, once per layer: 250 layers 2.7e-12."""
import numpy as np
import pytest
import torch

from openholo_gb300 import _lib, depthmap

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,layers,pad", [(64, 384, 250, 1), (48, 500, 120, 2), (33, 2000, 168, 1)])
def test_many_layers(ctx, monkeypatch, nx, ny, layers, pad):
    p = depthmap.make_params(pnx=nx, pny=ny, num_of_depth=layers, pad=pad, phase_mode=_lib.OH_PHASE_SEEDED, seed=5)
    rng = np.random.default_rng(layers)
    img = torch.from_numpy(rng.integers(1, 256, (ny, nx), dtype=np.uint8)).cuda()
    dep = torch.from_numpy(rng.integers(0, 256, (ny, nx), dtype=np.uint8)).cuda()
    out = []
    for step in ("1", "0"):
        monkeypatch.setenv("OH_DM_LAYER_STEP", step)
        out.append(depthmap.generate(ctx, p, img, dep, precision="fp64"))
    torch.cuda.synchronize()
    assert float((out[0] - out[1]).norm()) <= 2.7e-12 * float(out[1].norm())
