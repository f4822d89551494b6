"""Two-float frames where errors could build up: many evenly spaced layers, by the step from
layer to layer against the transfer function of every layer, and phases of several turns
(of the pixels, of the transfer function at fine pitches) against the frame in 64 bits.

Tolerances: a step rounds by 2^-46 in two floats, a random walk over the layers, and its
factor is off by 1e-14, once per layer: 250 layers 2.7e-12.  Phases: 20 turns to 2^-47, and
2 eps of the 1.5e4 radians that the 64-bit reference evaluates whole: 5e-12."""
import numpy as np
import pytest
import torch

from openholo_gb300 import _lib, depthmap, scenes
from oracle import depthmap as odm
from test_fft_generic_gpu import reference

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


@pytest.mark.parametrize("pitch,near", [(8e-6, 0.3), (1.5e-6, 0.02)])
def test_phases_of_several_turns(ctx, pitch, near):
    nx, ny = 128, 96
    kw = dict(pnx=nx, pny=ny, ppx=pitch, ppy=pitch, num_of_depth=6, pad=1, near=near, far=1.1 * near,
              transform_viewing_window=0)
    rng = np.random.default_rng(7)
    img, dep = (rng.integers(1, 256, (ny, nx), dtype=np.uint8) for _ in range(2))
    phase = scenes.seeded_phase(3, ny, nx).astype(np.float32)
    ref, _ = reference(img, dep, odm.DMParams(**kw), phase)
    p = depthmap.make_params(phase_mode=depthmap.OH_PHASE_ARRAY, **kw)
    f = torch.empty((ny, nx), dtype=torch.complex128, device="cuda")
    depthmap.generate(ctx, p, *(torch.from_numpy(v).cuda() for v in (img, dep, phase)), precision="fp64", field=f)
    torch.cuda.synchronize()
    assert np.linalg.norm(f.cpu().numpy() - ref) <= 5e-12 * np.linalg.norm(ref)
