"""Discs two thousand times as wide as thick, far from the camera: the traversal's cone test has to keep every
leaf that a ray hits although rounding is large against their thickness.  Against the oracle, images and
gradients, in both arithmetics and all tile layouts.

Tolerances.  Parity images: the drop-in's 1e-4.  A point 50 units away is rounded to 3e-6, which is a hundredth
of the threshold ellipsoid's half-thickness (1e-3): the fast samples' densities (2 at most) are off by a few per
cent of themselves, and a sample of 0.0025 that falls on the other side of the threshold 0.1 counts 2.5e-4; four
of those, 1e-3.  Gradients of the densities, sums over the same rounded points: 2e-2.  (Those of scales and
rotations say nothing here: the second moments of a disc that reaches 2.4 units are rounded to 6e-8 of 5, and
divided by its squared thickness that is a tenth or more of the gradient, whichever leaves are listed.)"""
import math

import numpy as np
import pytest
import torch

from helpers import rel_l2
from test_gpu_tile_split import _Rays

pytestmark = pytest.mark.gpu
W, H, N = 48, 32, 600


@pytest.mark.parametrize("split", [1, 2, 4])
@pytest.mark.parametrize("mode", ["parity", "fast"])
def test_flat_gaussians_against_oracle(cuda, oracle, mode, split):
    from ray_gauss_b200 import synthetic as S
    from ray_gauss_b200.batched import BatchedViews, _st
    from ray_gauss_b200.engine import Engine, make_gaussians
    rng = np.random.default_rng(17)
    p, _, white = S.workload("small_object", n=N, seed=2)
    p["positions"] = torch.as_tensor(rng.uniform(-6.0, 6.0, (N, 3)), dtype=torch.float32)
    p["scales"] = torch.as_tensor(np.array([5e-4, 1.0, 1.0]) * rng.uniform(0.7, 1.0, (N, 3)), dtype=torch.float32)
    p["densities"] = torch.as_tensor(rng.uniform(0.5, 2.0, N), dtype=torch.float32).reshape(p["densities"].shape)
    cam = S.look_at_camera([50.0, 0.0, 1.0], [0.0, 0.0, 0.0], W, H, fovx=math.radians(22.0), device=cuda)
    P = {k: v.to(cuda).contiguous() for k, v in p.items()}
    Q = {k: v.numpy() for k, v in p.items()}
    views = BatchedViews([cam], mode=mode)
    eng = Engine()
    # x = 1000 Gaussians / tiles^2 decides (render_split): below, between and above its lines
    eng.lib = _Rays(eng.lib, {1: 0, 2: 32 * int(math.sqrt(1000.0 * N / 15.0)), 4: 32}[split])
    g = make_gaussians(P["positions"], P["scales"], P["quaternions"], P["densities"], P["color_features"])
    cams_t, _, _ = eng.cameras([cam])
    img, _ = eng.render_forward(g, cams_t, 1, W * H, _st(views))
    cv = oracle.camera_vector(cam)
    rgb = oracle.forward_sh(cv[:3], Q["positions"], Q["color_features"], None, None, None)
    args = (Q["positions"], Q["scales"], Q["quaternions"], Q["densities"], rgb, cv, W, H)
    want, _, _ = oracle.render_forward(*args, white)
    assert np.abs(img.cpu().numpy() - want).max() <= {"parity": 1e-4, "fast": 1e-3}[mode]
    dL = torch.randn(img.shape, device=cuda, generator=torch.Generator(device=cuda).manual_seed(4)) * 1e-4
    gr = eng.render_backward(g, cams_t, 1, _st(views), img, dL)
    b = oracle.render_backward(*args, want, dL.cpu().numpy())
    assert rel_l2(gr["densities"].cpu().numpy(), b["d_dens"]) <= 2e-2
