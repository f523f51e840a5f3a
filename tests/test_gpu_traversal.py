"""The traversal's leaf culling and its shortened chunks, in both tile layouts, where they can go wrong: wide and narrow tile
cones, a camera inside Gaussians, needles, far and dense clusters that overfill a long chunk or a
single slab.  Parity images equal the oracle's within the drop-in's image bound; the fast
arithmetic, whose samples differ by rounding, is held to its own bound on small scenes (5e-4)."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
TOL = {"parity": 1e-4, "fast": 5e-4}


def _scene(kind):
    from ray_gauss_b200 import synthetic as S
    rng = np.random.default_rng(11)
    n = 12000 if kind in ("dense", "far_dense") else 800
    p, _, _ = S.workload("small_object", n=n, seed=5)
    eye, fov = [0.0, -3.0, 0.4], 40.0
    if kind == "needles":
        p["scales"] = torch.exp(torch.as_tensor(rng.normal(math.log(0.02), 1.2, (n, 3)), dtype=torch.float32))
    elif kind == "inside":
        p["scales"] = p["scales"] * 8.0
        eye, fov = [0.1, 0.05, 0.0], 110.0
    elif kind == "dense":          # hundreds of Gaussians in a slab: several passes
        p["positions"] = p["positions"] * 0.12
    elif kind == "far_dense":      # a long empty way, then a cluster: a 64-slab chunk overfills
        p["positions"] = p["positions"] * 0.25
        p["positions"][:6] = p["positions"][:6] * 200.0
        eye, fov = [0.0, -30.0, 0.5], 2.0
    p["densities"] = p["densities"] * (0.2 if "dense" in kind else 1.0)
    return {k: v.contiguous() for k, v in p.items()}, eye, fov


# a launch this small runs on split tiles with the list capacity of 64, on whole ones with 128
@pytest.mark.parametrize("capacity", [64, 128])
@pytest.mark.parametrize("mode", ["parity", "fast"])
@pytest.mark.parametrize("kind", ["needles", "inside", "dense", "far_dense"])
def test_traversal_against_oracle(cuda, oracle, kind, mode, capacity):
    from ray_gauss_b200 import synthetic as S
    from ray_gauss_b200.batched import BatchedViews, render_views
    from ray_gauss_b200.engine import Engine
    p, eye, fov = _scene(kind)
    w, h = 35, 22
    cam = S.look_at_camera(eye, [0.0, 0.0, 0.0], w, h, fovx=math.radians(fov), device=cuda)
    cv = oracle.camera_vector(cam)
    N = {k: v.numpy() for k, v in p.items()}
    P = {k: v.to(cuda) for k, v in p.items()}
    eng = Engine()
    eng.set_tuning(list_capacity=capacity)
    img = render_views(P, BatchedViews([cam], mode=mode, engine=eng)).cpu().numpy()
    rgb = oracle.forward_sh(cv[:3], N["positions"], N["color_features"], None, None, None)
    ref, _, _ = oracle.render_forward(N["positions"], N["scales"], N["quaternions"], N["densities"], rgb, cv, w, h, True)
    assert np.abs(img - ref).max() <= TOL[mode]
    st = eng.status()
    assert st["stack_overflows"] == 0 and st["watchdog_trips"] == 0
    if kind == "far_dense":
        assert st["chunk_splits"] > 0
