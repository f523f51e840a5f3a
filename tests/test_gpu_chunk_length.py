"""Chunks of a ray are shortened only when more Gaussians are hit than a list holds.  In the fast arithmetic
the chunk sequence decides which samples at a slab's edge count, so it may not depend on how many Gaussians
merely come near a tile: here thousands lie between the rays of one tile, and few are hit."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["parity", "fast"])
def test_near_misses_do_not_shorten_a_chunk(cuda, oracle, mode):
    from ray_gauss_b200 import synthetic as S
    from ray_gauss_b200.batched import BatchedViews, render_views
    from ray_gauss_b200.engine import Engine
    n, w, h = 3000, 8, 4
    rng = np.random.default_rng(3)
    p, _, _ = S.workload("small_object", n=n, seed=5)
    pos = rng.uniform(-1.0, 1.0, (n, 3)) * [0.6, 0.04, 0.3]
    p["positions"] = torch.as_tensor(pos, dtype=torch.float32)
    p["scales"] = torch.full((n, 3), 4e-3)
    cam = S.look_at_camera([0.0, -2.0, 0.0], [0.0, 0.0, 0.0], w, h, fovx=math.radians(40.0), device=cuda)
    cv = oracle.camera_vector(cam)
    N = {k: v.numpy() for k, v in p.items()}
    eng = Engine()
    eng.set_tuning(list_capacity=128)          # whole tiles
    img = render_views({k: v.to(cuda) for k, v in p.items()}, BatchedViews([cam], mode=mode, engine=eng)).cpu().numpy()
    st = eng.status()
    assert st["hit_pairs"] > 0
    assert st["chunk_splits"] == 0
    rgb = oracle.forward_sh(cv[:3], N["positions"], N["color_features"], None, None, None)
    ref, _, _ = oracle.render_forward(N["positions"], N["scales"], N["quaternions"], N["densities"], rgb, cv, w, h, True)
    assert np.abs(img - ref).max() <= {"parity": 1e-4, "fast": 5e-4}[mode]
