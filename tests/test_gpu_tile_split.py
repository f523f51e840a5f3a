"""The render kernels' tile layouts (1, 2 or 4 slabs of a ray side by side) on the same launch: images and
gradients against the FP32 oracle, with the drop-in's bounds (parity images 1e-4, gradients 1e-3
relative L2; fast images 5e-4 on small scenes), at a ragged image size, several views, few and many
slabs per ray, and with the hit lists replayed or traversed again."""
import math

import numpy as np
import pytest
import torch

from helpers import rel_l2

pytestmark = pytest.mark.gpu
TOL = {"parity": 1e-4, "fast": 5e-4}
W, H = 37, 23


class _Rays:
    """The engine library with another number of expected rays (which chooses the layout)."""

    def __init__(self, lib, rays):
        self._lib, self._rays = lib, rays

    def __getattr__(self, name):
        if name == "rg_expect_rays":
            return lambda h, n: self._lib.rg_expect_rays(h, self._rays)
        return getattr(self._lib, name)


@pytest.mark.parametrize("record", [1, -1])
@pytest.mark.parametrize("split", [1, 2, 4, "far"])
@pytest.mark.parametrize("mode", ["parity", "fast"])
def test_layouts_against_oracle(cuda, oracle, mode, split, record):
    from ray_gauss_b200 import synthetic as S
    from ray_gauss_b200.batched import BatchedViews, _st
    from ray_gauss_b200.engine import Engine, make_gaussians
    p, _, white = S.workload("small_object", n=1500, seed=2)
    p["scales"] = p["scales"] * 3.0
    if split == "far":        # a long scene box: of the two kernels that are launched, the other one runs
        p["positions"][:3] = p["positions"][:3] * 25.0
    cams = [S.look_at_camera(e, [0.0, 0.0, 0.0], W + 5 * i, H, fovx=math.radians(40.0), device=cuda)
            for i, e in enumerate(([2.5, 1.0, 0.6], [0.3, -2.8, 0.2]))]
    P = {k: v.to(cuda).contiguous() for k, v in p.items()}
    N = {k: v.numpy() for k, v in p.items()}
    views = BatchedViews(cams, mode=mode)
    eng = Engine()
    eng.set_tuning(record_hits=record)
    eng.lib = _Rays(eng.lib, {1: 0, 2: 3000 * 32, 4: views.n_rays, "far": 3000 * 32}[split])
    g = make_gaussians(P["positions"], P["scales"], P["quaternions"], P["densities"], P["color_features"])
    cams_t, _, _ = eng.cameras(cams)
    img, _ = eng.render_forward(g, cams_t, 2, views.n_rays, _st(views))
    dL = torch.randn(img.shape, device=cuda, generator=torch.Generator(device=cuda).manual_seed(4)) * 1e-4
    gr = eng.render_backward(g, cams_t, 2, _st(views), img, dL)
    st = eng.status()
    assert (st["replayed_chunks"] > 0) == (record == 1)
    ref = {k: 0.0 for k in ("positions", "scales", "quaternions", "densities", "color_features")}
    for v, cam in enumerate(cams):
        lo, hi = views.offsets[v], views.offsets[v + 1]
        cv = oracle.camera_vector(cam)
        rgb = oracle.forward_sh(cv[:3], N["positions"], N["color_features"], None, None, None)
        args = (N["positions"], N["scales"], N["quaternions"], N["densities"], rgb, cv, cam.image_width, cam.image_height)
        want, _, _ = oracle.render_forward(*args, white)
        assert np.abs(img[lo:hi].cpu().numpy() - want).max() <= TOL[mode]
        b = oracle.render_backward(*args, want, dL[lo:hi].cpu().numpy())
        dsh, dpos, _, _, _ = oracle.backward_sh(cv[:3], N["positions"], N["color_features"], None, None, None,
                                                b["d_rgb"].astype(np.float32), ref_quirks=True)
        for k, d in (("positions", b["d_pos"] + dpos), ("scales", b["d_scl"]), ("quaternions", b["d_quat"]),
                     ("densities", b["d_dens"]), ("color_features", dsh)):
            ref[k] = ref[k] + d
    for k, d in ref.items():
        assert rel_l2(gr[k].cpu().numpy(), d) <= 1e-3, k
