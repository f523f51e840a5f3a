"""The tile layout (1, 2 or 4 slabs of a ray side by side) is chosen by sizes and may not show in the results:
images and Gaussians per ray are the same bit for bit, gradients up to the order of the atomic sums (2e-5
relative L2, the bound of an FP32 output), in both arithmetics, with the hit lists replayed or traversed again,
in short and long scene boxes, and where a slab holds more Gaussians than a list."""
import math

import pytest
import torch

from helpers import rel_l2
from test_gpu_tile_split import _Rays

pytestmark = pytest.mark.gpu


def _scene(kind, cuda):
    from ray_gauss_b200 import synthetic as S
    n = 6000 if kind == "dense" else 1500
    p, _, _ = S.workload("small_object", n=n, seed=7)
    eye, w, h = [2.5, 1.0, 0.6], 93, 61
    p["scales"] = p["scales"] * 3.0
    if kind == "far":
        p["positions"][:60] = p["positions"][:60] * 25.0
    elif kind == "dense":
        p["positions"] = p["positions"] * 0.12
        p["densities"] = p["densities"] * 0.2
        eye, w, h = [0.0, -1.5, 0.1], 27, 19
    cams = [S.look_at_camera(e, [0.0, 0.0, 0.0], w + 3 * i, h, fovx=math.radians(40.0), device=cuda)
            for i, e in enumerate((eye, [-eye[1], eye[0], 0.3]))]
    return {k: v.to(cuda).contiguous() for k, v in p.items()}, cams


@pytest.mark.parametrize("record", [1, -1])
@pytest.mark.parametrize("kind", ["box", "far", "dense"])
@pytest.mark.parametrize("mode", ["parity", "fast"])
def test_layouts_agree(cuda, mode, kind, record):
    from ray_gauss_b200.batched import BatchedViews, _st
    from ray_gauss_b200.engine import Engine, make_gaussians
    P, cams = _scene(kind, cuda)
    views = BatchedViews(cams, mode=mode)
    g = make_gaussians(P["positions"], P["scales"], P["quaternions"], P["densities"], P["color_features"])
    n = P["positions"].shape[0]
    dL = torch.randn((views.n_rays, 3), device=cuda, generator=torch.Generator(device=cuda).manual_seed(4)) * 1e-4
    # x = 1000 Gaussians views / tiles^2 decides (render_split): above every line, or between the two lines
    line = 15.0 if kind == "far" else 1.0
    got = {}
    for split, rays in ((1, 0), (2, 32 * int(math.sqrt(2000.0 * n / line))), (4, 32)):
        eng = Engine()
        eng.set_tuning(record_hits=record)
        eng.lib = _Rays(eng.lib, rays)
        cams_t, _, _ = eng.cameras(cams)
        img, _ = eng.render_forward(g, cams_t, 2, views.n_rays, _st(views))
        gr = eng.render_backward(g, cams_t, 2, _st(views), img, dL)
        frame, counts = eng.render_inference(g, cams_t, 2, views.n_rays, _st(views), counts=True)
        got[split] = img, gr, frame, counts
        if kind == "dense" and split == 1:
            assert eng.status()["list_passes"] > 0
    for split in (2, 4):
        assert torch.equal(got[split][0], got[1][0])
        assert torch.equal(got[split][2], got[1][2])
        assert torch.equal(got[split][3], got[1][3])
        for k, ref in got[1][1].items():
            if ref is not None:
                assert rel_l2(got[split][1][k].cpu().numpy(), ref.cpu().numpy()) <= 2e-5, (split, k)
