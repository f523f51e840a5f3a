"""Which tile layout a launch runs on: the lines of render_split in short and long scene boxes, where only the device
knows which of two kernels it is, and the callers that stay on whole tiles.  Launches in long boxes are compared
with whole tiles bit for bit as well, replayed and traversed."""
import math

import pytest
import torch

from test_gpu_tile_split import _Rays

pytestmark = pytest.mark.gpu
N = 1500


def _launch(cuda, mode, far, x, record=1, rnd_sample=0, capacity=64):
    from ray_gauss_b200 import synthetic as S
    from ray_gauss_b200.batched import BatchedViews, _st
    from ray_gauss_b200.engine import Engine, make_gaussians
    p, _, _ = S.workload("small_object", n=N, seed=7)
    p["scales"] = p["scales"] * 3.0
    if far:
        p["positions"][:60] = p["positions"][:60] * 25.0
    cam = S.look_at_camera([2.5, 1.0, 0.6], [0.0, 0.0, 0.0], 61, 43, fovx=math.radians(40.0), device=cuda)
    P = {k: v.to(cuda).contiguous() for k, v in p.items()}
    views = BatchedViews([cam], mode=mode, rnd_sample=rnd_sample)
    eng = Engine()
    eng.set_tuning(record_hits=record, list_capacity=capacity)
    # x = 1000 Gaussians views / tiles^2 decides
    eng.lib = _Rays(eng.lib, 32 * int(math.sqrt(1000.0 * N / x)) if x else 0)
    g = make_gaussians(P["positions"], P["scales"], P["quaternions"], P["densities"], P["color_features"])
    cams_t, _, _ = eng.cameras([cam])
    img, _ = eng.render_forward(g, cams_t, 1, views.n_rays, _st(views))
    layout = eng.tile_layout()
    gr = eng.render_backward(g, cams_t, 1, _st(views), img, torch.full_like(img, 1e-4))
    assert eng.tile_layout() == layout
    return layout, img, gr


@pytest.mark.parametrize("mode,far,x,layout", [
    ("fast", False, 0.1, 1), ("fast", False, 1.0, 2), ("fast", False, 5.0, 4),
    ("fast", True, 1.0, 1), ("fast", True, 15.0, 2), ("fast", True, 90.0, 4),
    ("parity", False, 0.1, 1), ("parity", False, 0.5, 2), ("parity", False, 5.0, 4),
    ("parity", True, 1.0, 1), ("parity", True, 15.0, 2), ("parity", True, 90.0, 4)])
@pytest.mark.parametrize("record", [1, -1])
def test_layout_of_a_launch(cuda, mode, far, x, layout, record):
    got, img, gr = _launch(cuda, mode, far, x, record)
    assert got == layout
    whole, ref, gr0 = _launch(cuda, mode, far, 0, record)
    assert whole == 1 and torch.equal(img, ref)
    for k in ("positions", "scales", "quaternions", "densities", "color_features"):
        d = (gr[k].double() - gr0[k].double()).norm() / gr0[k].double().norm()
        assert d <= 2e-5, k          # the order of the atomic sums


@pytest.mark.parametrize("change", [dict(rnd_sample=1), dict(capacity=128)])
def test_launches_that_stay_whole(cuda, change):
    assert _launch(cuda, "parity", False, 50.0, **change)[0] == 1
