"""The 3D filter's camera table, gathered for all cameras at once, against a row per camera
(``PointCloud.compute_3D_filter``, classes/point_cloud.py:1153-1215), over the forms that cameras come in."""
import types

import numpy as np
import pytest
import torch

from ray_gauss_b200.filter3d import camera_table, fov2focal


def _row(cam):
    wvt = cam.world_view_transform.detach().to("cpu", torch.float32).numpy()
    W, H = cam.image_width, cam.image_height
    row = np.empty(20, np.float32)
    row[0:9] = wvt[:3, :3].reshape(-1)
    row[9:12] = wvt[3, :3]
    row[12:20] = [fov2focal(cam.FoVx, W), fov2focal(cam.FoVy, H), W / 2.0, H / 2.0, -0.15 * W, W * 1.15,
                  -0.15 * H, 1.15 * H]
    return row


@pytest.mark.parametrize("number", [float, np.float32, np.asarray, torch.tensor])
@pytest.mark.parametrize("matrices", ["alike", "transposed", "types", "shapes"])
def test_rows_equal_those_of_single_cameras(number, matrices):
    g = torch.Generator().manual_seed(5)
    cams = []
    for i in range(7):
        wvt = torch.randn(4, 4, generator=g)
        if matrices == "transposed":
            wvt = wvt.t()
        elif matrices == "types":
            wvt = wvt.to((torch.float32, torch.float64, torch.float16)[i % 3])
        elif matrices == "shapes" and i % 2:
            wvt = wvt[:, :3]
        cams.append(types.SimpleNamespace(world_view_transform=wvt.requires_grad_(i == 3), FoVx=number(0.6 + 0.1 * (i // 3)),
                                          FoVy=number(0.5), image_width=640 + i % 2, image_height=480))
    table, focal = camera_table(cams)
    assert table.dtype == np.float32
    assert np.array_equal(table, np.stack([_row(c) for c in cams]))
    assert focal == max(max(fov2focal(c.FoVx, c.image_width), fov2focal(c.FoVy, c.image_height)) for c in cams)
