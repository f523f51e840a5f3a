"""The 3D filter's camera table for image sizes in other kinds of numbers, alone and side by side: a size held in
32 or 16 bits is multiplied in that precision (a row per camera, as the reference's loop has it,
classes/point_cloud.py:1153-1215), and matrices of several types are converted one by one."""
import types

import numpy as np
import pytest
import torch

from ray_gauss_b200.filter3d import camera_table
from test_filter3d_cameras import _row

SIZES = {"int": 801, "float": 801.0, "int16": np.int16(801), "float32": np.float32(801), "float16": np.float16(801),
         "array32": np.asarray(801, np.float32), "tensor": torch.tensor(801), "tensor32": torch.tensor(801.0)}


def _cam(size, wvt=None):
    return types.SimpleNamespace(world_view_transform=torch.eye(4) if wvt is None else wvt, FoVx=1.1, FoVy=0.9,
                                 image_width=size, image_height=size)


@pytest.mark.parametrize("first", SIZES)
def test_sizes_in_any_kind_of_number(first):
    for second in SIZES:
        cams = [_cam(SIZES[first]), _cam(SIZES[second])]
        table, _ = camera_table(cams)
        assert np.array_equal(table, np.stack([_row(c) for c in cams])), second


def test_matrices_of_several_types():
    g = torch.Generator().manual_seed(1)
    cams = [_cam(801, torch.randint(0, 2 ** 30, (4, 4), generator=g)), _cam(801, torch.randn(4, 4, generator=g).half())]
    assert np.array_equal(camera_table(cams)[0], np.stack([_row(c) for c in cams]))
