"""The engine tells the library how many rays a launch has, from colours of any shape."""
import contextlib

import pytest
import torch

from ray_gauss_b200 import engine as E


class _Lib:
    def __init__(self):
        self.rays = []

    def rg_expect_rays(self, h, n):
        self.rays.append(n)
        return 0

    def __getattr__(self, name):
        return lambda *a: 0


@pytest.mark.parametrize("shape", [(35, 3), (5, 7, 3), (105,)])
def test_rays_of_colours_in_any_shape(monkeypatch, shape):
    monkeypatch.setattr(E, "_stream", lambda dev: None)
    eng = E.Engine.__new__(E.Engine)
    eng.lib, eng.h, eng.device, eng.timers = _Lib(), None, torch.device("cpu"), None
    eng._timed = lambda name: contextlib.nullcontext()
    s = E.settings_struct()
    colors, cams = torch.zeros(shape), torch.zeros(1, dtype=torch.uint8)
    eng.launch_forward(cams, 1, s, colors)
    eng.launch_backward(cams, 1, s, colors, torch.zeros(shape))
    eng.launch_inference(cams, 1, s, colors)
    assert eng.lib.rays == [35, 35, 35]
