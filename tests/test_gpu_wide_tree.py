"""Wide nodes of the LBVH at the sizes where their collapse can go wrong (a node that is just full, one
unit too many, chains of one leaf per level, equal Morton codes), built and refitted, against the
oracle.  The bound is the drop-in's image bound."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
IMG_TOL = 1e-4


def _cloud(layout, n):
    from ray_gauss_b200 import synthetic as S
    p, _, _ = S.workload("small_object", n=n, seed=n)
    p["scales"] = p["scales"] * (2.0 if n > 500 else 5.0)
    if layout == "chain":      # one leaf splits off per level of the binary tree
        k = torch.arange(n, dtype=torch.float32) % 19
        p["positions"] = (2.0 ** -k)[:, None] * torch.tensor([0.9, 0.7, 0.5]) * torch.sign(p["positions"])
    elif layout == "equal":    # many equal centres: ties broken by index
        p["positions"] = torch.round(p["positions"] * 1.5) * 0.5
    return {k: v.contiguous() for k, v in p.items()}


@pytest.mark.parametrize("layout", ["uniform", "chain", "equal"])
@pytest.mark.parametrize("n", [2, 32, 33, 63, 65, 1024, 1025])
def test_wide_nodes_against_oracle(cuda, oracle, n, layout):
    from ray_gauss_b200 import synthetic as S
    from ray_gauss_b200.batched import BatchedViews, render_views
    from ray_gauss_b200.engine import Engine
    p = _cloud(layout, n)
    cam = S.sphere_camera(3.0, 24, 20, 40.0, seed=n, device=cuda)
    cv = oracle.camera_vector(cam)
    eng = Engine()
    for update in (False, True):
        if update:             # other positions in the tree of the first build
            p["positions"] = (p["positions"].flip(0) * 0.9).contiguous()
        P = {k: v.to(cuda).contiguous() for k, v in p.items()}
        N = {k: v.numpy() for k, v in p.items()}
        img = render_views(P, BatchedViews([cam], mode="parity", engine=eng, update=update)).cpu().numpy()
        rgb = oracle.forward_sh(cv[:3], N["positions"], N["color_features"], None, None, None)
        ref, _, _ = oracle.render_forward(N["positions"], N["scales"], N["quaternions"], N["densities"], rgb, cv, 24, 20,
                                          True)
        assert np.abs(img - ref).max() <= IMG_TOL
        st = eng.status(reset=True)
        assert st["stack_overflows"] == 0 and st["watchdog_trips"] == 0
