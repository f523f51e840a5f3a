"""The workloads this framework's speed is judged on, through its public entry points.

listed() names the cases, draw(rng) gives one more of the same ranges, prepare(case, seed) makes what a
program holds before the call, run(state) is one pass, work(case) the bytes and operations the pass
cannot do without, exact(case, seed) its result in 64-bit arithmetic.

Scenes have the layouts and value distributions of ray_gauss_b200/synthetic.py, generated on the GPU:
  box      Gaussians uniform in [-1, 1]^3 (an object of a few thousand Gaussians)
  shells   Gaussians on 8 spheres and ellipsoid shells (a bounded object)
  ball     80 % in the unit ball, 20 % at log-uniform radius 1-50 (an unbounded scene)
"""
import copy
import math

import numpy as np
import torch

from ray_gauss_b200.batched import BatchedRenderFunction, BatchedViews, render_views_inference
from ray_gauss_b200.densify import densify_and_prune
from ray_gauss_b200.engine import Engine
from ray_gauss_b200.filter3d import compute_3D_filter
from ray_gauss_b200.graph import GraphedStep
from ray_gauss_b200.knn import initial_log_scales
from ray_gauss_b200.optix_raycasting.render_optix import RenderOptixFunction, RenderOptixSettings
from ray_gauss_b200.synthetic import look_at_camera
from ray_gauss_b200.train_tail import FusedTrainTail, LrSchedule

KEYS = ("positions", "scales", "quaternions", "densities", "color_features", "sph_gauss_features",
        "bandwidth_sharpness", "lobe_axis")
SH = {"sh0": 1, "sh1": 4, "sh2": 9, "sh3": 16}


def listed():
    return [
        # a training iteration of the drop-in renderer on a small object: launches and latency
        dict(name="object_step_small", kind="step", scene="box", n=10_000, sh="sh3", nsg=0, views=1, width=200,
             height=200, form="dropin", storage="f32"),
        # the same on a bounded object of ordinary size with SH and spherical Gaussians, odd image size
        dict(name="object_step", kind="step", scene="shells", n=300_000, sh="sh3", nsg=8, views=1, width=797,
             height=801, form="dropin", storage="f32"),
        # a batched training step on a few small uneven views in FP32 storage
        dict(name="views_step_ragged", kind="step", scene="shells", n=60_000, sh="sh2", nsg=3, views=3, width=317,
             height=211, form="batched", storage="f32"),
        # the headline: 16 views of an unbounded scene, BF16 storage
        dict(name="views_step_1m", kind="step", scene="ball", n=1_000_000, sh="sh3", nsg=8, views=16, width=1000,
             height=750, form="batched", storage="bf16"),
        # the largest: 3M Gaussians, 4 views at 1920x1080, FP32
        dict(name="views_step_3m", kind="step", scene="ball", n=3_000_000, sh="sh3", nsg=8, views=4, width=1920,
             height=1080, form="batched", storage="f32"),
        # a captured training step (LBVH refit, forward, loss, backward) of a small scene, replayed
        dict(name="graph_step_small", kind="graph", scene="box", n=20_000, sh="sh1", nsg=0, views=2, width=160,
             height=120, form="batched", storage="f32"),
        # evaluation of a bounded object in the reference's arithmetic, with the Gaussians per ray
        dict(name="eval_object", kind="infer", scene="shells", n=100_000, sh="sh3", nsg=8, views=1, width=641,
             height=479, form="parity", counts=True, storage="f32"),
        # a viewer's frame of an unbounded scene, BF16 storage
        dict(name="viewer_frame_1m", kind="infer", scene="ball", n=1_000_000, sh="sh3", nsg=8, views=1, width=1280,
             height=720, form="fast", counts=False, storage="bf16"),
        # the end of a training iteration: Adam, densification statistics and clamps
        dict(name="tail_1m", kind="tail", n=1_000_000, sh="sh3", nsg=8),
        # densification of a growing cloud
        dict(name="densify_300k", kind="densify", n=300_000, sh="sh3", nsg=8),
        # the minimum-size filter over the training cameras
        dict(name="filter_500k", kind="filter", n=500_000, cams=100),
        # initial scales of a point cloud
        dict(name="scales_200k", kind="scales", n=200_001),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "infer", "infer", "graph", "tail", "densify", "filter",
                       "scales"])
    if kind == "tail":
        return dict(kind=kind, n=_log(rng, 10_000, 1_000_000), sh=rng.choice(["sh1", "sh3"]), nsg=rng.choice([0, 3, 8]))
    if kind == "densify":
        return dict(kind=kind, n=_log(rng, 20_000, 700_000), sh=rng.choice(["sh1", "sh3"]), nsg=rng.choice([0, 8]))
    if kind == "filter":
        return dict(kind=kind, n=_log(rng, 20_000, 1_000_000), cams=_log(rng, 20, 300))
    if kind == "scales":
        return dict(kind=kind, n=_log(rng, 10_000, 1_000_000))
    sh, nsg = rng.choice(["sh0", "sh1", "sh2", "sh3", "sh3"]), rng.choice([0, 0, 3, 8])
    if kind == "graph":
        w = _log(rng, 80, 320)
        return dict(kind=kind, scene=rng.choice(["box", "shells"]), n=_log(rng, 5_000, 50_000), sh=sh, nsg=nsg,
                    views=rng.randint(1, 4), width=w, height=int(w * rng.uniform(0.6, 1.0)), form="batched",
                    storage="f32")
    w = _log(rng, 120, 1280)
    h = int(w * rng.uniform(0.55, 1.0))
    if kind == "infer":
        form = rng.choice(["parity", "fast"])
        return dict(kind=kind, scene=rng.choice(["box", "shells", "ball"]), n=_log(rng, 10_000, 1_000_000), sh=sh, nsg=nsg,
                    views=1, width=w, height=h, form=form, counts=form == "parity" and rng.random() < 0.5,
                    storage=rng.choice(["f32", "bf16"]))
    form = rng.choice(["dropin", "batched"])
    if form == "dropin":
        w, h = min(w, 800), min(h, 800)
        return dict(kind=kind, scene=rng.choice(["box", "shells"]), n=_log(rng, 5_000, 300_000), sh=sh, nsg=nsg, views=1,
                    width=w, height=h, form=form, storage="f32")
    return dict(kind=kind, scene=rng.choice(["shells", "ball", "ball"]), n=_log(rng, 20_000, 1_000_000), sh=sh, nsg=nsg,
                views=rng.randint(2, max(2, min(12, 6_000_000 // (w * h)))), width=w, height=h, form=form,
                storage=rng.choice(["f32", "bf16"]))


# ---- inputs -----------------------------------------------------------------------------------------

def _dev():
    return torch.device("cuda", torch.cuda.current_device())


def _gen(seed):
    return torch.Generator(device=_dev()).manual_seed(int(seed))


def _unit(g, n, d):
    v = torch.randn((n, d), generator=g, device=_dev())
    return v / v.norm(dim=1, keepdim=True)


def _points(kind, n, g):
    """Positions, log scales and raw densities of a scene layout."""
    dev = _dev()
    rand = lambda *s: torch.rand(s, generator=g, device=dev)     # noqa: E731
    randn = lambda *s: torch.randn(s, generator=g, device=dev)   # noqa: E731
    if kind == "box":
        return (2 * rand(n, 3) - 1, math.log(0.02) + 0.3 * randn(n, 3),
                torch.nn.functional.softplus(randn(n)))
    if kind == "shells":
        ctr, rad = 1.8 * rand(8, 3) - 0.9, 0.2 + 0.4 * rand(8, 3)
        rad[::2] = rad[::2, :1]
        which = torch.randint(0, 8, (n,), generator=g, device=dev)
        pos = (ctr[which] + _unit(g, n, 3) * rad[which]).clamp_(-1.5, 1.5)
        return pos, math.log(0.01) + 0.4 * randn(n, 3), randn(n).exp_()
    n_in = int(round(0.8 * n))
    r = torch.cat([rand(n_in) ** (1.0 / 3.0), torch.exp(rand(n - n_in) * math.log(50.0))])
    perm = torch.randperm(n, generator=g, device=dev)
    r = r[perm]
    pos = _unit(g, n, 3) * r[:, None]
    return pos, math.log(0.015) + 0.5 * randn(n, 3) + r.clamp_min(1.0).log_()[:, None], randn(n).exp_()


def _scene(case, seed):
    g, dev, n, nsg = _gen(seed), _dev(), case["n"], case["nsg"]
    pos, log_s, dens = _points(case["scene"], n, g)
    p = dict(positions=pos, scales=log_s.exp_(), quaternions=_unit(g, n, 4), densities=dens,
             color_features=0.2 * torch.randn((n, 3, SH[case["sh"]]), generator=g, device=dev),
             sph_gauss_features=0.1 * torch.randn((n, 3, nsg), generator=g, device=dev),
             bandwidth_sharpness=1.0 + 19.0 * torch.rand((n, nsg), generator=g, device=dev),
             lobe_axis=_unit(g, n * nsg, 3).reshape(n, nsg, 3) if nsg else torch.zeros((n, 0, 3), device=dev))
    if case.get("storage") == "bf16":
        for k in ("densities", "color_features", "sph_gauss_features"):
            p[k] = p[k].to(torch.bfloat16)
    return {k: v.contiguous() for k, v in p.items()}


def _cameras(case, seed, device="cuda"):
    """Inward-facing cameras; the views of a batch have uneven sizes around the case's."""
    rng = np.random.default_rng(int(seed) + 1000)
    cams = []
    for v in range(case["views"]):
        s = 1.0 if case["views"] == 1 else 0.5 + 1.0 * v / (case["views"] - 1)
        if case["n"] >= 3_000_000:
            s = 1.0
        w, h = max(8, int(case["width"] * s)), max(8, int(case["height"] * s))
        ang = 2.0 * math.pi * (v + 0.5 * rng.random()) / case["views"]
        r = rng.uniform(3.0, 4.5)
        eye = [r * math.cos(ang), r * math.sin(ang), rng.uniform(-0.5, 0.5)]
        cams.append(look_at_camera(eye, [0.0, 0.0, 0.0], w, h, fovx=math.radians(45.0), device=device))
    return cams


def _target(n_rays, seed):
    return torch.rand((n_rays, 3), generator=_gen(int(seed) + 7), device=_dev())


def _settings(cam, case):
    return RenderOptixSettings(context=None, update=False, gas=None, program_grps_fwd=None, pipeline_fwd=None,
                               program_grps_bwd=None, pipeline_bwd=None, viewpoint_cam=cam, max_prim_slice=1024,
                               num_sph_gauss=case["nsg"], iteration=0, jitter=0, rnd_sample=0, supersampling=(1, 1),
                               white_background=True, hit_prim_idx=None)


def _raw_cloud(case, seed):
    """Trained tensors of the reference's point cloud (log scales, rgb and SH apart) and its roles."""
    g, dev, n, nsg = _gen(seed), _dev(), case["n"], case["nsg"]
    randn = lambda *s: torch.randn(s, generator=g, device=dev)   # noqa: E731
    pos, log_s, dens = _points("ball", n, g)
    p = dict(positions=pos, scales=log_s, quaternions=_unit(g, n, 4), densities=dens, rgb=0.2 * randn(n, 3),
             spherical_harmonics=0.2 * randn(n, 3, SH[case["sh"]] - 1))
    if nsg:
        p |= dict(sph_gauss_features=0.1 * randn(n, 3, nsg), bandwidth_sharpness=randn(n, nsg),
                  lobe_axis=_unit(g, n * nsg, 3).reshape(n, nsg, 3))
    p = {k: v.contiguous() for k, v in p.items()}
    roles = {k: k for k in ("positions", "scales", "quaternions", "densities", "lobe_axis") if k in p}
    lrs = dict(positions=1e-4, scales=5e-3, quaternions=1e-3, densities=5e-2, rgb=2.5e-3, spherical_harmonics=1.25e-4,
               sph_gauss_features=2.5e-3, bandwidth_sharpness=2.5e-2, lobe_axis=1e-3)
    tail = FusedTrainTail(p, {k: LrSchedule(lrs[k]) for k in p}, roles=roles, normalize_lobe_axis=bool(nsg),
                          max_scale=math.log(2.0))
    for k in p:                                    # moments of a run under way
        tail.exp_avg[k].copy_(1e-3 * randn(*p[k].shape))
        tail.exp_avg_sq[k].copy_(1e-5 * torch.rand(p[k].shape, generator=g, device=dev))
        tail.adam_step[k] = tail.manager_step[k] = 500
    return p, tail, g


def prepare(case, seed):
    kind = case["kind"]
    if kind == "tail":
        p, tail, g = _raw_cloud(case, seed)
        grads = {k: 1e-2 * torch.randn(v.shape, generator=g, device=_dev()) for k, v in p.items()}
        grads["positions"][::5] = 0.0              # Gaussians no ray saw
        floor = torch.full((case["n"], 1), math.log(0.006), device=_dev())
        return dict(case=case, tail=tail, grads=grads, floor=floor)
    if kind == "densify":
        p, tail, g = _raw_cloud(case, seed)
        n, dev = case["n"], _dev()
        # what decides the new size (scales, densities, mean gradients) is the same for every seed, in
        # another order
        g0, perm = _gen(n), torch.randperm(n, generator=g, device=dev)
        _, log_s, dens = _points("ball", n, g0)
        p["scales"].copy_(log_s[perm])
        p["densities"].copy_(dens[perm])
        tail.stats["xyz_gradient_accum_norm"].copy_(torch.randn(n, generator=g0, device=dev).exp_()[perm])
        tail.stats["num_accum"].copy_(torch.randint(0, 40, (n,), generator=g0, device=dev).float()[perm])
        tail.stats["num_accum_gnv"].copy_(tail.stats["num_accum"])
        return dict(case=case, tail=tail, seed=int(seed),
                    f3d=torch.full((n, 1), math.log(0.004), device=_dev()))
    if kind == "filter":
        pos, _, _ = _points("ball", case["n"], _gen(seed))
        cams = _cameras(dict(views=case["cams"], width=800, height=800, n=case["n"]), seed, device="cpu")
        return dict(case=case, pos=pos.contiguous(), cams=cams)
    if kind == "scales":
        pos, _, _ = _points("ball", case["n"], _gen(seed))
        return dict(case=case, pos=pos.contiguous())
    p, cams = _scene(case, seed), _cameras(case, seed)
    st = dict(case=case, params=p)
    n_rays = sum(c.image_width * c.image_height for c in cams)
    if kind == "infer":
        st["views"] = BatchedViews(cams, mode=case["form"])
        return st
    st["target"] = _target(n_rays, seed)
    if kind == "graph":
        st["step"] = GraphedStep(p, BatchedViews(cams, engine=Engine()), st["target"])
        return st
    st["leaves"] = [p[k].requires_grad_(True) for k in KEYS]
    st["settings"] = _settings(cams[0], case) if case["form"] == "dropin" else BatchedViews(cams)
    return st


# ---- one pass ---------------------------------------------------------------------------------------

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        render = RenderOptixFunction if case["form"] == "dropin" else BatchedRenderFunction
        out = render.apply(*state["leaves"], state["settings"])
        loss = torch.nn.functional.mse_loss(out, state["target"])
        trained = state["leaves"] if case["nsg"] else state["leaves"][:5]
        return {"image": out.detach(), "grads": torch.autograd.grad(loss, trained)}
    if kind == "graph":
        step = state["step"]
        loss = step.replay()
        return {"loss": loss, "grads": [step.grads[k] for k in KEYS if step.grads.get(k) is not None]}
    if kind == "infer":
        if case["counts"]:
            img, cnt = render_views_inference(state["params"], state["views"], counts=True)
            return {"image": img, "counts": cnt}
        return {"image": render_views_inference(state["params"], state["views"])}
    if kind == "tail":
        t = state["tail"]
        t.step(min_scale=state["floor"], grads=state["grads"])
        return {"params": t.params, "exp_avg": t.exp_avg, "exp_avg_sq": t.exp_avg_sq, "stats": t.stats}
    if kind == "densify":
        tail = copy.copy(state["tail"])            # the call rebinds its tail: the state keeps the old cloud
        gen = torch.Generator(device=state["f3d"].device).manual_seed(state["seed"])
        r = densify_and_prune(tail, state["f3d"], 0.1, 0.1, 4.0, generator=gen)
        return {"params": {k: v.detach() for k, v in r["params"].items()}, "filter": r["filter_3D"],
                "exp_avg": tail.exp_avg, "exp_avg_sq": tail.exp_avg_sq, "n": r["n"]}
    if kind == "filter":
        return {"filter": compute_3D_filter(state["pos"], state["cams"])}
    return {"scales": initial_log_scales(state["pos"])}


def work(case):
    """Inputs read once and outputs written once; operations of the samples a ray takes before it
    ends (about 24 Gaussians of 14 samples, 20 operations each, three times that with a backward)."""
    n, kind = case["n"], case["kind"]
    if kind == "filter":
        return {"bytes": 16.0 * n + 80.0 * case["cams"], "flops": 25.0 * n * case["cams"]}
    if kind == "scales":
        return {"bytes": 24.0 * n, "flops": 9.0 * n * 64}
    nsh, nsg = SH[case["sh"]], case["nsg"]
    floats = 11 + 3 * nsh + 7 * nsg                # trained floats of a Gaussian
    if kind == "tail":
        return {"bytes": n * (28.0 * floats + 28.0), "flops": 12.0 * n * floats}
    if kind == "densify":
        return {"bytes": n * (24.0 * floats + 20.0), "flops": 30.0 * n}
    stored = 2 if case["storage"] == "bf16" else 4
    par = 40 + stored * (1 + 3 * nsh + 3 * nsg) + 16 * nsg
    grad = 40 + stored * (1 + 3 * nsh + 3 * nsg) + 16 * nsg
    rays = 0
    for v in range(case["views"]):
        s = 1.0 if case["views"] == 1 or n >= 3_000_000 else 0.5 + 1.0 * v / (case["views"] - 1)
        rays += max(8, int(case["width"] * s)) * max(8, int(case["height"] * s))
    ops = rays * 24 * 14 * 20.0
    if kind == "infer":
        return {"bytes": float(n * par + 12 * rays), "flops": ops}
    return {"bytes": float(n * (2 * par + grad) + 36 * rays), "flops": 3 * ops}


# ---- the same results in 64 bits --------------------------------------------------------------------

DT, THR, TEPS = (float(np.float32(v)) for v in (0.0025, 0.1, 0.003))
PAIRS = 30_000_000       # (ray, Gaussian) tests at a time


def _rotation(q):
    w, x, y, z = q.unbind(1)
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                        2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                        2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], 1).reshape(-1, 3, 3)


def _colors(p, eye):
    """(N, 3) colours towards `eye`.  The renderer's default keeps the reference's derivative of the
    degree-3 function y (3 x^2 - y^2) along y, which holds the y^2 fixed."""
    d = p["positions"] - eye
    d = d / d.norm(dim=1, keepdim=True)
    x, y, z = d.unbind(1)
    xx, yy, zz = x * x, y * y, z * z
    b = [0.28209479177387814 * torch.ones_like(x), -0.4886025119029199 * y, 0.4886025119029199 * z,
         -0.4886025119029199 * x, 1.0925484305920792 * x * y, -1.0925484305920792 * y * z,
         0.31539156525252005 * (2 * zz - xx - yy), -1.0925484305920792 * x * z, 0.5462742152960396 * (xx - yy),
         -0.5900435899266435 * y * (3 * xx - yy.detach()), 2.890611442640554 * x * y * z,
         -0.4570457994644658 * y * (4 * zz - xx - yy), 0.3731763325901154 * z * (2 * zz - 3 * xx - 3 * yy),
         -0.4570457994644658 * x * (4 * zz - xx - yy), 1.445305721320277 * z * (xx - yy),
         -0.5900435899266435 * x * (xx - 3 * yy)]
    f = p["color_features"]
    rgb = 0.5 + (f * torch.stack(b[:f.shape[2]], 1)[:, None, :]).sum(2)
    if p["sph_gauss_features"].shape[2]:
        wgt = torch.exp(p["bandwidth_sharpness"] * ((p["lobe_axis"] * d[:, None, :]).sum(2) - 1.0))
        rgb = rgb + (p["sph_gauss_features"] * wgt[:, None, :]).sum(2)
    return rgb


def _exact_view(p, cam, target, n_total):
    """Image of one view and, with a target, the sum of the gradients of the mean squared error into
    the parameters' .grad."""
    dev = p["positions"].device
    W, H = cam.image_width, cam.image_height
    eye = cam.camera_center.to(dev, torch.float64)
    wvt = cam.world_view_transform.to(dev, torch.float64)
    idx = torch.arange(W * H, device=dev)
    sx = (2 * ((idx % W) + 0.5) / W - 1) * float(np.float32(math.tan(cam.FoVx / 2)))
    sy = (2 * ((idx // W) + 0.5) / H - 1) * float(np.float32(math.tan(cam.FoVy / 2)))
    dirs = sx[:, None] * wvt[:3, 0] + sy[:, None] * wvt[:3, 1] + wvt[:3, 2]
    dirs = dirs / dirs.norm(dim=1, keepdim=True)
    with torch.no_grad():
        R = _rotation(p["quaternions"])
        lg = 2.0 * torch.log(p["densities"] / THR)
        delta = lg.clamp_min(0.0).sqrt()
        ext = ((R * (delta[:, None] * p["scales"])[:, None, :]) ** 2).sum(2).sqrt()
        lo, hi = (p["positions"] - ext).amin(0), (p["positions"] + ext).amax(0)
        live = torch.nonzero(lg > 0.0)[:, 0]
        A = R[live].transpose(1, 2) / (p["scales"][live] * delta[live, None])[:, :, None]   # rows of k S^-1 R^T
        Q = A.transpose(1, 2) @ A
        O = eye - p["positions"][live]
        QO = (Q @ O[:, :, None])[:, :, 0]
        c = (O * QO).sum(1) - 1.0
        q6 = torch.stack([Q[:, 0, 0], Q[:, 1, 1], Q[:, 2, 2], 2 * Q[:, 0, 1], 2 * Q[:, 0, 2], 2 * Q[:, 1, 2]])
        t0, t1 = (lo - eye) / dirs, (hi - eye) / dirs
        tin = torch.minimum(t0, t1).amax(1).clamp_min(0.0)
        tout = torch.maximum(t0, t1).amin(1)
    image = torch.empty((W * H, 3), dtype=torch.float64, device=dev)
    step = max(1, min(8192, PAIRS // max(1, len(live))))
    need = target is not None
    for r0 in range(0, W * H, step):
        d, ti, to = dirs[r0:r0 + step], tin[r0:r0 + step], tout[r0:r0 + step]
        with torch.no_grad():
            d6 = torch.stack([d[:, 0] ** 2, d[:, 1] ** 2, d[:, 2] ** 2, d[:, 0] * d[:, 1], d[:, 0] * d[:, 2],
                              d[:, 1] * d[:, 2]], 1)
            a, b = d6 @ q6, -(d @ QO.t())
            disc = b * b - a * c
            ray, k = torch.nonzero((disc > 0) & (b > 0) & (ti < to)[:, None], as_tuple=True)
            s, a, b = disc[ray, k].sqrt(), a[ray, k], b[ray, k]
            first = torch.ceil(((b - s) / a - ti[ray]) / DT).clamp_min(0).long()
            last = torch.floor(((b + s) / a - ti[ray]) / DT).long()
            num = (last - first + 1).clamp_min(0)
            k = live[k]
            n_s = 8 * (int(last.max()) // 8 + 1) if len(last) and int(last.max()) >= 0 else 8
            pair = torch.repeat_interleave(torch.arange(len(ray), device=dev), num)
            off = torch.arange(len(pair), device=dev) - torch.repeat_interleave(torch.cumsum(num, 0) - num, num)
            j = first[pair] + off
            where = ray[pair] * n_s + j
            t = ti[ray][pair] + j * DT
        with torch.set_grad_enabled(need):
            col = _colors(p, eye)
            M = _rotation(p["quaternions"][k]).transpose(1, 2) / p["scales"][k][:, :, None]
            m0 = (M @ (eye - p["positions"][k])[:, :, None])[:, :, 0]
            md = (M @ d[ray][:, :, None])[:, :, 0]
            q0, q1, q2 = (m0 * m0).sum(1), 2 * (m0 * md).sum(1), (md * md).sum(1)
            w = p["densities"][k][pair] * torch.exp(-0.5 * (q0[pair] + t * (q1[pair] + t * q2[pair])))
            sig = torch.zeros(len(d) * n_s, dtype=torch.float64, device=dev).index_add(0, where, w)
            num_c = torch.zeros((len(d) * n_s, 3), dtype=torch.float64, device=dev).index_add(
                0, where, col[k][pair] * w[:, None])
            sig = sig.reshape(len(d), n_s)
            x = sig * DT
            before = torch.cumsum(x, 1) - x
            with torch.no_grad():                       # a slab is marched while T > 0.003 at its start
                on = (torch.exp(-before[:, ::8]) > TEPS).repeat_interleave(8, 1)
            x = x * on
            T = torch.exp(-(torch.cumsum(x, 1) - x))
            wgt = T * -torch.expm1(-x)
            frac = torch.where(sig > 0, wgt / torch.where(sig > 0, sig, torch.ones_like(sig)), torch.zeros_like(sig))
            img = (num_c.reshape(len(d), n_s, 3) * frac[:, :, None]).sum(1) + torch.exp(-x.sum(1))[:, None]
            if need:
                (((img - target[r0:r0 + step]) ** 2).sum() / n_total).backward()
        image[r0:r0 + step] = img.detach()
    return image


def exact(case, seed):
    kind = case["kind"]
    if kind == "tail":
        return _exact_tail(prepare(case, seed))
    if kind == "densify":
        return None                                     # rows copied from the cloud that went in
    if kind == "filter":
        return _exact_filter(prepare(case, seed))
    if kind == "scales":
        return _exact_scales(prepare(case, seed)["pos"].double())
    cams = _cameras(case, seed)
    rays = sum(c.image_width * c.image_height for c in cams)
    if case["scene"] == "ball" or rays * case["n"] > 2.5e11:
        return None                                     # hours of samples over the far field, or minutes of tests
    p = {k: v.double() for k, v in _scene(case, seed).items()}
    target = None if kind == "infer" else _target(rays, seed).double()
    if target is not None:
        for v in p.values():
            v.requires_grad_(True)
    off, images = 0, []
    for c in cams:
        m = c.image_width * c.image_height
        images.append(_exact_view(p, c, None if target is None else target[off:off + m], 3 * rays))
        off += m
    image = torch.cat(images)
    if kind == "infer":
        return {"image": image, "counts": None} if case["counts"] else {"image": image}
    grads = [p[k].grad if p[k].grad is not None else torch.zeros_like(p[k])
             for k in (KEYS if case["nsg"] else KEYS[:5])]
    if kind == "graph":
        return {"loss": ((image - target) ** 2).mean(), "grads": grads}
    return {"image": image, "grads": grads}


def _exact_tail(st):
    t, grads, lo = st["tail"], st["grads"], st["floor"].double()
    p = {k: v.double() for k, v in t.params.items()}
    m = {k: v.double() for k, v in t.exp_avg.items()}
    s = {k: v.double() for k, v in t.exp_avg_sq.items()}
    b1, b2, step = 0.9, 0.999, 501
    for k in p:
        g = grads[k].double()
        m[k] = m[k] + (1 - b1) * (g - m[k])
        s[k] = b2 * s[k] + (1 - b2) * g * g
        p[k] = p[k] - t.lr[k] / (1 - b1 ** step) * m[k] / (s[k].sqrt() / math.sqrt(1 - b2 ** step) + 1e-15)
    p["densities"] = p["densities"].clamp_min(0.0)
    p["quaternions"] = p["quaternions"] / p["quaternions"].norm(dim=1, keepdim=True)
    if "lobe_axis" in p:
        p["lobe_axis"] = p["lobe_axis"] / p["lobe_axis"].norm(dim=2, keepdim=True)
    p["scales"] = torch.maximum(p["scales"], lo).clamp_max(math.log(2.0))
    gn = grads["positions"].double().norm(dim=1)
    seen = (gn > 0).double()
    return {"params": p, "exp_avg": m, "exp_avg_sq": s,
            "stats": {"xyz_gradient_accum_norm": gn, "num_accum": seen, "num_accum_gnv": seen}}


def _exact_filter(st):
    pos = st["pos"].double()
    best = torch.full((len(pos),), math.inf, dtype=torch.float64, device=pos.device)
    focal = 0.0
    for c in st["cams"]:
        wvt = c.world_view_transform.to(pos.device, torch.float64)
        W, H = c.image_width, c.image_height
        fx, fy = W / (2 * math.tan(c.FoVx / 2)), H / (2 * math.tan(c.FoVy / 2))
        focal = max(focal, fx, fy)
        x, y, z = (pos @ wvt[:3, :3] + wvt[3, :3]).unbind(1)
        zc = z.clamp_min(0.001)
        u, v = x / zc * fx + W / 2, y / zc * fy + H / 2
        ok = (z > 0.2) & (u >= -0.15 * W) & (u <= 1.15 * W) & (v >= -0.15 * H) & (v <= 1.15 * H)
        best = torch.where(ok, torch.minimum(best, zc), best)
    seen = torch.isfinite(best)
    best = torch.where(seen, best, best[seen].max())
    return {"filter": torch.log(0.5 * best / focal)[:, None]}


def _exact_scales(pos):
    n = len(pos)
    if n > 250_000:
        return None
    out = torch.empty(n, dtype=torch.float64, device=pos.device)
    step = max(1, 250_000_000 // n)
    for i in range(0, n, step):
        d = (pos[i:i + step, 0:1] - pos[None, :, 0]) ** 2
        for a in (1, 2):
            d += (pos[i:i + step, a:a + 1] - pos[None, :, a]) ** 2
        j = torch.arange(len(d), device=pos.device)
        d[j, i + j] = math.inf
        out[i:i + step] = sum(_pop_min(d) for _ in range(3)) / 3
    return {"scales": torch.log(torch.sqrt(out.clamp_min(1e-7)))[:, None].repeat(1, 3)}


def _pop_min(d):
    """Row minima of d, each replaced by infinity."""
    v, at = d.min(1)
    d.scatter_(1, at[:, None], math.inf)
    return v
