"""The work this framework is used for, as cases that can be timed and checked one by one.

Kinds of case (the sizes are those of the workload shapes in aniso_b200/scenes.py and their ragged
neighbours; every scene is seeded and synthetic, with the distributions listed there):

- ``frame``  one view of a resident scene into device memory (GpuRenderer.render_device): a viewer or
  a server that keeps its images on the GPU.
- ``host``   one view into host memory (GpuRenderer.render, the drop-in for the reference's call):
  what `aniso render` does per camera.
- ``batch``  several views of several scenes in one replayed launch sequence (BatchRenderer): the
  camera path stream and offline rendering of whole view sets.
- ``grad``   one view forward and backward (autograd.rasterize): a user's own training loop.
- ``gradbatch``  views of several scenes forward and backward in one call (autograd.rasterize_batch).
- ``step``   one whole step of the training loop (train.Trainer.step): render, L1 + SSIM, adjoint, Adam.
"""
import math

import numpy as np
import torch
import torch.nn.functional as F

from aniso_b200.autograd import rasterize, rasterize_batch
from aniso_b200.renderer import BatchOptions, BatchRenderer, GpuRenderer, RenderOptions
from aniso_b200.scenes import RESOLUTIONS_4, Camera, fibonacci_cameras, front_camera, ring_cameras
from aniso_b200.train import GaussianModel, Trainer

# Scene boxes and camera placements of the workload shapes: (box low, box high).
BOXES = {
    "cloud": ((-4.0, -4.0, 2.0), (4.0, 4.0, 12.0)),       # camera at the origin looking down +z
    "ring": ((-10.0, -3.0, -10.0), (10.0, 3.0, 10.0)),    # cameras on a ring of radius 8 inside it
    "wide": ((-15.0, -4.0, -15.0), (15.0, 4.0, 15.0)),    # camera 8 units back, or a ring of radius 8
    "cube": ((-10.0, -10.0, -10.0), (10.0, 10.0, 10.0)),  # cameras on a sphere of radius 10
}


def listed():
    return [
        # The smallest call in earnest: 100k Gaussians at 640x360, where launches and latency count.
        dict(name="frame_100k_640x360", kind="frame", n=100_000, box="cloud", width=640, height=360, degree=3,
             option_degree=3, splat_scale=1.0, view=0),
        # The headline view: 740k Gaussians with degree-3 colour at 1280x720.
        dict(name="frame_740k_1280x720", kind="frame", n=740_000, box="ring", width=1280, height=720, degree=3,
             option_degree=3, splat_scale=1.0, view=0),
        # A large scene on a full-HD screen: more tiles (8160) and several million splat-tile pairs.
        dict(name="frame_2200k_1920x1080", kind="frame", n=2_200_000, box="wide", width=1920, height=1080, degree=3,
             option_degree=3, splat_scale=1.0, view=0),
        # Ragged sizes: an odd Gaussian count and image size, degree-1 colour, shrunken splats.
        dict(name="frame_411003_1277x713_sh1", kind="frame", n=411_003, box="ring", width=1277, height=713, degree=1,
             option_degree=3, splat_scale=0.75, view=3),
        # The drop-in call: the headline view into a pinned host image.
        dict(name="host_740k_1280x720", kind="host", n=740_000, box="ring", width=1280, height=720, degree=3,
             option_degree=3, splat_scale=1.0, view=5, pinned=True),
        # A camera path: 16 consecutive frames of one scene per batch, as the path streamer renders them.
        dict(name="batch_16x740k_1280x720", kind="batch", n=740_000, scenes=1, box="ring", views=16, width=1280,
             height=720, degree=3, tile_h=16, blend_batch=256, radix_bits=8),
        # A whole view set: 64 views of mixed resolution (320x180 to 1920x1080) of a 1M-Gaussian scene.
        dict(name="batch_64x1m_mixed", kind="batch", n=1_000_000, scenes=1, box="cube", views=64, width=0, height=0,
             degree=3, tile_h=32, blend_batch=256, radix_bits=9),
        # A small view forward and backward: the early steps of a training run.
        dict(name="grad_100k_640x360", kind="grad", n=100_000, box="cloud", width=640, height=360, degree=3,
             option_degree=3, splat_scale=1.0, view=0),
        # The large view forward and backward.
        dict(name="grad_2200k_1280x720", kind="grad", n=2_200_000, box="wide", width=1280, height=720, degree=3,
             option_degree=3, splat_scale=1.0, view=0),
        # Eight scenes of uneven size, three views each, forward and backward as one replayed batch.
        dict(name="gradbatch_8scenes_24views", kind="gradbatch", n=200_000, n_last=3_000_000, scenes=8, box="wide",
             views=3, width=1280, height=720, degree=3, tile_h=16, blend_batch=256),
        # One step of the training loop past densification: loss, adjoint and optimizer included.
        dict(name="step_740k_1280x720", kind="step", n=740_000, box="ring", width=1280, height=720, degree=3,
             view=2, steps=16_000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "host", "batch", "grad", "grad", "gradbatch", "step"])
    box = rng.choice(["cloud", "ring", "wide"])
    w = _log(rng, 160, 1920)
    h = max(90, min(1080, int(w * rng.uniform(0.5, 0.7))))
    base = dict(kind=kind, box=box, width=w, height=h, degree=3)
    if kind in ("frame", "host"):
        base.update(n=_log(rng, 20_000, 2_200_000), degree=rng.randint(0, 3), option_degree=rng.randint(1, 3),
                    splat_scale=round(rng.uniform(0.6, 1.2), 3), view=rng.randint(0, 15))
        if kind == "host":
            base.update(pinned=rng.random() < 0.5)
    elif kind == "batch":
        base.update(n=_log(rng, 20_000, 500_000), scenes=rng.randint(1, 2), views=rng.randint(2, 12),
                    tile_h=rng.choice([8, 16, 32]), blend_batch=rng.choice([128, 256]), radix_bits=rng.choice([8, 9]))
    elif kind == "grad":
        base.update(n=_log(rng, 10_000, 1_500_000), degree=rng.choice([1, 3]), option_degree=rng.randint(0, 3),
                    splat_scale=round(rng.uniform(0.6, 1.2), 3), view=rng.randint(0, 15))
    elif kind == "gradbatch":
        n = _log(rng, 10_000, 200_000)
        base.update(n=n, n_last=2 * n + 1, scenes=rng.randint(1, 3), views=rng.randint(1, 4),
                    tile_h=rng.choice([16, 32]), blend_batch=rng.choice([128, 256]))
    else:
        base.update(n=_log(rng, 20_000, 740_000), view=rng.randint(0, 15), steps=16_000 + rng.randint(0, 5_000))
    return base


# ---- inputs ---------------------------------------------------------------------------------------


def _gen(seed, part=0):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 64 + part)


def _raw(n, box, degree, gen):
    """The optimizer's raw tensors of one scene on the GPU: means, log-scales, quaternions, opacity
    logits, SH (n, K, 3)."""
    lo, hi = (torch.tensor(v, device="cuda") for v in BOXES[box])
    k = (degree + 1) ** 2
    means = lo + (hi - lo) * torch.rand(n, 3, device="cuda", generator=gen)
    log_scales = torch.randn(n, 3, device="cuda", generator=gen) * 0.5 - 4.0
    quats = F.normalize(torch.randn(n, 4, device="cuda", generator=gen), dim=-1)
    logits = torch.randn(n, device="cuda", generator=gen) * 1.5
    sh = torch.randn(n, k, 3, device="cuda", generator=gen) * 0.05
    sh[:, 0] *= 10.0
    return [means, log_scales, quats, logits, sh]


def _renderer(raw, degree):
    """An uploaded scene: (n, 11) activated Gaussians and their SH, as a loader hands them over."""
    means, log_scales, quats, logits, sh = raw
    g = torch.cat([means, torch.exp(log_scales), quats, torch.sigmoid(logits)[:, None]], dim=1)
    return GpuRenderer(g.cpu().numpy(), sh.reshape(sh.shape[0], -1).cpu().numpy(), degree)


def _camera(case, k=None):
    w, h = case["width"], case["height"]
    f = 1100.0 * w / 1280.0
    view = case.get("view", 0) if k is None else k
    if case["box"] == "cloud":
        t = np.array([0.02 * view, 0.01 * view, 0.0])
        return Camera(w, h, 500.0 * w / 640.0, 500.0 * w / 640.0, w / 2.0, h / 2.0, np.eye(3), t, "origin")
    if case["box"] == "wide" and view == 0:
        return front_camera(w, h, f, 8.0)
    return ring_cameras(16, 8.0, w, h, f)[view % 16]


def _cameras(case):
    if case["width"] == 0:  # the mixed view set
        return fibonacci_cameras(case["views"], 10.0, RESOLUTIONS_4, seed=3)
    return [_camera(case, k) for k in range(case["views"])]


def _scene_sizes(case):
    """Gaussians per scene, spread evenly from n to n_last."""
    s, a, b = case["scenes"], case["n"], case["n_last"]
    return [a] if s == 1 else [int(a + (b - a) * i // (s - 1)) for i in range(s)]


def _grad_batch_views(case):
    """Per view its scene and its camera; every other view at three quarters of the size."""
    scenes, cams = [], []
    for s in range(case["scenes"]):
        for v in range(case["views"]):
            small = v % 2 == 0
            c = dict(case, width=case["width"] * 3 // 4 if small else case["width"],
                     height=case["height"] * 3 // 4 if small else case["height"])
            scenes.append(s)
            cams.append(_camera(c, 4 * v))
    return scenes, cams


# Scales of the gradients met in training, for optimizer moments as a running loop holds them.
_MOMENTS = {"means": 1e-4, "log_scales": 1e-6, "quats": 1e-6, "opacity_logits": 1e-6, "sh": 1e-6}


def _step_inputs(case, seed):
    """Raw tensors, target image and Adam moments of a training run under way."""
    raw = _raw(case["n"], case["box"], 3, _gen(seed))
    cam = _camera(case)
    gen = _gen(seed, 1)
    moved = [t.clone() for t in raw]
    moved[0] += 0.01 * torch.randn(moved[0].shape, device="cuda", generator=gen)
    moved[4][:, 0] += 0.05 * torch.randn(moved[4][:, 0].shape, device="cuda", generator=gen)
    with torch.no_grad():
        target = rasterize(*moved, cam).clamp(0, 1)
    m, v = {}, {}
    for (k, s), t in zip(_MOMENTS.items(), raw):
        m[k] = s * torch.randn(t.shape, device="cuda", generator=gen)
        v[k] = (s * torch.exp(torch.randn(t.shape, device="cuda", generator=gen))) ** 2
    return raw, cam, target, m, v


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("frame", "host"):
        r = _renderer(_raw(case["n"], case["box"], case["degree"], _gen(seed)), case["degree"])
        cam = _camera(case)
        options = RenderOptions(case["option_degree"], case["splat_scale"])
        r.render(cam, options=options)  # sizes the scene's buffers for its views
        state = dict(kind=kind, r=r, cam=cam, options=options)
        if kind == "frame":
            state["image"] = torch.empty(cam.height, cam.width, 3, dtype=torch.uint8, device="cuda")
        else:
            state["image"] = torch.empty(cam.height, cam.width, 3, dtype=torch.uint8,
                                         pin_memory=case["pinned"]).numpy()
        return state
    if kind == "batch":
        rs = [_renderer(_raw(case["n"], case["box"], case["degree"], _gen(seed, s)), case["degree"])
              for s in range(case["scenes"])]
        views = _cameras(case)
        scene = [s for s in range(case["scenes"]) for _ in views]
        cams = views * case["scenes"]
        tile = (8, 8) if case["tile_h"] == 8 else (16, case["tile_h"])
        b = BatchRenderer(rs, scene, BatchOptions(3, 1.0, tile, case["blend_batch"], True, case["radix_bits"]))
        images = [torch.empty(c.height, c.width, 3, dtype=torch.uint8, device="cuda") for c in cams]
        ptrs = [t.data_ptr() for t in images]
        for attempt in range(3):  # sizes the pair buffers and records the launch sequence
            b.render_device(cams, ptrs)
            try:
                b.sync()
                break
            except RuntimeError:
                if attempt == 2:
                    raise
        b.render_device(cams, ptrs)
        return dict(kind=kind, b=b, cams=cams, ptrs=ptrs, images=images, rs=rs)
    if kind == "grad":
        raw = _raw(case["n"], case["box"], case["degree"], _gen(seed))
        cam = _camera(case)
        up = torch.randn(cam.height, cam.width, 3, device="cuda", generator=_gen(seed, 1))
        return dict(kind=kind, leaves=[t.requires_grad_(True) for t in raw], cam=cam, up=up,
                    options=(case["option_degree"], case["splat_scale"]))
    if kind == "gradbatch":
        scenes = [[t.requires_grad_(True) for t in _raw(n, case["box"], 3, _gen(seed, s))]
                  for s, n in enumerate(_scene_sizes(case))]
        vs, cams = _grad_batch_views(case)
        gen = _gen(seed, 63)
        ups = [torch.randn(c.height, c.width, 3, device="cuda", generator=gen) for c in cams]
        return dict(kind=kind, scenes=scenes, vs=vs, cams=cams, ups=ups,
                    options=BatchOptions(3, 1.0, (16, case["tile_h"]), case["blend_batch"], True, 8))
    raw, cam, target, m, v = _step_inputs(case, seed)
    model = GaussianModel.from_raw(*raw, scene_scale=10.0)
    model.m, model.v = m, v
    trainer = Trainer(model, total_steps=30_000)
    trainer.steps = case["steps"]
    return dict(kind=kind, trainer=trainer, cam=cam, target=target)


# ---- one pass -------------------------------------------------------------------------------------


def run(state):
    kind = state["kind"]
    if kind == "frame":
        state["r"].render_device(state["cam"], state["image"].data_ptr(), torch.cuda.current_stream().cuda_stream,
                                 state["options"])
        return state["image"]
    if kind == "host":
        return state["r"].render(state["cam"], options=state["options"], out=state["image"])
    if kind == "batch":
        state["b"].render_device(state["cams"], state["ptrs"], torch.cuda.current_stream().cuda_stream)
        return state["images"]
    if kind == "grad":
        image = rasterize(*state["leaves"], state["cam"], *state["options"])
        return {"image": image.detach(), "grads": list(torch.autograd.grad(image, state["leaves"], state["up"]))}
    if kind == "gradbatch":
        images = rasterize_batch(state["scenes"], state["cams"], state["vs"], options=state["options"])
        leaves = [t for s in state["scenes"] for t in s]
        grads = torch.autograd.grad(images, leaves, state["ups"])
        return {"images": [t.detach() for t in images], "grads": list(grads)}
    trainer = state["trainer"]
    loss = trainer.step(state["cam"], state["target"])
    model = trainer.model
    return {"loss": loss, "params": [t.detach() for t in model.tensors()], "m": list(model.m.values()),
            "v": list(model.v.values())}


def work(case):
    """Bytes: the scene's tensors read once, the images (and gradients, and optimizer state) written
    once. Flops: the projection (about 250 per Gaussian and view) and one splat evaluation (about 20)
    for each of a nominal 50 splats a pixel blends."""
    kind = case["kind"]
    k = (case["degree"] + 1) ** 2 * 3
    if kind == "gradbatch":
        n = sum(_scene_sizes(case))
        pixels = sum(c.width * c.height for c in _grad_batch_views(case)[1])
        entries = n * case["views"]
    elif kind == "batch":
        n = case["n"] * case["scenes"]
        pixels = sum(c.width * c.height for c in _cameras(case)) * case["scenes"]
        entries = n * case["views"]
    else:
        n = entries = case["n"]
        pixels = case["width"] * case["height"]
    scene = 4 * n * (11 + k)
    flops = 250 * entries + 50 * 20 * pixels
    if kind in ("frame", "host", "batch"):
        return {"bytes": scene + 3 * pixels, "flops": flops}
    if kind == "step":  # parameters and both moments read and written, the target read
        return {"bytes": 6 * scene + 12 * pixels, "flops": 4 * flops + 20 * n * (11 + k)}
    return {"bytes": 2 * scene + 24 * pixels, "flops": 4 * flops}


# ---- the same in 64 bits --------------------------------------------------------------------------


def _sh_basis(degree, d):
    x, y, z = d.unbind(-1)
    one = torch.ones_like(x)
    b = [0.28209479177387814 * one]
    if degree >= 1:
        c = 0.4886025119029199
        b += [-c * y, c * z, -c * x]
    if degree >= 2:
        xx, yy, zz = x * x, y * y, z * z
        b += [1.0925484305920792 * x * y, -1.0925484305920792 * y * z, 0.31539156525252005 * (2 * zz - xx - yy),
              -1.0925484305920792 * x * z, 0.5462742152960396 * (xx - yy)]
    if degree >= 3:
        b += [-0.5900435899266435 * y * (3 * xx - yy), 2.890611442640554 * x * y * z,
              -0.4570457994644658 * y * (4 * zz - xx - yy), 0.3731763325901154 * z * (2 * zz - 3 * xx - 3 * yy),
              -0.4570457994644658 * x * (4 * zz - xx - yy), 1.445305721320277 * z * (xx - yy),
              -0.5900435899266435 * x * (xx - 3 * yy)]
    return torch.stack(b, -1)


def _project64(raw, cam, degree, splat_scale):
    """The visible splats in 64 bits, nearest first: (parameters (V, 9) of u, v, conic a, b, c,
    opacity, rgb; pixel rectangle (V, 4) of the 8x8 tiles each covers)."""
    means, log_scales, quats, logits, sh = raw
    dev = means.device
    W = torch.tensor(cam.R, dtype=torch.float64, device=dev)
    t = torch.tensor(cam.t, dtype=torch.float64, device=dev)
    q = F.normalize(quats, dim=-1)
    w, x, y, z = q.unbind(-1)
    R = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                     2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                     2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], -1).view(-1, 3, 3)
    M = R * (torch.exp(log_scales) * splat_scale)[:, None, :]
    p = means @ W.T + t
    px, py, pz = p.unbind(-1)
    near = pz < 0.2
    pz = torch.where(near, torch.ones_like(pz), pz)
    lx, ly = 1.3 * 0.5 * cam.width / cam.fx, 1.3 * 0.5 * cam.height / cam.fy
    tx, ty = (px / pz).clamp(-lx, lx) * pz, (py / pz).clamp(-ly, ly) * pz
    zero = torch.zeros_like(pz)
    J = torch.stack([cam.fx / pz, zero, -cam.fx * tx / pz ** 2, zero, cam.fy / pz, -cam.fy * ty / pz ** 2], -1)
    TM = J.view(-1, 2, 3) @ W @ M
    cov = TM @ TM.transpose(1, 2)
    a, b, c = cov[:, 0, 0] + 0.3, cov[:, 0, 1], cov[:, 1, 1] + 0.3
    det = a * c - b * b
    u, v = cam.fx * px / pz + cam.cx, cam.fy * py / pz + cam.cy
    with torch.no_grad():
        mid = 0.5 * (a + c)
        radius = torch.ceil(3 * torch.sqrt(mid + torch.sqrt((mid * mid - det).clamp_min(0.1))))
        seen = ~near & (det > 0) & (u + radius >= 0) & (v + radius >= 0) & (u - radius < cam.width) & \
            (v - radius < cam.height)
        order = torch.argsort(pz[seen], stable=True)
        pick = torch.nonzero(seen)[:, 0][order]
        rect = torch.stack([(torch.trunc(e) / 8).trunc() * 8 for e in (u - radius, v - radius, u + radius, v + radius)],
                           -1)[pick].long()
        rect[:, :2].clamp_min_(0)
        rect[:, 2] = (rect[:, 2] + 7).clamp_max(cam.width - 1)
        rect[:, 3] = (rect[:, 3] + 7).clamp_max(cam.height - 1)
    eye = -(W.T @ t)
    basis = _sh_basis(degree, F.normalize(means[pick] - eye, dim=-1))
    rgb = (0.5 + torch.einsum("nk,nkc->nc", basis, sh[pick][:, : basis.shape[1]])).clamp_min(0)
    conic = torch.stack([c, -b, a], -1)[pick] / det[pick][:, None]
    uv = torch.stack([u, v], -1)[pick]
    return torch.cat([uv, conic, torch.sigmoid(logits)[pick][:, None], rgb], -1), rect


def _tiles64(rect, width, height, edge=16):
    """(tile index, splats nearest first) of every tile that has any."""
    tx = (width + edge - 1) // edge
    x0, y0, x1, y1 = (rect // edge).unbind(-1)
    wide, high = (x1 - x0 + 1).clamp_min(0), (y1 - y0 + 1).clamp_min(0)
    count = wide * high
    splat = torch.repeat_interleave(torch.arange(rect.shape[0], device=rect.device), count)
    k = torch.arange(splat.shape[0], device=rect.device) - (count.cumsum(0) - count)[splat]
    tile = (y0[splat] + k // wide[splat]) * tx + x0[splat] + k % wide[splat]
    tile, at = torch.sort(tile, stable=True)
    ids, n = torch.unique_consecutive(tile, return_counts=True)
    return list(zip(ids.tolist(), torch.split(splat[at], n.tolist()))), tx


def _blend64(s, rect, xs, ys):
    """Colour (pixels, 3) of splats s (nearest first) at pixels (xs, ys)."""
    dx, dy = xs[None] + 0.5 - s[:, 0:1], ys[None] + 0.5 - s[:, 1:2]
    power = -0.5 * (s[:, 2:3] * dx * dx + s[:, 4:5] * dy * dy) - s[:, 3:4] * dx * dy
    inside = (xs[None] >= rect[:, 0:1]) & (xs[None] <= rect[:, 2:3]) & (ys[None] >= rect[:, 1:2]) & \
        (ys[None] <= rect[:, 3:4])
    alpha = (s[:, 5:6] * torch.exp(power)).clamp(max=0.99)
    alpha = torch.where(inside & (power <= 0) & (alpha >= 1.0 / 255.0), alpha, torch.zeros_like(alpha))
    T = torch.cumprod(1 - alpha, 0)
    before = torch.cat([torch.ones_like(T[:1]), T[:-1]])
    weight = torch.where(T >= 1e-4, alpha * before, torch.zeros_like(alpha))
    return weight.T @ s[:, 6:9]


def _render64(raw, cam, degree, splat_scale, upstream):
    """(image, gradients of the raw tensors) in 64 bits; upstream(image) gives dL/d(image)."""
    leaves = [t.detach().double().requires_grad_(True) for t in raw]
    splats, rect = _project64(leaves, cam, degree, splat_scale)
    flat = splats.detach()
    tiles, tx = _tiles64(rect, cam.width, cam.height)
    image = torch.zeros(cam.height, cam.width, 3, dtype=torch.float64, device=flat.device)
    grad, up = torch.zeros_like(flat), None
    for backward in (False, True):
        for tile, idx in tiles:
            x0, y0 = tile % tx * 16, tile // tx * 16
            ys, xs = torch.meshgrid(torch.arange(y0, min(y0 + 16, cam.height), device=flat.device),
                                    torch.arange(x0, min(x0 + 16, cam.width), device=flat.device), indexing="ij")
            xs, ys = xs.reshape(-1), ys.reshape(-1)
            s = flat[idx]
            if not backward:
                image[ys, xs] = _blend64(s, rect[idx], xs, ys)
            else:
                s.requires_grad_(True)
                (g,) = torch.autograd.grad(_blend64(s, rect[idx], xs, ys), s, up[ys, xs])
                grad.index_add_(0, idx, g)
        if not backward:
            up = upstream(image)
    return image, torch.autograd.grad(splats, leaves, grad)


def _ssim64(a, b):
    """Mean SSIM of (H, W, 3) images: an 11x11 Gaussian window of sigma 1.5, as two 11-tap passes."""
    g = torch.exp(-((torch.arange(11, device=a.device) - 5) ** 2).double() / 4.5)
    g = g / g.sum()

    def blur(t):
        t = sum(g[k] * t[k:t.shape[0] - 10 + k] for k in range(11))
        return sum(g[k] * t[:, k:t.shape[1] - 10 + k] for k in range(11))

    ma, mb = blur(a), blur(b)
    va, vb, vab = blur(a * a) - ma ** 2, blur(b * b) - mb ** 2, blur(a * b) - ma * mb
    c1, c2 = 0.01 ** 2, 0.03 ** 2
    return (((2 * ma * mb + c1) * (2 * vab + c2)) / ((ma ** 2 + mb ** 2 + c1) * (va + vb + c2))).mean()


def exact(case, seed):
    kind = case["kind"]
    if kind == "grad":
        state = prepare(case, seed)
        degree = min(case["option_degree"], case["degree"])
        image, grads = _render64(state["leaves"], state["cam"], degree, case["splat_scale"],
                                 lambda img: state["up"].double())
        return {"image": image, "grads": list(grads)}
    if kind == "step":
        raw, cam, target, m, v = _step_inputs(case, seed)
        target = target.double()
        loss = []

        def upstream(image):
            image = image.detach().requires_grad_(True)
            value = 0.8 * (image - target).abs().mean() + 0.2 * (1 - _ssim64(image, target))
            loss.append(float(value.detach()))
            return torch.autograd.grad(value, image)[0]

        _, grads = _render64(raw, cam, 3, 1.0, upstream)
        t = case["steps"] + 1
        rate = {"means": 1.6e-4 * 10.0 * 0.01 ** (case["steps"] / 30_000), "log_scales": 5e-3, "quats": 1e-3,
                "opacity_logits": 5e-2, "sh": 2.5e-3}
        params, ms, vs = [], [], []
        for (k, lr), p, g in zip(rate.items(), raw, grads):
            a = m[k].double() * 0.9 + 0.1 * g
            b = v[k].double() * 0.999 + 0.001 * g * g
            size = torch.full_like(a, lr)
            if k == "sh":
                size[:, 1:] = 2.5e-3 / 20
            params.append(p.double() - size / (1 - 0.9 ** t) * a / (torch.sqrt(b / (1 - 0.999 ** t)) + 1e-15))
            ms.append(a)
            vs.append(b)
        return {"loss": torch.tensor(loss[0], dtype=torch.float64), "params": params, "m": ms, "v": vs}
    return None  # 8-bit images are whole numbers; a batch's gradients are sums of the single views' above
