"""Performance cases: the work that users of this framework have it do, through its public API.

The framework trains 3D Gaussian splatting scenes. A user creates a Trainer (or a Batch of scenes) from
host arrays and steps it, reading the model, the statistics, rendered views or the PSNR now and then; a
program with its own training loop uses the Rasterizer (forward and backward); ground-truth or preview
views are rendered with renderViewsSh; and a scene may start from the learned warm-start. Sizes follow
the Fast / Balanced / High presets (scenes.PRESETS) and the tests' scenes, with odd sizes beside them.

Kinds of cases:
  train   Trainer.step(steps), then the model and the statistics. The model is one part-way through its
          schedule (anisotropic, opaque Gaussians); densification is over, as in the last 40 % of every
          schedule; learning rates are those the means schedule ends with, for every group
          (means_lr_final is 1/100 of the first rate).
  batch   Batch.step(steps) of several scenes at once, then every scene's model.
  eval    Trainer.evaluatePsnr over the training views and one rendered view.
  raster  Rasterizer.forward and, with backward, Rasterizer.backward on host arrays.
  views   renderViewsSh: quantised views of a model with spherical harmonics.
  warm    warmstartInit: the initial model of a point cloud through the network.
  mlp     WarmStartNet.loss_grad: one training pass of the warm-start network over `rows` samples.
"""
from __future__ import annotations

import dataclasses
import math

import numpy as np
import torch

from univeral_3d_reconstruction_system_b200 import api, scenes
from univeral_3d_reconstruction_system_b200.types import SH_C0, GaussianModel, LearningRates, RasterSettings, \
    TrainImage, TrainOptions

GROUPS = ("means", "scales", "quats", "opacities", "colors")


def listed():
    return [
        # The smallest call: one step of a test-sized scene (4k Gaussians, 96x72), as an interactive
        # program steps and shows the model; launches and host work count.
        dict(name="train-tiny-1step", kind="train", gaussians=4_000, width=96, height=72, views=8, steps=1, tile=16,
             bg=False, mixed=False),
        # The Fast preset at its cap, stepped between two progress reports.
        dict(name="train-fast", kind="train", gaussians=80_000, width=320, height=240, views=32, steps=100, tile=16,
             bg=False, mixed=False),
        # The Balanced preset at its cap.
        dict(name="train-balanced", kind="train", gaussians=150_000, width=480, height=360, views=24, steps=50,
             tile=16, bg=False, mixed=False),
        # The High preset at its cap: the framework's headline workload.
        dict(name="train-high", kind="train", gaussians=300_000, width=640, height=480, views=24, steps=50, tile=16,
             bg=False, mixed=False),
        # Photos in landscape and portrait format of an odd size over a coloured background: views of two
        # sizes, so every step is launched by itself.
        dict(name="train-mixed-odd", kind="train", gaussians=33_333, width=357, height=203, views=13, steps=40, tile=16,
             bg=True, mixed=True),
        # Four scenes of different size trained at once on one GPU.
        dict(name="batch-4", kind="batch", gaussians=40_000, scenes=4, views=12, steps=40),
        # Progress evaluation of a High-sized scene: PSNR over its views and a preview.
        dict(name="eval-high", kind="eval", gaussians=250_000, width=640, height=480, views=16, tile=16, bg=False),
        # A program's own loop around the rasterizer, odd sizes and a background.
        dict(name="raster-odd", kind="raster", gaussians=7_919, width=161, height=121, tile=16, bg=True,
             backward=True),
        # The same at High size.
        dict(name="raster-high", kind="raster", gaussians=250_000, width=640, height=480, tile=16, bg=False,
             backward=True),
        # Ground-truth or preview views of a finished model with degree-3 harmonics.
        dict(name="views-high", kind="views", gaussians=250_000, width=640, height=480, views=16, degree=3, tile=16),
        # Warm start of a High-sized scene's sparse points (30k points).
        dict(name="warm-30k", kind="warm", points=30_000, width=640, height=480, views=40),
        # A training pass of the warm-start network over one scene's samples.
        dict(name="mlp-grad-16k", kind="mlp", rows=16_384),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "batch", "eval", "raster", "raster", "views", "warm", "mlp"])
    w, h = rng.randint(96, 640), rng.randint(72, 480)
    tile = rng.choice([16, 16, 16, 8, 32])
    if kind == "train":
        return dict(kind=kind, gaussians=_log(rng, 4_000, 300_000), width=w, height=h, views=rng.randint(4, 24),
                    steps=rng.choice([1, 5, 15]), tile=tile, bg=rng.random() < 0.3, mixed=rng.random() < 0.3)
    if kind == "batch":
        return dict(kind=kind, gaussians=_log(rng, 5_000, 40_000), scenes=rng.randint(2, 4), views=rng.randint(4, 12),
                    steps=rng.choice([10, 20, 33, 40]))
    if kind == "eval":
        return dict(kind=kind, gaussians=_log(rng, 4_000, 250_000), width=w, height=h, views=rng.randint(4, 16),
                    tile=tile, bg=rng.random() < 0.3)
    if kind == "raster":
        return dict(kind=kind, gaussians=_log(rng, 1_000, 250_000), width=w, height=h, tile=tile,
                    bg=rng.random() < 0.5, backward=rng.random() < 0.75)
    if kind == "views":
        return dict(kind=kind, gaussians=_log(rng, 4_000, 250_000), width=w, height=h, views=rng.randint(2, 16),
                    degree=rng.randint(0, 3), tile=tile)
    if kind == "warm":
        return dict(kind=kind, points=_log(rng, 1_000, 30_000), width=w, height=h, views=rng.randint(4, 40))
    return dict(kind=kind, rows=_log(rng, 256, 16_384))


# ---------------------------------------------------------------- inputs


def _settings(case):
    bg = (0.2, 0.5, 0.8) if case.get("bg") else (0.0, 0.0, 0.0)
    return RasterSettings(tile_size=case.get("tile", 16), background=bg)


def _scene(gaussians, width, height, views, seed, degree=0):
    """The High preset's kind of scene (hemisphere of cameras around a cube of Gaussians) at this size;
    focal length in proportion to the larger side. Fewer Gaussians are larger ones, so that a small scene
    covers its images as a large one does."""
    spec = dataclasses.replace(scenes.PRESETS["high"], name="case", gt_count=gaussians, views=views, width=width,
                               height=height, focal=600.0 * max(width, height) / 640.0, sh_degree=degree,
                               init_count=min(1000, gaussians))
    sc = scenes.make_scene(spec, seed)
    sc.truth.scales += np.float32(math.log(250_000 / gaussians) / 3.0)
    return sc


def _part_trained(sc, count, rng):
    """A model part-way through training: the truth's Gaussians (some twice) with every group off by noise."""
    n, t = sc.truth.size(), sc.truth
    i = np.concatenate([np.arange(min(n, count)), rng.integers(0, n, size=max(0, count - n))])

    def off(a, s):
        return (a[i] + rng.normal(0.0, s, size=a[i].shape)).astype(np.float32)

    sigma = float(np.exp(t.scales.mean()))
    return GaussianModel(off(t.means, 0.3 * sigma), off(t.scales, 0.2), off(t.quats, 0.1), off(t.opacities, 0.5),
                         off(t.colors, 0.2))


def _options(case, gaussians):
    return TrainOptions(iterations=10_000_000, max_gaussians=gaussians,
                        lr=LearningRates(means=1.6e-6, scales=5e-5, quats=1e-5, opacities=1e-4, colors=2.5e-5),
                        means_lr_final=1.6e-6, refine_start=0, refine_stop=0, opacity_reset_interval=0,
                        raster=_settings(case))


def _training(case, seed):
    """(initial model, images, extent, options) of a training scene."""
    n = case["gaussians"]
    sc = _scene(max(1, n * 5 // 6), case["width"], case["height"], case["views"], seed)
    if case.get("mixed"):  # every other photo in portrait format
        for k in range(1, len(sc.cameras), 2):
            c = sc.cameras[k]
            sc.cameras[k] = dataclasses.replace(c, width=c.height, height=c.width, cx=c.cy, cy=c.cx)
    views = api.renderViewsSh(sc.truth, None, 0, sc.cameras, RasterSettings(background=_settings(case).background))
    images = [TrainImage(c, v) for c, v in zip(sc.cameras, views)]
    return _part_trained(sc, n, np.random.default_rng([seed, 1])), images, sc.extent, _options(case, n)


def _batch_scenes(case, seed):
    sizes = [(320, 240, 1), (480, 360, 2), (320, 240, 2), (640, 480, 4)]  # width, height, share of the Gaussians
    return [dict(gaussians=case["gaussians"] * f, width=w, height=h, views=case["views"]) for w, h, f in
            sizes[: case["scenes"]]]


def _raster_inputs(case, seed):
    sc = _scene(case["gaussians"], case["width"], case["height"], 5, seed)
    model = _part_trained(sc, case["gaussians"], np.random.default_rng([seed, 2]))
    dl = np.random.default_rng([seed, 3]).normal(0.0, 1e-6, (case["height"], case["width"], 3)).astype(np.float32)
    return model, sc.cameras[seed % 5], dl


def _eval_inputs(case, seed):
    sc = _scene(case["gaussians"], case["width"], case["height"], case["views"], seed)
    return sc, _part_trained(sc, case["gaussians"], np.random.default_rng([seed, 4]))


def _photos(cameras, rng):
    """Smooth coloured photos (bytes) of the cameras' size."""
    out = []
    for c in cameras:
        y, x = np.mgrid[0:c.height, 0:c.width].astype(np.float32)
        f, p = rng.uniform(0.01, 0.1, (3, 2)), rng.uniform(0.0, 6.28, 3)
        rgb = np.stack([0.5 + 0.5 * np.sin(f[k, 0] * x + f[k, 1] * y + p[k]) for k in range(3)], axis=-1)
        out.append(TrainImage(c, TrainImage.quantize(rgb)))
    return out


def _mlp_inputs(case, seed):
    rng = np.random.default_rng([seed, 5])
    x = rng.normal(0.0, 1.0, (case["rows"], api.MLP_INPUTS)).astype(np.float32)
    x[:, 64:] = rng.uniform(0.0, 1.0, (case["rows"], api.MLP_INPUTS - 64))
    t = rng.normal(0.0, 0.5, (case["rows"], api.MLP_OUTPUTS)).astype(np.float32)
    p = rng.normal(0.0, 0.1, api.MLP_PARAMS).astype(np.float32)  # a trained network's weights
    return x, t, p


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        return dict(case=case, trainer=api.Trainer(*_training(case, seed)))
    if kind == "batch":
        return dict(case=case, batch=api.Batch([_training(c, seed + k) for k, c in
                                                enumerate(_batch_scenes(case, seed))], autotune=False))
    if kind == "eval":
        sc, model = _eval_inputs(case, seed)
        photos = _photos(sc.cameras, np.random.default_rng([seed, 6]))
        return dict(case=case, camera=sc.cameras[0],
                    trainer=api.Trainer(model, photos, sc.extent, _options(case, case["gaussians"])))
    if kind == "raster":
        model, cam, dl = _raster_inputs(case, seed)
        return dict(case=case, raster=api.Rasterizer(), model=model, camera=cam, dl=dl, settings=_settings(case))
    if kind == "views":
        sc = _scene(case["gaussians"], case["width"], case["height"], case["views"], seed, degree=case["degree"])
        return dict(case=case, scene=sc, settings=_settings(case))
    if kind == "warm":
        sc = _scene(max(case["points"], 10_000), case["width"], case["height"], case["views"], seed)
        pick = np.random.default_rng([seed, 7]).choice(sc.truth.size(), case["points"], replace=False)
        rgb = np.clip(0.5 + SH_C0 * sc.truth.colors[pick], 0.0, 1.0).astype(np.float32)
        return dict(case=case, xyz=sc.truth.means[pick], rgb=rgb, net=api.WarmStartNet(seed=seed),
                    images=_photos(sc.cameras, np.random.default_rng([seed, 8])))
    x, t, p = _mlp_inputs(case, seed)
    return dict(case=case, x=x, t=t, net=api.WarmStartNet(p))


# ---------------------------------------------------------------- one pass


def _groups(model):
    return {g: getattr(model, g) for g in GROUPS}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "train":
        t = state["trainer"]
        t.step(case["steps"])
        s = t.stats()
        return dict(model=_groups(t.model()), loss=np.float32(s.loss), psnr=np.float32(s.psnr))
    if kind == "batch":
        b = state["batch"]
        b.step(case["steps"])
        return [_groups(b.trainer(k).model()) for k in range(len(b))]
    if kind == "eval":
        t = state["trainer"]
        return dict(psnr=np.float32(t.evaluatePsnr()), image=t.render(state["camera"]))
    if kind == "raster":
        r, model = state["raster"], state["model"]
        out = dict(image=r.forward(model, state["camera"], state["settings"]))
        if case["backward"]:
            ndc = np.zeros(model.size(), np.float32)
            out["grads"] = _groups(r.backward(model, state["dl"], mean2d_grad_ndc=ndc))
            out["ndc"] = ndc
        return out
    if kind == "views":
        sc = state["scene"]
        rest = sc.sh_rest if case["degree"] > 0 else None
        return api.renderViewsSh(sc.truth, rest, case["degree"], sc.cameras, state["settings"])
    if kind == "warm":
        return _groups(api.warmstartInit(state["net"], state["xyz"], state["rgb"], state["images"]))
    loss, grad = state["net"].loss_grad(state["x"], state["t"])
    return dict(loss=np.float32(loss), grad=grad)


def work(case):
    """Bytes read and written once and the arithmetic of one pass. Compositing is counted as 40 blended
    Gaussians per pixel, 25 operations each forward and 60 backward; the loss as two separable 11-tap
    blurs of 5 and 3 maps per channel; projection and its chain rule as 400 operations per Gaussian each."""
    kind = case["kind"]

    def step(n, pixels):
        return 336 * n + 3 * pixels, 800 * n + pixels * (40 * 85 + 3 * 2 * 2 * 11 * 8)

    def forward(n, pixels):
        return 56 * n, 400 * n + pixels * 40 * 25

    if kind == "train":
        b, f = step(case["gaussians"], case["width"] * case["height"])
        return dict(bytes=case["steps"] * b + 56 * case["gaussians"], flops=case["steps"] * f)
    if kind == "batch":
        each = [step(c["gaussians"], c["width"] * c["height"]) + (56 * c["gaussians"],) for c in
                _batch_scenes(case, 0)]
        return dict(bytes=sum(case["steps"] * b + m for b, _, m in each), flops=case["steps"] * sum(f for _, f, _ in each))
    if kind == "eval":
        P = case["width"] * case["height"]
        b, f = forward(case["gaussians"], P)
        return dict(bytes=b + 3 * P * case["views"] + 12 * P, flops=(case["views"] + 1) * f)
    if kind == "raster":
        n, P = case["gaussians"], case["width"] * case["height"]
        b, f = forward(n, P)
        if not case["backward"]:
            return dict(bytes=b + 12 * P, flops=f)
        return dict(bytes=b + 24 * P + 56 * n + 4 * n, flops=f + 400 * n + P * 40 * 60)
    if kind == "views":
        n, P, K = case["gaussians"], case["width"] * case["height"], (case["degree"] + 1) ** 2 - 1
        b, f = forward(n, P)
        return dict(bytes=b + 12 * K * n + 3 * P * case["views"], flops=case["views"] * (f + 6 * K * n))
    if kind == "warm":
        n, P = case["points"], case["width"] * case["height"]
        return dict(bytes=24 * n + 56 * n + 3 * P * case["views"], flops=n * (2 * 51_712 + 27 * 16 * 8 + 40 * case["views"]))
    n = case["rows"]
    return dict(bytes=4 * n * (api.MLP_INPUTS + api.MLP_OUTPUTS) + 8 * api.MLP_PARAMS, flops=6 * n * 51_712)


# ---------------------------------------------------------------- 64-bit values


def _tensors(model):
    return {g: torch.from_numpy(np.ascontiguousarray(getattr(model, g))).to("cuda", torch.float64) for g in GROUPS}


def _project64(m, cam, st):
    """EWA projection of every Gaussian in 64 bits; `mean2d`, `conic`, `rgb`, `alpha` keep the graph."""
    R = torch.tensor(np.asarray(cam.R, np.float64), device="cuda")
    t = torch.tensor(np.asarray(cam.t, np.float64), device="cuda")
    pc = m["means"] @ R.T + t
    x, y, z = pc[:, 0], pc[:, 1], pc[:, 2]
    near = z >= st.near_plane
    z = torch.where(near, z, torch.ones_like(z))
    w, qx, qy, qz = (m["quats"] / m["quats"].norm(dim=1, keepdim=True)).unbind(1)
    rot = torch.stack([1 - 2 * (qy * qy + qz * qz), 2 * (qx * qy - w * qz), 2 * (qx * qz + w * qy),
                       2 * (qx * qy + w * qz), 1 - 2 * (qx * qx + qz * qz), 2 * (qy * qz - w * qx),
                       2 * (qx * qz - w * qy), 2 * (qy * qz + w * qx), 1 - 2 * (qx * qx + qy * qy)], 1).view(-1, 3, 3)
    M = rot * torch.exp(m["scales"])[:, None, :]
    sigma = M @ M.transpose(1, 2)
    W, H = float(cam.width), float(cam.height)
    ax, ay = 0.15 * W / cam.fx, 0.15 * H / cam.fy
    tx = z * torch.clamp(x / z, -(cam.cx / cam.fx + ax), (W - cam.cx) / cam.fx + ax)
    ty = z * torch.clamp(y / z, -(cam.cy / cam.fy + ay), (H - cam.cy) / cam.fy + ay)
    T0 = (cam.fx / z)[:, None] * R[0] - (cam.fx * tx / (z * z))[:, None] * R[2]
    T1 = (cam.fy / z)[:, None] * R[1] - (cam.fy * ty / (z * z))[:, None] * R[2]
    S0, S1 = (sigma @ T0[:, :, None])[:, :, 0], (sigma @ T1[:, :, None])[:, :, 0]
    a, b, c = (T0 * S0).sum(1) + st.eps2d, (T0 * S1).sum(1), (T1 * S1).sum(1) + st.eps2d
    det = a * c - b * b
    mean2d = torch.stack([cam.fx * x / z + cam.cx, cam.fy * y / z + cam.cy], 1)
    conic = torch.stack([c / det, -b / det, a / det], 1)
    with torch.no_grad():
        mid = 0.5 * (a + c)
        radius = torch.ceil(3.0 * torch.sqrt(mid + torch.sqrt(torch.clamp(mid * mid - det, min=0.1))))
        u, v, ts = mean2d[:, 0], mean2d[:, 1], st.tile_size
        tilesX, tilesY = -(-cam.width // ts), -(-cam.height // ts)
        x0 = torch.clamp(torch.floor((u - radius) / ts), min=0).long()
        y0 = torch.clamp(torch.floor((v - radius) / ts), min=0).long()
        x1 = torch.clamp(torch.floor((u + radius) / ts) + 1, max=tilesX).long()
        y1 = torch.clamp(torch.floor((v + radius) / ts) + 1, max=tilesY).long()
        seen = near & (det > 0) & (u + radius >= 0) & (v + radius >= 0) & (u - radius < W) & (v - radius < H)
        seen &= (x0 < x1) & (y0 < y1)
    return dict(mean2d=mean2d, conic=conic, rgb=torch.clamp(0.5 + SH_C0 * m["colors"], min=0.0),
                alpha=torch.sigmoid(m["opacities"]), depth=z.detach(), seen=seen, rect=(x0, y0, x1, y1),
                tiles=(tilesX, tilesY))


def _tile_lists(p):
    """(Gaussian ids sorted by tile, then depth; offsets per tile)."""
    x0, y0, x1, y1 = p["rect"]
    ids = torch.nonzero(p["seen"])[:, 0]
    ids = ids[torch.sort(p["depth"][ids], stable=True)[1]]
    wide, high = (x1 - x0)[ids], (y1 - y0)[ids]
    count = wide * high
    owner = torch.repeat_interleave(torch.arange(len(ids), device="cuda"), count)
    k = torch.arange(len(owner), device="cuda") - (torch.cumsum(count, 0) - count)[owner]
    tile = (y0[ids][owner] + k // wide[owner]) * p["tiles"][0] + x0[ids][owner] + k % wide[owner]
    order = torch.sort(tile, stable=True)[1]
    lengths = torch.bincount(tile, minlength=p["tiles"][0] * p["tiles"][1])
    return ids[owner[order]], lengths, torch.cumsum(lengths, 0) - lengths


def _render64(model, cam, st, dl=None):
    """The image in 64 bits and, for a given dL/dimage, the gradients of every group and the NDC statistic."""
    m = _tensors(model)
    if dl is not None:
        for v in m.values():
            v.requires_grad_(True)
    with torch.set_grad_enabled(dl is not None):
        p = _project64(m, cam, st)
    leaves = [p[k].detach().requires_grad_(dl is not None) for k in ("mean2d", "conic", "rgb", "alpha")]
    grads = [torch.zeros_like(v) for v in leaves]
    ids, lengths, starts = _tile_lists(p)
    ts, (tilesX, _) = st.tile_size, p["tiles"]
    H, W = cam.height, cam.width
    bg = torch.tensor(st.background, dtype=torch.float64, device="cuda")
    image = torch.zeros(H * W, 3, dtype=torch.float64, device="cuda")
    dl64 = None if dl is None else torch.from_numpy(dl).to("cuda", torch.float64).view(-1, 3)
    grid = torch.arange(ts, device="cuda")
    py, px = (g.reshape(-1) for g in torch.meshgrid(grid, grid, indexing="ij"))
    order = torch.sort(lengths, descending=True)[1].tolist()
    sizes = lengths.tolist()
    at = 0
    while at < len(order):  # tiles of like length together, padded to the longest
        L = max(sizes[order[at]], 1)
        some = torch.tensor(order[at: at + max(1, (1 << 15) * 256 // (L * ts * ts))], device="cuda")
        at += len(some)
        pos = torch.arange(L, device="cuda")
        real = pos[None, :] < lengths[some][:, None]
        g = ids[torch.clamp(starts[some][:, None] + pos, max=max(len(ids) - 1, 0))] if len(ids) else None
        X = (some % tilesX)[:, None] * ts + px
        Y = (some // tilesX)[:, None] * ts + py
        inside = (X < W) & (Y < H)
        pix = (Y * W + X)[inside]
        if g is None:
            image[pix] = bg
            continue
        with torch.set_grad_enabled(dl is not None):
            # The padded lists' values, gathered once so that backward adds them up per Gaussian.
            mean, con, col, al = (v[g] for v in leaves)
            dx, dy = mean[:, :, None, 0] - X[:, None, :], mean[:, :, None, 1] - Y[:, None, :]
            power = -0.5 * (con[:, :, None, 0] * dx * dx + con[:, :, None, 2] * dy * dy) - con[:, :, None, 1] * dx * dy
            alpha = torch.clamp(al[:, :, None] * torch.exp(torch.clamp(power, max=0.0)), max=0.99)
            ok = real[:, :, None] & (power <= 0) & (alpha >= st.min_alpha)
            rest = torch.log1p(-torch.where(ok, alpha, torch.zeros_like(alpha)))
            through = torch.cumsum(rest, 1)
            ok = ok & (through.detach() >= math.log(st.min_transmittance))
            rest = torch.where(ok, rest, torch.zeros_like(rest))
            through = torch.cumsum(rest, 1)
            weight = torch.where(ok, alpha, torch.zeros_like(alpha)) * torch.exp(through - rest)
            rgb = torch.einsum("tlp,tlc->tpc", weight, col) + torch.exp(through[:, -1])[:, :, None] * bg
        image[pix] = rgb.detach()[inside]
        if dl is not None:
            d = torch.autograd.grad((rgb[inside] * dl64[pix]).sum(), leaves)
            for total, one in zip(grads, d):
                total += one
    out = dict(image=image.view(H, W, 3).cpu().numpy())
    if dl is not None:
        back = torch.autograd.grad([p["mean2d"], p["conic"], p["rgb"], p["alpha"]], [m[k] for k in GROUPS],
                                   [torch.where(p["seen"].view(-1, *[1] * (g.dim() - 1)), g, torch.zeros_like(g))
                                    for g in grads])
        out["grads"] = {k: torch.where(p["seen"].view(-1, *[1] * (v.dim() - 1)), v, torch.zeros_like(v)).cpu().numpy()
                        for k, v in zip(GROUPS, back)}
        half = torch.tensor([0.5 * W, 0.5 * H], dtype=torch.float64, device="cuda")
        out["ndc"] = torch.where(p["seen"], (grads[0] * half).norm(dim=1), torch.zeros_like(p["depth"])).cpu().numpy()
    return out


def _mlp64(case, seed):
    x, t, p = (torch.from_numpy(a).to("cuda", torch.float64) for a in _mlp_inputs(case, seed))
    p.requires_grad_(True)
    at, h = 0, x
    widths = [api.MLP_INPUTS, 128, 128, 128, api.MLP_OUTPUTS]
    for k, (i, o) in enumerate(zip(widths[:-1], widths[1:])):
        h = h @ p[at: at + i * o].view(o, i).T + p[at + i * o: at + i * o + o]
        h = torch.relu(h) if k < 3 else h
        at += i * o + o
    w = torch.tensor([1, 1, 1, 0.5, 0.5, 0.5, 0.5, 0.25, 1, 1, 1], dtype=torch.float64, device="cuda")
    loss = (w * (h - t) ** 2).mean()
    loss.backward()
    return dict(loss=np.float64(loss.item()), grad=p.grad.cpu().numpy())


def exact(case, seed):
    """What run() returns, in 64 bits; None where there is no such value (whole training runs, quantised
    views, the initialisation's hash-grid neighbours)."""
    if case["kind"] == "raster":
        model, cam, dl = _raster_inputs(case, seed)
        return _render64(model, cam, _settings(case), dl if case["backward"] else None)
    if case["kind"] == "eval":
        sc, model = _eval_inputs(case, seed)
        return dict(psnr=None, image=_render64(model, sc.cameras[0], _settings(case))["image"])
    if case["kind"] == "mlp":
        return _mlp64(case, seed)
    return None
