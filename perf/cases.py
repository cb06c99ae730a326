"""What a user of this framework has it do, as cases that can be timed and compared.

Every case goes through `vet_b200.render.Rasterizer`, the host side of the C ABI, the way a training loop or a viewer
does.  The kinds:

  frame    one call of the rasterizer without gradients (a viewer, an evaluation render)
  step     forward, L1 loss against a target pyramid and its gradient, backward, gradient epilogue (a training batch)
  envmap   the texture environment map behind rendered images, and its parameter gradients
  errgrid  the error-grid rasterisation of one training image at the end of an epoch
  surgery  point removal from all per-point tensors, then the drop-out radius of what is left

`listed()` gives the cases, `draw()` more of the same ranges: clouds of 5 thousand to 20 million points, images of
96 x 64 to 1920 x 1080 pixels (odd sizes among them), 1 to 8 views, 3 to 5 pyramid levels, 3 or 4 descriptor channels, all
four blend modes (1 is the code's default, 3 the mode of shipped configurations, 0 and 2 are its options), with and without
camera gradients and point drop-out.  Points are at most ten per pixel of the full-size image, as in captured scenes.
Everything is synthetic and made on the GPU from the seed.
"""
import math

import numpy as np
import torch

from vet_b200.render import Rasterizer, default_params, level_sizes
from vet_b200.scenes import View, look_at_pose, orbit_poses

DEVICE = 0


def _step(name, points, w, h, views, mode, cloud="planar", layers=4, channels=4, cameras=False, drop=0.0):
    return dict(name=name, kind="step", points=points, w=w, h=h, views=views, mode=mode, cloud=cloud, layers=layers,
                channels=channels, cameras=cameras, drop=drop)


def _frame(name, points, w, h, mode, cloud="planar", layers=4, channels=4):
    return dict(name=name, kind="frame", points=points, w=w, h=h, views=1, mode=mode, cloud=cloud, layers=layers,
                channels=channels, cameras=False, drop=0.0)


def listed():
    return [
        # the smallest training batch: a toy scene, two small views, pose and intrinsics refined too; launches and host time
        _step("step_small", 5_000, 96, 64, 2, 1, cloud="cube", cameras=True),
        # an object scan at the crop size of a training loop (the first benchmark configuration)
        _step("step_crop_512", 100_000, 512, 512, 1, 1, cloud="cube"),
        # a viewer frame of a captured scene (the second benchmark configuration)
        _frame("frame_1080p", 3_000_000, 1920, 1080, 1),
        # a training batch with camera refinement (the third benchmark configuration)
        _step("step_batch4", 8_000_000, 1024, 768, 4, 1, cameras=True),
        # one launch group of the largest batch (the fifth benchmark configuration: 20 M points, full-HD views)
        _step("step_largest", 20_000_000, 1920, 1080, 8, 1),
        # the mode of shipped configurations: a viewer frame with three channels, and a training batch of odd-sized images
        _frame("frame_bilinear", 1_000_000, 1280, 720, 3, channels=3),
        _step("step_bilinear_odd", 3_000_001, 1237, 823, 2, 3, cameras=True),
        # the remaining two blend modes, at the odd sizes that cropping leaves; mode 0 with point drop-out
        _step("step_fuzzy_odd", 1_000_003, 801, 603, 1, 2),
        _step("step_depth_test", 2_000_000, 1280, 720, 2, 0, drop=0.1),
        # the environment map behind one full-HD training image: four spheres of 1024 x 1024 texels, all pyramid levels
        dict(name="envmap_1080p", kind="envmap", w=1920, h=1080, views=1, layers=4, channels=4, spheres=4, resolution=1024),
        # error grid of 128^3 cells, one full-HD image: once per training image at the end of an epoch
        dict(name="errgrid_128", kind="errgrid", w=1920, h=1080, cells=128, channels=3),
        # point surgery between epochs: a twentieth of the cloud goes, the radius column is formed anew
        dict(name="surgery_4m", kind="surgery", points=4_000_000, channels=4, removed=0.05, neighbours=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _image_size(rng):
    w = _log_int(rng, 96, 1920)
    return w, max(64, min(1080, int(round(w * rng.choice((9 / 16, 2 / 3, 3 / 4, 1.0))))))


def draw(rng):
    kind = rng.choices(("step", "frame", "envmap", "errgrid", "surgery"), (10, 5, 2, 2, 2))[0]
    w, h = _image_size(rng)
    channels = rng.choice((3, 4, 4))
    if kind == "envmap":
        return dict(kind=kind, w=w, h=h, views=rng.randint(1, 2), layers=rng.choice((3, 4, 4, 5)), channels=channels,
                    spheres=rng.randint(2, 4), resolution=_log_int(rng, 128, 1024))
    if kind == "errgrid":
        return dict(kind=kind, w=max(w, 160), h=max(h, 120), cells=_log_int(rng, 16, 128), channels=channels)
    if kind == "surgery":
        return dict(kind=kind, points=_log_int(rng, 20_000, 8_000_000), channels=channels, removed=rng.uniform(0.005, 0.3),
                    neighbours=rng.choice((4, 4, 4, 8)))
    mode = rng.choices((0, 1, 2, 3), (2, 9, 2, 7))[0]
    views = 1 if kind == "frame" else rng.choice((1, 1, 2, 3, 4, 8))
    most = {0: 40_000_000, 1: 160_000_000, 2: 8_000_000, 3: 24_000_000}[mode] // views
    points = min(_log_int(rng, 5_000, 20_000_000), 10 * w * h, most)
    return dict(kind=kind, points=points, w=w, h=h, views=views, mode=mode, cloud=rng.choice(("planar", "planar", "cube")),
                layers=rng.choice((3, 4, 4, 4, 5)), channels=channels, cameras=kind == "step" and rng.random() < 0.5,
                drop=0.1 if kind == "step" and rng.random() < 0.2 else 0.0)


# ---------------------------------------------------------------------------------------------------------------------
# inputs


def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed) & 0x7FFFFFFF)


def _uniform(gen, *shape, lo=0.0, hi=1.0):
    return torch.rand(*shape, generator=gen, device=DEVICE) * (hi - lo) + lo


def _normal(gen, *shape):
    return torch.randn(*shape, generator=gen, device=DEVICE)


def _spread_bits(v):
    """Puts two zero bits between the 21 bits of v (for a Morton code)."""
    for shift, mask in ((32, 0x1F00000000FFFF), (16, 0x1F0000FF0000FF), (8, 0x100F00F00F00F00F), (4, 0x10C30C30C30C30C3),
                        (2, 0x1249249249249249)):
        v = (v | (v << shift)) & mask
    return v


def _prepared_order(xyz, gen, block=256):
    """The order of a prepared cloud: by Morton code, then whole blocks of 256 points shuffled (vet_b200.scenes does the
    same on the host)."""
    lo = xyz.amin(0)
    q = ((xyz - lo) / (xyz.amax(0) - lo).clamp_min(1e-9) * (2 ** 21 - 1)).long().clamp_(0, 2 ** 21 - 1)
    order = torch.argsort(_spread_bits(q[:, 0]) | (_spread_bits(q[:, 1]) << 1) | (_spread_bits(q[:, 2]) << 2))
    n = xyz.shape[0]
    blocks = torch.randperm((n + block - 1) // block, generator=gen, device=DEVICE)
    at = (blocks[:, None] * block + torch.arange(block, device=DEVICE)).reshape(-1)
    return order[at[at < n]]


def _cloud(kind, n, gen, host):
    """Positions and drop-out radius [n,4] in the order of a prepared cloud.  "planar": 40 random rectangles in a 20-unit box
    and 5 % outliers; "cube": the surface of the unit cube.  The radius is a neighbour distance (from the known density)
    scaled by sqrt(1 / u), u uniform."""
    if kind == "cube":
        face = torch.randint(0, 6, (n,), generator=gen, device=DEVICE)
        xyz = _uniform(gen, n, 3, lo=-0.5, hi=0.5)
        xyz.scatter_(1, (face // 2)[:, None], torch.where(face % 2 == 0, -0.5, 0.5)[:, None])
        xyz += 0.005 * _normal(gen, n, 3)
        distance = torch.full((n,), math.sqrt(4.0 / (math.pi * n / 6.0)), device=DEVICE)
    else:
        outliers = int(round(n * 0.05))
        m = n - outliers
        ext = host.uniform(2.0, 10.0, (40, 2))
        area = ext[:, 0] * ext[:, 1]
        centre = host.uniform(-7.0, 7.0, (40, 3))
        basis = np.stack([np.linalg.qr(host.normal(size=(3, 3)))[0] for _ in range(40)])
        counts = np.floor(area / area.sum() * m).astype(np.int64)
        counts[0] += m - counts.sum()
        on = lambda a: torch.as_tensor(a, dtype=torch.float32, device=DEVICE)  # noqa: E731
        plane = torch.repeat_interleave(torch.arange(40, device=DEVICE), torch.as_tensor(counts, device=DEVICE))
        uv = _uniform(gen, m, 2, lo=-0.5, hi=0.5) * on(ext)[plane]
        xyz = on(centre)[plane] + uv[:, :1] * on(basis[:, :, 0])[plane] + uv[:, 1:] * on(basis[:, :, 1])[plane]
        xyz += 0.01 * _normal(gen, m, 3)
        distance = on(np.sqrt(4.0 * area / (math.pi * counts.clip(1))))[plane]
        if outliers:
            xyz = torch.cat([xyz, _uniform(gen, outliers, 3, lo=-10.0, hi=10.0)])
            far = (3.0 / (math.pi * outliers / 8000.0)) ** (1.0 / 3.0)
            distance = torch.cat([distance, torch.full((outliers,), far, device=DEVICE)])
    position = torch.empty(n, 4, device=DEVICE)
    position[:, :3] = xyz
    position[:, 3] = distance * torch.rsqrt(_uniform(gen, n, lo=1e-3, hi=1.0))
    return position[_prepared_order(xyz, gen)].contiguous()


def _cameras(case, host, cloud="planar"):
    """Poses on an orbit around the scene and one pinhole camera: (poses [n,8] f64, intrinsics [1,13], views)."""
    w, h, n = case["w"], case["h"], case.get("views", 1)
    if cloud == "cube":
        poses = np.stack([look_at_pose(3.0 * np.array([math.cos(e) * math.cos(a), -math.sin(e), math.cos(e) * math.sin(a)]), (0, 0, 0))
                          for a, e in zip(host.uniform(0, 2 * math.pi, n), host.uniform(0.2, 0.6, n))])
        focal = 450.0 / 512.0 * min(w, h)
    else:
        poses, focal = orbit_poses(host, n, 9.0), 0.625 * w
    intrinsics = np.zeros((1, 13), dtype=np.float32)
    intrinsics[0, :4] = focal, focal, w / 2, h / 2
    return (torch.as_tensor(poses, device=DEVICE).contiguous(), torch.as_tensor(intrinsics, device=DEVICE),
            [View(w, h, image_index=i) for i in range(n)])


def prepare(case, seed):
    torch.cuda.set_device(DEVICE)
    gen, host = _generator(seed), np.random.default_rng(seed)
    s = dict(case=case, rast=Rasterizer(DEVICE))
    kind = case["kind"]
    if kind in ("step", "frame"):
        n, c = case["points"], case["channels"]
        s["position"] = _cloud(case["cloud"], n, gen, host)
        s["index"] = torch.arange(n, dtype=torch.int32, device=DEVICE)
        s["texture"] = _normal(gen, c, n)
        # opacities of a trained cloud spread over (0, 1); those of a fresh scan are saturated: sigmoid(10 x), x in (-2, 2)
        s["confidence"] = torch.sigmoid(10.0 * _uniform(gen, n, lo=-2.0, hi=2.0)) if case["cloud"] == "cube" else _uniform(gen, n)
        s["background"] = torch.full((c,), -1.0, device=DEVICE)
        s["poses"], s["intrinsics"], s["views"] = _cameras(case, host, case["cloud"])
        s["params"] = default_params(render_mode=case["mode"], num_layers=case["layers"], num_channels=c)
        s["dropout"] = (_uniform(gen, case["views"], n) < case["drop"]).float() if case["drop"] else None
        if kind == "step":
            sizes = level_sizes(case["w"], case["h"], case["layers"])
            s["targets"] = [_uniform(gen, case["views"], c, h, w) for w, h in sizes]
            s["grads"] = [torch.empty(case["views"], c, h, w, device=DEVICE) for w, h in sizes]
            s["loss"] = torch.zeros((), device=DEVICE)
    elif kind == "envmap":
        c, ns, r = case["channels"], case["spheres"], case["resolution"]
        s["poses"], s["intrinsics"], s["views"] = _cameras(case, host)
        s["density"] = _normal(gen, ns, r, r)
        s["color"] = _uniform(gen, c, ns, r, r)
        s["radii"] = [20.0 * 5.0 ** i for i in range(ns)]
        sizes = level_sizes(case["w"], case["h"], case["layers"])
        # what the blend leaves of a pixel: one factor per fragment of its list; a quarter of the pixels are empty
        deep = [torch.randint(-2, 7, (case["views"], 1, h, w), generator=gen, device=DEVICE).clamp_min_(0) for w, h in sizes]
        s["weight"] = [_uniform(gen, *d.shape).pow(d) for d in deep]
        s["grads"] = [_normal(gen, case["views"], c, h, w) for w, h in sizes]
    elif kind == "errgrid":
        s["poses"], s["intrinsics"], s["views"] = _cameras(case, host)
        k = case["cells"]
        a = torch.arange(k, device=DEVICE, dtype=torch.float32) * (20.0 / k) - 10.0
        s["cell_min"] = torch.stack(torch.meshgrid(a, a, a, indexing="ij"), -1).reshape(-1, 3).contiguous()
        s["cell_len"] = torch.full_like(s["cell_min"], 20.0 / k)
        s["error"] = _uniform(gen, case["channels"], case["h"], case["w"])
    else:
        n, c = case["points"], case["channels"]
        s["position"] = _cloud("planar", n, gen, host)
        s["index"] = torch.arange(n, dtype=torch.int32, device=DEVICE)[:, None].contiguous()
        # descriptors, confidences and their optimizer moments
        s["per_point"] = [_normal(gen, c, n), _uniform(gen, 1, n), _normal(gen, c, n), _normal(gen, c, n), _normal(gen, 1, n),
                          _normal(gen, 1, n)]
        s["remove"] = torch.randperm(n, generator=gen, device=DEVICE)[:max(1, int(n * case["removed"]))].contiguous()
    return s


def run(s):
    case, rast = s["case"], s["rast"]
    kind = case["kind"]
    if kind in ("step", "frame"):
        out = rast.forward(s["position"], s["index"], s["texture"], s["confidence"], s["background"], s["poses"],
                           s["intrinsics"], s["views"], s["params"], dropout=s["dropout"], want_weight=True,
                           want_depth=kind == "frame")
        if kind == "frame":
            return dict(color=out["color"], weight=out["weight"], depth=out["depth"])
        rast.l1_loss_grad(out["color"], s["targets"], s["grads"], s["loss"])
        raw = rast.backward_raw(s["grads"], want_points=True, want_pose=case["cameras"], want_intrinsics=case["cameras"])
        return dict(color=out["color"], weight=out["weight"], loss=s["loss"], **rast.finalize(raw))
    if kind == "envmap":
        # flag 8: the cameras have no distortion (the caller vouches for it)
        where = (s["poses"], s["intrinsics"], s["views"], case["layers"], s["density"], s["color"], s["radii"], s["weight"])
        images = rast.envmap_forward(*where, flags=8)
        g_density, g_color = rast.envmap_backward(*where, s["grads"], flags=8)
        return dict(images=images, density=g_density, color=g_color)
    if kind == "errgrid":
        value = torch.zeros(s["cell_min"].shape[0], device=DEVICE)
        count = torch.zeros(s["cell_min"].shape[0], dtype=torch.int32, device=DEVICE)
        rast.grid_loss(s["poses"], s["intrinsics"], s["views"][0], s["cell_min"], s["cell_len"], s["error"], value, count)
        return dict(value=value, count=count)
    new_index, per_point, (position, index) = rast.remove_points(case["points"], s["remove"], s["per_point"],
                                                                 [s["position"], s["index"]])
    rast.knn_radius(position, case["neighbours"], out="w")
    return dict(new_index=new_index, per_point=per_point, position=position, index=index)


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without


def work(case):
    """Every input read once and every output written once; operations of the parts that no shortcut avoids."""
    kind = case["kind"]
    if kind == "surgery":
        n, rows = case["points"], 3 * case["channels"] + 3
        kept = n - max(1, int(n * case["removed"]))
        # six per-point arrays, position and index in and out, the list in, the new index out; per neighbour candidate
        # (about 27 for a 3^3 search at one point per cell) one squared distance
        return {"bytes": 4 * (n + kept) * (rows + 5) + 8 * (n - kept) + 4 * n, "flops": 27 * 8 * kept}
    if kind == "errgrid":
        cells = case["cells"] ** 3
        # eight corner projections of about 40 operations per cell; the pixels under a cell depend on the camera
        return {"bytes": cells * (24 + 8) + 4 * case["channels"] * case["w"] * case["h"], "flops": cells * 8 * 40}
    pixels = case["views"] * sum(w * h for w, h in level_sizes(case["w"], case["h"], case["layers"]))
    c = case["channels"]
    if kind == "envmap":
        texels = case["spheres"] * case["resolution"] ** 2 * (c + 1)
        # transmittance and gradient in, image out; textures read, their gradients written; per pixel and sphere one
        # intersection (about 60) and eight taps per plane in each direction
        return {"bytes": 4 * pixels * (1 + 2 * c) + 4 * 2 * texels, "flops": pixels * case["spheres"] * 2 * (60 + 16 * (c + 1))}
    n = case["points"]
    inputs = n * (16 + 4 + 4 + 4 * c) + (4 * case["views"] * n if case["drop"] else 0)
    # one projection of about 40 operations per point and view
    if kind == "frame":
        return {"bytes": inputs + 4 * pixels * (c + 2), "flops": 40 * n * case["views"]}
    # images, weight, target pyramid; gradients of descriptors, confidence and position
    return {"bytes": inputs + 4 * pixels * (2 * c + 1) + n * (4 * c + 4 + 16), "flops": 2 * 40 * n * case["views"]}


def tolerance(case):
    # fp32 throughout; sums over fragments, pixels and corners in no fixed order.  The environment map's sample coordinates
    # are fp32 numbers as large as the resolution: half a unit of theirs is resolution x 2^-24 of a texel.  Whole numbers
    # (hit counts, covered pixels, indices) are exact.
    if case["kind"] == "envmap":
        return {"rel": 1e-4}
    return {"rel": 1e-5}
