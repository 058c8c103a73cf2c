"""The work this framework is used for, as cases that can be timed.

Every case goes through a public entry point: single frames through
``Rasterizer.forward`` (the fused FP16-SH pipeline, the drop-in default with
FP32 SH, and the staged pipeline), batches of views through ``Batcher``, a
request stream through ``Server``, training steps through ``render`` and
``render_views``, and the pair sort as an operator.  Scenes follow the
distributions of :mod:`polysplat_gb300.scenes` and are drawn on the GPU.

Sizes are those of the framework's own workloads and tests, odd image sizes
among them: 100 k to 20 M Gaussians, 800x600 to 7680x4320.
"""
import dataclasses
import math

import numpy as np
import torch

from polysplat_gb300 import Camera, Rasterizer, Scene, ops, scenes
from polysplat_gb300 import _lib as R
from polysplat_gb300.batch import Batcher, View, tiles_of
from polysplat_gb300.diff import render, render_views
from polysplat_gb300.rasterizer import E2E, LITE
from polysplat_gb300.serving import Server, TuneConfig

DEV = "cuda"
VARIANTS = {"e2e": E2E, "default": "default", "lite": LITE}


def listed():
    return [
        # a thumbnail-sized preview: launches and the host path count
        {"name": "e2e_100k_800x600", "kind": "frame", "scene": "plain", "gaussians": 100_000, "width": 800,
         "height": 600, "variant": "e2e"},
        # the headline frame: a trained scene's size at 1080p
        {"name": "e2e_3m_1080p", "kind": "frame", "scene": "clustered", "gaussians": 3_000_000, "width": 1920,
         "height": 1080, "variant": "e2e"},
        # the largest frame: a city at 8K, small Gaussians, the blend is half of it
        {"name": "e2e_20m_8k", "kind": "frame", "scene": "city", "gaussians": 20_000_000, "width": 7680,
         "height": 4320, "variant": "e2e"},
        # the drop-in default (FP32 SH) at a dataset's odd image size
        {"name": "default_1m_1237x823", "kind": "frame", "scene": "clustered", "gaussians": 1_000_003, "width": 1237,
         "height": 823, "variant": "default"},
        # the default on a large scene: its automatic choice is the depth-first pipeline
        {"name": "default_6m_1440p", "kind": "frame", "scene": "clustered", "gaussians": 6_000_000, "width": 2560,
         "height": 1440, "variant": "default"},
        # the staged pipeline: preprocess, sort, ranges and render as separate operators
        {"name": "lite_500k_1271x717", "kind": "frame", "scene": "plain", "gaussians": 500_000, "width": 1271,
         "height": 717, "variant": "lite"},
        # one batch of the serving layer: views of two scenes and four resolutions, quad keys, graph replay
        {"name": "batch_8_views", "kind": "batch", "gaussians_a": 500_000, "gaussians_b": 2_000_000, "views": 8,
         "first_resolution": 0},
        # a stream of requests over resident scenes, images delivered to host memory
        {"name": "serve_24_requests", "kind": "serve", "gaussians_a": 500_000, "gaussians_b": 2_000_000,
         "requests": 24},
        # a training step over eight cameras: forward, loss and every parameter's gradient
        {"name": "train_1m_8x720p", "kind": "train", "gaussians": 1_000_000, "width": 1280, "height": 720, "views": 8},
        # a training step of one camera on a small scene
        {"name": "train_100k_800x600", "kind": "train", "gaussians": 100_000, "width": 800, "height": 600,
         "views": 1},
        # the pair sort alone: one 1080p frame's 64-bit keys
        {"name": "sort_9m_1080p", "kind": "sort", "pairs": 9_208_343, "width": 1920, "height": 1080},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "batch", "serve", "train", "train", "sort"])
    if kind == "frame":
        variant = rng.choice(["e2e", "e2e", "default", "lite"])
        scene = rng.choice(["plain", "clustered", "clustered", "city"])
        width = _log_uniform(rng, 320, 7680 if scene == "city" else 3840)
        height = max(200, int(width * rng.choice([0.5625, 0.6667, 0.75])) + rng.randint(-7, 7))
        n = _log_uniform(rng, 50_000, 20_000_000 if scene == "city" else 6_000_000)
        if scene != "city":  # their keys grow with the pixels
            n = min(n, int(2.4e13 / (width * height)))
        if scene == "plain":
            n = min(n, 2_000_000)
        return {"kind": kind, "scene": scene, "gaussians": n, "width": width, "height": height, "variant": variant}
    if kind == "batch":
        return {"kind": kind, "gaussians_a": _log_uniform(rng, 50_000, 1_000_000),
                "gaussians_b": _log_uniform(rng, 200_000, 2_000_000), "views": rng.randint(2, 8),
                "first_resolution": rng.randint(0, 3)}
    if kind == "serve":
        return {"kind": kind, "gaussians_a": _log_uniform(rng, 50_000, 1_000_000),
                "gaussians_b": _log_uniform(rng, 200_000, 2_000_000), "requests": rng.randint(6, 24)}
    if kind == "train":
        width = _log_uniform(rng, 320, 1280)
        return {"kind": kind, "gaussians": _log_uniform(rng, 20_000, 1_000_000), "width": width,
                "height": max(200, int(width * rng.choice([0.5625, 0.6667, 0.75])) + rng.randint(-7, 7)),
                "views": rng.choice([1, 2, 4, 8])}
    width = _log_uniform(rng, 320, 3840)
    return {"kind": kind, "pairs": _log_uniform(rng, 100_000, 12_000_000), "width": width,
            "height": int(width * 0.5625) + rng.randint(0, 9)}


# --------------------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 2654435761 % (1 << 62) + 17)
    return g


def _raw(kind, n, seed):
    """Raw parameters on the GPU with the distributions of `scenes`:
    (means, log_scales, quats, logits, shs [n, 48])."""
    g, host = _gen(seed), np.random.Generator(np.random.PCG64(int(seed)))

    def randn(*s):
        return torch.randn(*s, device=DEV, generator=g)

    if kind == "plain":
        means = randn(n, 3) * (2.0 if n <= 200_000 else 3.0)
        log_scales = -3.5 + 0.5 * randn(n, 3)
    elif kind == "clustered":
        n_cl = int(round(n * 0.9))
        centres = torch.from_numpy(host.uniform(-10.0, 10.0, (64, 3))).float().to(DEV)
        sig = torch.from_numpy(host.uniform(0.1, 2.0, (64, 3))).float().to(DEV)
        which = torch.randint(0, 64, (n_cl,), device=DEV, generator=g)
        shell = torch.nn.functional.normalize(randn(n - n_cl, 3), dim=1) * 30.0
        means = torch.cat([centres[which] + randn(n_cl, 3) * sig[which], shell])
        chi2 = randn(n, 3).square_() + randn(n, 3).square_() + randn(n, 3).square_()
        log_scales = -4.0 + 0.6 * randn(n, 3) / torch.sqrt(chi2 / 3.0)  # Student t, 3 degrees of freedom
    else:  # city
        n_cl = min(n * 2 // 5, 4096 * 2000)

        def ground(k):
            xz = torch.rand(k, 2, device=DEV, generator=g) * 200.0 - 100.0
            y = 8.0 * torch.log(torch.rand(k, device=DEV, generator=g).clamp_min(1e-12))
            return torch.stack([xz[:, 0], y, xz[:, 1]], 1)

        centres = ground(4096)
        csig = torch.rand(4096, 1, device=DEV, generator=g) * 1.2 + 0.3
        which = torch.randint(0, 4096, (n_cl,), device=DEV, generator=g).sort()[0]
        means = torch.cat([ground(n - n_cl), centres[which] + randn(n_cl, 3) * csig[which]])
        log_scales = -4.5 + 0.7 * randn(n, 3)
    quats = torch.nn.functional.normalize(randn(n, 4), dim=1)
    logits = 1.5 * randn(n)
    shs = 0.05 * randn(n, 48)
    shs[:, :3] *= 10.0
    return means.contiguous(), log_scales.contiguous(), quats, logits, shs


def _scene(kind, n, seed, fp32):
    """A resident scene, as ``Scene.from_raw`` builds it."""
    means, log_scales, quats, logits, shs = _raw(kind, n, seed)
    s = Scene(DEV)
    s.num_vertex, s.position = n, means
    s.shs_half, s.shs = shs.half(), shs if fp32 else None
    s.opacity, s.cov3d = ops.prepare_scene(log_scales, quats, logits)
    return s


def _camera(kind, width, height, seed):
    rng = np.random.Generator(np.random.PCG64(int(seed) + 7))
    f = scenes.focal_for(width) if kind != "plain" else 0.75 * width
    if kind == "city":
        at = [rng.uniform(-10.0, 10.0), -25.0, -130.0]
        return Camera.from_spec(scenes.look_at(at, [0.0, -5.0, 0.0], width, height, 0.651 * width, 0.651 * width))
    return Camera.from_spec(scenes.orbit_camera(8.0 if kind == "clustered" else 9.0, rng.uniform(0, 2 * math.pi),
                                                rng.uniform(-0.3, 0.3), width, height, f))


def _capacity(case):
    """Key capacity a user of this scene and image size would choose."""
    per_g = 12.0 * case["width"] * case["height"] / (1920 * 1080) if case["scene"] != "city" else 4.0
    need = max(1 << 22, case["gaussians"] * max(per_g, 4.0))
    return min(1 << 28, 1 << math.ceil(math.log2(need)))


def _request_views(case, seed, count, first):
    """(arrival, scene, camera): orbits of the two scenes at the served
    resolutions, arriving at 240 requests per second."""
    rng = np.random.Generator(np.random.PCG64(int(seed) + 11))
    out, at = [], 0.0
    for k in range(count):
        at += rng.exponential(1.0 / 240.0)
        w, h = scenes.RESOLUTIONS[(first + k) % 4]
        spec = scenes.orbit_camera(rng.uniform(6.0, 12.0), rng.uniform(0, 2 * math.pi),
                                   rng.uniform(-math.pi / 6, math.pi / 6), w, h, scenes.focal_for(w), id=k)
        out.append((at, k // 2 % 2, spec))
    return out


def _train_inputs(case, seed):
    params = _raw("plain", case["gaussians"], seed)
    W, H, V = case["width"], case["height"], case["views"]
    specs = [scenes.orbit_camera(10.0, 2 * math.pi * (k + 0.1 * (seed % 7)) / max(V, 3), 0.1, W, H,
                                 scenes.focal_for(W), id=k) for k in range(V)]
    # photographs: smooth images with the scene's range of colours
    low = torch.rand(V, 3, 9, 16, device=DEV, generator=_gen(seed + 1))
    target = torch.nn.functional.interpolate(low, size=(H, W), mode="bilinear").permute(0, 2, 3, 1).contiguous()
    return params, specs, target


def prepare(case, seed):
    kind = case["kind"]
    if kind == "frame":
        scene = _scene(case["scene"], case["gaussians"], seed, case["variant"] == "default")
        cam = _camera(case["scene"], case["width"], case["height"], seed)
        tiles = tiles_of(cam)
        rast = Rasterizer(scene, _capacity(case), tiles)
        return {"kind": kind, "rast": rast, "scene": scene, "cam": cam, "bg": torch.zeros(3),
                "variant": VARIANTS[case["variant"]]}
    if kind == "batch":
        resident = [_scene("clustered", case["gaussians_a"], seed, False),
                    _scene("clustered", case["gaussians_b"], seed + 1, False)]
        views = [View(s, Camera.from_spec(c)) for _, s, c in _request_views(case, seed, case["views"],
                                                                            case["first_resolution"])]
        max_g = sum(resident[v.scene].num_vertex for v in views)
        b = Batcher(len(views), 1 << 25, max_g, sum(tiles_of(v.camera) for v in views))
        return {"kind": kind, "batcher": b, "scenes": resident, "views": views, "stream": torch.cuda.Stream()}
    if kind == "serve":
        resident = [_scene("clustered", case["gaussians_a"], seed, False),
                    _scene("clustered", case["gaussians_b"], seed + 1, False)]
        reqs = [scenes.Request(t, s, c) for t, s, c in _request_views(case, seed, case["requests"], 0)]
        config = TuneConfig(max_views=8, large_keys=1 << 40, massive_area=64, huge_area=4096,
                            max_batch_tiles=1 << 14, quad=True)
        srv = Server(resident, DEV, 12 << 30, config)
        return {"kind": kind, "server": srv, "requests": reqs}
    if kind == "train":
        params, specs, target = _train_inputs(case, seed)
        return {"kind": kind, "params": [p.requires_grad_(True) for p in params],
                "cams": [Camera.from_spec(c) for c in specs], "target": target}
    # sort: the pairs of one frame in emission order, a Gaussian's tiles together
    n, gx = case["pairs"], (case["width"] + 15) // 16
    tiles = gx * ((case["height"] + 15) // 16)
    g = _gen(seed)
    gid = torch.rand(n, device=DEV, generator=g).mul_(max(1, n // 5)).int().sort()[0]
    depth = torch.randn(n // 5 + 2, device=DEV, generator=g).mul_(4.0).add_(9.0).clamp_(0.21, 40.0)
    base = torch.randint(0, tiles, (n // 5 + 2,), device=DEV, generator=g)
    near = torch.randint(0, 3, (n,), device=DEV, generator=g) + gx * torch.randint(0, 3, (n,), device=DEV, generator=g)
    tile = (base[gid.long()] + near) % tiles
    keys = (tile << 32) | depth[gid.long()].view(torch.int32).long()
    return {"kind": kind, "n": n, "size": (case["width"], case["height"]), "keys": keys, "vals": gid,
            "ws": torch.zeros(ops.get_sort_buffer_size(n), dtype=torch.int8, device=DEV),
            "keys_out": torch.zeros_like(keys), "vals_out": torch.zeros_like(gid)}


# --------------------------------------------------------------------------- one pass
def run(state):
    kind = state["kind"]
    if kind == "frame":
        img, stats = state["rast"].forward(state["scene"], state["cam"], state["bg"], render_variant=state["variant"],
                                           return_stats=True)
        return {"image": img, "pairs": stats["num_rendered"]}
    if kind == "batch":
        b, s = state["batcher"], state["stream"]
        b.render(state["scenes"], state["views"], variant=R.RENDER_PERSISTENT_FUSED | R.QUAD_KEYS, stream=s)
        keys = b.finish(s)
        return {"images": [v.out for v in state["views"]], "keys": keys}
    if kind == "serve":
        srv, reqs = state["server"], state["requests"]
        for r in reqs:  # the client has read the images of the last pass
            srv.release(r)
        srv.run(reqs, realtime=False, deliver=True)
        return {"images": [r.host for r in reqs]}
    if kind == "train":
        params, cams = state["params"], state["cams"]
        for p in params:
            p.grad = None
        if len(cams) == 1:
            img = render(*params, cams[0])[None]
        else:
            img = render_views(*params, cams, stacked=True)
        loss = (img - state["target"]).square().mean()
        loss.backward()
        return {"image": img.detach(), "grads": [p.grad for p in params]}
    w, h = state["size"]
    ops.sort_gaussian(state["n"], w, h, 16, 16, state["ws"], state["keys"], state["vals"], state["keys_out"],
                      state["vals_out"])
    return {"keys": state["keys_out"], "vals": state["vals_out"]}


def work(case):
    """Each input read once and each output written once, and the arithmetic
    of every Gaussian's projection and colour."""
    kind = case["kind"]
    if kind == "frame":
        per_g = 40 + (192 if case["variant"] == "default" else 96)
        return {"bytes": case["gaussians"] * per_g + 3 * case["width"] * case["height"],
                "flops": 250 * case["gaussians"]}
    if kind in ("batch", "serve"):
        count = case["views"] if kind == "batch" else case["requests"]
        first = case["first_resolution"] if kind == "batch" else 0
        total = {"bytes": 0, "flops": 0}
        for k in range(count):
            n = case["gaussians_a"] if k // 2 % 2 == 0 else case["gaussians_b"]
            w, h = scenes.RESOLUTIONS[(first + k) % 4]
            total["bytes"] += 136 * n + 3 * w * h
            total["flops"] += 250 * n
        return total
    if kind == "train":
        pixels = case["views"] * case["width"] * case["height"]
        # parameters and their gradients; image, target and image gradient
        return {"bytes": 2 * 236 * case["gaussians"] + 3 * 12 * pixels,
                "flops": 1200 * case["gaussians"] * case["views"]}
    return {"bytes": 24 * case["pairs"], "flops": 0}


# --------------------------------------------------------------------------- 64-bit results
@dataclasses.dataclass
class _Features:
    xy: torch.Tensor     # [P,2] pixel centre
    con: torch.Tensor    # [P,4] conic in log2 units and log2 opacity
    rgb: torch.Tensor    # [P,3]
    depth: torch.Tensor  # [P]
    cov: torch.Tensor    # [P,3] 2D covariance (xx, xy, yy)
    opacity: torch.Tensor


def _project64(means, log_scales, quats, logits, shs, spec):
    """Raw parameters (float64) to screen-space features, as the 3DGS papers
    define them: EWA projection, +0.3 low pass, degree-3 SH, +0.5, clamp at 0."""
    W, H, fx, fy = spec.width, spec.height, spec.fx, spec.fy
    rot = torch.tensor(np.asarray(spec.rotation, np.float32), dtype=torch.float64, device=DEV)
    pos = torch.tensor(np.asarray(spec.position, np.float32), dtype=torch.float64, device=DEV)
    t = (means - pos) @ rot  # world to view: the transpose of camera-to-world
    tx, ty, tz = t.unbind(1)
    # clip w is the depth times zfar/(zfar - znear) folded out: x/w = x / z
    x = (2 * fx / W) * tx / (tz + 1e-7)
    y = (2 * fy / H) * ty / (tz + 1e-7)
    xy = torch.stack([((x + 1) * W - 1) / 2, ((y + 1) * H - 1) / 2], 1)
    limx, limy = 1.3 * W / (2 * fx), 1.3 * H / (2 * fy)
    cx, cy = (tx / tz).clamp(-limx, limx) * tz, (ty / tz).clamp(-limy, limy) * tz
    zero = torch.zeros_like(tz)
    J = torch.stack([torch.stack([fx / tz, zero, -fx * cx / tz ** 2], 1),
                     torch.stack([zero, fy / tz, -fy * cy / tz ** 2], 1)], 1)
    r, qx, qy, qz = (quats / quats.norm(dim=1, keepdim=True)).unbind(1)
    Rm = torch.stack([1 - 2 * (qy * qy + qz * qz), 2 * (qx * qy - r * qz), 2 * (qx * qz + r * qy),
                      2 * (qx * qy + r * qz), 1 - 2 * (qx * qx + qz * qz), 2 * (qy * qz - r * qx),
                      2 * (qx * qz - r * qy), 2 * (qy * qz + r * qx), 1 - 2 * (qx * qx + qy * qy)], 1).view(-1, 3, 3)
    A = (J @ rot.T) @ Rm * torch.exp(log_scales)[:, None, :]
    cov = A @ A.transpose(1, 2)
    a, b, c = cov[:, 0, 0] + 0.3, cov[:, 0, 1], cov[:, 1, 1] + 0.3
    det = a * c - b * b
    opacity = torch.sigmoid(logits)
    l2e = math.log2(math.e)
    con = torch.stack([-0.5 * l2e * c / det, l2e * b / det, -0.5 * l2e * a / det, torch.log2(opacity)], 1)
    d = means - pos
    x, y, z = (d / d.norm(dim=1, keepdim=True)).unbind(1)
    xx, yy, zz = x * x, y * y, z * z
    basis = torch.stack([
        0.28209479177387814 * torch.ones_like(x), -0.4886025119029199 * y, 0.4886025119029199 * z,
        -0.4886025119029199 * x, 1.0925484305920792 * x * y, -1.0925484305920792 * y * z,
        0.31539156525252005 * (2 * zz - xx - yy), -1.0925484305920792 * x * z, 0.5462742152960396 * (xx - yy),
        -0.5900435899266435 * y * (3 * xx - yy), 2.890611442640554 * x * y * z,
        -0.4570457994644658 * y * (4 * zz - xx - yy), 0.3731763325901154 * z * (2 * zz - 3 * xx - 3 * yy),
        -0.4570457994644658 * x * (4 * zz - xx - yy), 1.445305721320277 * z * (xx - yy),
        -0.5900435899266435 * x * (xx - 3 * yy)], 1)
    rgb = (torch.einsum("pk,pkc->pc", basis, shs.view(-1, 16, 3)) + 0.5).clamp_min(0.0)
    return _Features(xy, con, rgb, tz, torch.stack([a, b, c], 1), opacity)


def _tile_lists64(f, W, H):
    """Per 16x16 tile the Gaussians that reach it, front to back:
    (sorted Gaussian ids, start of each tile, gx)."""
    gx, gy = (W + 15) // 16, (H + 15) // 16
    a, b, c = f.cov.unbind(1)
    det = a * c - b * b
    power = math.log(2.0) * (8.0 + torch.log2(f.opacity))
    keep = (f.depth > 0.2) & ~((2 * det * power < 0.09 * (a + c)) & (f.opacity < 0.5))
    rx = torch.floor(1.414214 * torch.sqrt((a * power).clamp_min(0)) + 1.0)
    ry = torch.floor(1.414214 * torch.sqrt((c * power).clamp_min(0)) + 1.0)
    x0 = torch.trunc((f.xy[:, 0] - rx) / 16).clamp(0, gx).long()
    y0 = torch.trunc((f.xy[:, 1] - ry) / 16).clamp(0, gy).long()
    x1 = (torch.trunc((f.xy[:, 0] + rx) / 16) + 1).clamp(0, gx).long()
    y1 = (torch.trunc((f.xy[:, 1] + ry) / 16) + 1).clamp(0, gy).long()
    area = torch.where(keep, (x1 - x0) * (y1 - y0), 0).clamp_min(0)
    g = torch.repeat_interleave(torch.arange(area.numel(), device=DEV), area)
    k = torch.arange(g.numel(), device=DEV) - (area.cumsum(0) - area)[g]
    wd = (x1 - x0)[g]
    tx, ty = x0[g] + k % wd, y0[g] + k // wd
    lx, ly = tx * 16.0, ty * 16.0
    cx, cy = f.xy[g, 0], f.xy[g, 1]
    ca, cb, cc = (c / det)[g], (-b / det)[g], (a / det)[g]
    w = 2 * power[g]

    def edge(A, B, C, near, ctr, lo, hi):  # the ellipse meets the segment of the nearer edge
        qa, qb, qc = C, -2 * B * near, A * near * near - w
        delta = qb * qb - 4 * qa * qc
        t1, t2 = (lo - ctr) * 2 * qa + qb, (hi - ctr) * 2 * qa + qb
        return (delta >= 0) & ((t1 <= 0) | (t1 * t1 <= delta)) & ((t2 >= 0) | (t2 * t2 <= delta))

    dx = cx - torch.where(2 * cx < 2 * lx + 15, lx, lx + 15)
    dy = cy - torch.where(2 * cy < 2 * ly + 15, ly, ly + 15)
    inside = (cx >= lx) & (cx <= lx + 15) & (cy >= ly) & (cy <= ly + 15)
    hit = inside | ((w > 0) & (edge(ca, cb, cc, dx, cy, ly, ly + 15) | edge(cc, cb, ca, dy, cx, lx, lx + 15)))
    g, tile = g[hit], (ty * gx + tx)[hit]
    order = torch.argsort(f.depth[g], stable=True)
    g, tile = g[order], tile[order]
    order = torch.argsort(tile, stable=True)
    g, tile = g[order], tile[order]
    return g, torch.searchsorted(tile, torch.arange(gx * gy + 1, device=DEV)), gx


@torch.no_grad()
def _view64(f, spec, target, count):
    """Image of one view and the feature gradients of its share of the mean
    squared error over `count` values.  A tile stops when, at a multiple of 8
    Gaussians, every pixel's transmittance is below 1e-4."""
    W, H = spec.width, spec.height
    ids, starts, gx = _tile_lists64(f, W, H)
    tiles = starts.numel() - 1
    P = f.depth.numel()
    feat = torch.cat([f.xy, f.con, f.rgb], 1)
    grad = torch.zeros(P + 1, 9, dtype=torch.float64, device=DEV)
    feat = torch.cat([feat, torch.tensor([[0, 0, 0, 0, 0, -1e30, 0, 0, 0]], dtype=torch.float64, device=DEV)])
    image = torch.zeros(((H + 15) // 16) * 16, gx * 16, 3, dtype=torch.float64, device=DEV)
    padded = torch.zeros_like(image)
    padded[:H, :W] = target
    py, px = torch.meshgrid(torch.arange(16, device=DEV), torch.arange(16, device=DEV), indexing="ij")

    def listing(t, lo, hi):  # [T, hi - lo] ids of list positions lo.., P where the list has ended
        k = starts[t][:, None] + torch.arange(lo, hi, device=DEV)
        return torch.where(k < starts[t + 1][:, None], ids[k.clamp_max(max(0, ids.numel() - 1))], P)

    def alphas(t, g):  # [T, L, 256]
        ox, oy = (t % gx * 16)[:, None] + px.reshape(-1), (t // gx * 16)[:, None] + py.reshape(-1)
        v = feat[g]
        dx, dy = v[..., 0, None] - ox[:, None], v[..., 1, None] - oy[:, None]
        power = v[..., 5, None] + v[..., 2, None] * dx * dx + v[..., 4, None] * dy * dy + v[..., 3, None] * dx * dy
        return torch.exp2(power), dx, dy, v

    lengths = starts[1:] - starts[:-1]
    used = torch.zeros_like(lengths)
    for chunk in torch.argsort(lengths).split(1024):
        live = chunk
        T = torch.ones(chunk.numel(), 256, dtype=torch.float64, device=DEV)
        lo = 0
        while live.numel():
            a = alphas(live, listing(live, lo, lo + 8))[0]
            T = T * (1 - a).prod(1)
            lo += 8
            used[live] = torch.minimum(lengths[live], torch.tensor(lo, device=DEV))
            more = (lengths[live] > lo) & ~(T < 1e-4).all(1)
            live, T = live[more], T[more]
    order = torch.argsort(used)
    sizes = used[order].clamp_min(1).tolist()
    at = 0
    while at < tiles:
        end = at + 1
        while end < tiles and (end + 1 - at) * sizes[end] * 256 <= 12_000_000:
            end += 1
        t, L = order[at:end], sizes[end - 1]
        g = listing(t, 0, L)
        g = torch.where(torch.arange(L, device=DEV) < used[t][:, None], g, P)
        a, dx, dy, v = alphas(t, g)
        T = torch.cumprod(1 - a, 1)
        before = torch.cat([torch.ones_like(T[:, :1]), T[:, :-1]], 1)
        wgt = a * before
        col = v[..., 6:9]
        C = torch.einsum("tlp,tlc->tpc", wgt, col)  # the background is black
        rows, cols = (t // gx * 16)[:, None] + py.reshape(-1), (t % gx * 16)[:, None] + px.reshape(-1)
        image[rows, cols] = C
        inside = ((rows < H) & (cols < W))[..., None]
        G = torch.where(inside, 2.0 * (C - padded[rows, cols]) / count, 0.0)
        cg = torch.einsum("tlc,tpc->tlp", col, G)
        s = wgt * cg
        behind = s.flip(1).cumsum(1).flip(1) - s
        dp = (before * cg - behind / (1 - a)) * a * math.log(2.0)
        out = torch.stack([(dp * (2 * v[..., 2, None] * dx + v[..., 3, None] * dy)).sum(2),
                           (dp * (2 * v[..., 4, None] * dy + v[..., 3, None] * dx)).sum(2),
                           (dp * dx * dx).sum(2), (dp * dx * dy).sum(2), (dp * dy * dy).sum(2), dp.sum(2)], 2)
        out = torch.cat([out, torch.einsum("tlp,tpc->tlc", wgt, G)], 2)
        grad.index_add_(0, g.reshape(-1), out.reshape(-1, 9))
        at = end
    return image[:H, :W], grad[:P]


def exact(case, seed):
    """What `run` returns in 64 bits: the training steps' images and gradients
    and the sorted pairs.  A frame's outputs are bytes and counts whose
    rounding follows the 32-bit arithmetic: they have no 64-bit value."""
    if case["kind"] == "sort":
        st = prepare(case, seed)
        w, h = st["size"]
        bits = 32 + (((w + 15) // 16) * ((h + 15) // 16)).bit_length()
        order = torch.argsort(st["keys"] & ((1 << bits) - 1), stable=True)
        return {"keys": st["keys"][order], "vals": st["vals"][order]}
    if case["kind"] != "train":
        return None
    params, specs, target = _train_inputs(case, seed)
    leaves = [p.double().requires_grad_(True) for p in params]
    images = []
    for k, spec in enumerate(specs):
        f = _project64(*leaves, spec)
        img, grad = _view64(f, spec, target[k].double(), target.numel())
        images.append(img)
        seen = grad.abs().sum(1) > 0
        out = torch.cat([f.xy, f.con, f.rgb], 1)
        (out[seen] * grad[seen]).sum().backward()
    return {"image": torch.stack(images), "grads": [p.grad for p in leaves]}
