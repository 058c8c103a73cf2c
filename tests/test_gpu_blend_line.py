"""Renders on either side of the line between a tile per CTA and a tile per warp
(16 tiles per SM of the device), each side's tile count checked: bytes of the
forward render on the same sorted lists, and the training render's float image
of one camera against the same camera repeated until its tiles pass the line.
The training scene has no two equal depths, so its lists have one order."""
import numpy as np
import pytest
import torch

from polysplat_gb300 import Camera, Rasterizer, Scene, ops, scenes
from polysplat_gb300.diff import render, render_views

pytestmark = pytest.mark.gpu


def _line(dev):
    return 16 * torch.cuda.get_device_properties(dev).multi_processor_count


def _tiles(w, h):
    return ((w + 15) // 16) * ((h + 15) // 16)


@pytest.mark.parametrize("W,H", [(637, 351), (17, 250)])
def test_forward(cuda_device, W, H):
    raw = scenes.subsample(scenes.scene_clustered(600_000, seed=1), 40_000, seed=2)
    scene = Scene.from_raw(raw, cuda_device)
    cam = Camera.from_spec(scenes.orbit_camera(8.0, 0.5, 0.1, W, H, scenes.focal_for(W)))
    line, gx = _line(cuda_device), (W + 15) // 16
    tall = 16 * (line // gx + 1)
    assert _tiles(W, H) <= line < _tiles(W, tall)
    rast = Rasterizer(scene, 1 << 22, 1 << 16)
    bg = torch.tensor([0.2, 0.1, 0.4])
    _, st = rast.forward(scene, cam, bg, render_variant="preranges_smem_persistent_lite", return_stats=True)
    n, images = st["num_rendered"], []
    for h in (H, tall):
        ranges = torch.full((_tiles(W, h), 2), n, dtype=torch.int32, device=cuda_device)
        ranges[:_tiles(W, H)] = rast.tile_ranges_buf[:_tiles(W, H)]
        out = torch.zeros((h, W, 3), dtype=torch.uint8, device=cuda_device)
        ops.render_16x16_preranges_smem_persistent_lite(n, W, h, rast.points_xy, rast.rgb_depth, rast.conic_opacity,
                                                        rast.gaussian_values_sorted, ranges, bg, out)
        images.append(out)
    assert torch.equal(images[0], images[1][:H])


@pytest.mark.parametrize("quad", [True, False])
def test_training(cuda_device, quad):
    W, H, P = 637, 351, 20_000
    raw = scenes.scene_plain_small(P)
    rng = np.random.default_rng(1)
    means = raw.means.astype(np.float32).copy()
    means[:, 2] = rng.permutation(np.linspace(-4.0, 4.0, P)).astype(np.float32)  # depths 4 to 12, 3 ulp apart at least
    args = [torch.from_numpy(np.ascontiguousarray(a, np.float32)).to(cuda_device)
            for a in (means, raw.log_scales, raw.quats, raw.opacity_logits, raw.shs.reshape(P, 48))]
    cam = Camera.from_spec(scenes.camera_front(W, H, 400.0))
    assert np.unique((means[:, 2] - cam.position[2].item()).astype(np.float32)).size == P
    line = _line(cuda_device)
    views = line // _tiles(W, H) + 1
    assert _tiles(W, H) <= line < views * _tiles(W, H)
    with torch.no_grad():
        one = render(*args, cam, (0.1, 0.2, 0.3))
        many = render_views(*args, [cam] * views, (0.1, 0.2, 0.3), stacked=True, quad_keys=quad)
    assert one.std() > 0.01
    for v in range(views):
        assert torch.equal(one, many[v])
