"""Renders of few tiles share a tile between the warps of a CTA; others take a
tile per warp.  Both give the same bytes on the same sorted lists: a small
image against the top rows of a taller one whose further tiles are empty (its
tile ids and lists are the small image's), for every exit cadence, at ragged
sizes, and with tiles that saturate, end inside a batch and have no Gaussian.
Quad keys: the depth-first forward, whose lists have a fixed order, gives the
same bytes with quad and per-tile keys on both sides of the line.  (Two
single-pass sorts may order equal keys differently, so their images are not
compared here.)"""
import pytest
import torch

from polysplat_gb300 import Camera, Rasterizer, Scene, ops, scenes
from polysplat_gb300 import _lib as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cadence", [2, 8, 16])
@pytest.mark.parametrize("W,H", [(640, 360), (637, 351), (17, 250), (800, 481)])
def test_few_tiles_render_as_many(cuda_device, W, H, cadence):
    raw = scenes.subsample(scenes.scene_clustered(600_000, seed=1), 40_000, seed=2)
    scene = Scene.from_raw(raw, cuda_device)
    cam = Camera.from_spec(scenes.orbit_camera(8.0, 0.5, 0.1, W, H, scenes.focal_for(W)))
    rast = Rasterizer(scene, 1 << 22, 1 << 13)
    bg = torch.tensor([0.2, 0.1, 0.4])
    _, st = rast.forward(scene, cam, bg, render_variant="preranges_smem_persistent_lite", return_stats=True)
    n, gx = st["num_rendered"], (W + 15) // 16
    tall = ((2433 + gx) // gx + 1) * 16  # more than 16 tiles per SM
    feats = (rast.points_xy, rast.rgb_depth, rast.conic_opacity)
    images = []
    for h in (H, tall):
        ranges = torch.full((gx * ((h + 15) // 16), 2), n, dtype=torch.int32, device=cuda_device)
        tiles = gx * ((H + 15) // 16)
        ranges[:tiles] = rast.tile_ranges_buf[:tiles]
        out = torch.zeros((h, W, 3), dtype=torch.uint8, device=cuda_device)
        if cadence == 16:
            ops.render_16x16_preranges_smem_persistent_lite_fused(n, W, h, *feats, rast.gaussian_keys_sorted[:n],
                                                                  rast.gaussian_values_sorted, bg, out)
        else:
            op = ops.render_16x16_preranges if cadence == 2 else ops.render_16x16_preranges_smem_persistent_lite
            op(n, W, h, *feats, rast.gaussian_values_sorted, ranges, bg, out)
        images.append(out)
    # rows past the small image's last tile row hold the background; a ragged
    # last tile has pixels below H in the tall image only
    assert torch.equal(images[0], images[1][:H])


@pytest.mark.parametrize("W,H", [(640, 360), (637, 351), (1600, 1000)])
def test_quad_lists_render_as_tile_lists(cuda_device, W, H):
    raw = scenes.subsample(scenes.scene_clustered(600_000, seed=1), 40_000, seed=2)
    scene = Scene.from_raw(raw, cuda_device)
    cam = Camera.from_spec(scenes.orbit_camera(8.0, 0.5, 0.1, W, H, scenes.focal_for(W)))
    cap = 1 << 22
    i32 = lambda k: torch.zeros(k, dtype=torch.int32, device=cuda_device)  # noqa: E731
    f32 = lambda k: torch.zeros((scene.num_vertex, k), device=cuda_device)  # noqa: E731
    images = []
    for flag in (0, R.QUAD_KEYS):
        out = torch.zeros((H, W, 3), dtype=torch.uint8, device=cuda_device)
        ops.forward_depth_first(R.RENDER_PERSISTENT_FUSED | flag, True, scene.position, scene.shs_half, scene.opacity,
                                scene.cov3d, W, H, 16, 16, cam.position, cam.rotation, cam.focal_x, cam.focal_y,
                                cam.zFar, cam.zNear, i32(1),
                                torch.zeros(ops.get_sort_buffer_size(cap), dtype=torch.int8, device=cuda_device),
                                torch.zeros(ops.depth_first_scratch_size(scene.num_vertex), dtype=torch.int8,
                                            device=cuda_device),
                                i32(cap), i32(cap), i32(cap), i32(cap), f32(2), f32(4), f32(4),
                                i32(2 << 13).view(-1, 2), torch.tensor([0.2, 0.1, 0.4]), out)
        images.append(out)
    assert torch.equal(images[0], images[1])
