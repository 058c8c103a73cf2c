"""GSR_EXPAND_QUADS: the fused 16x16 forward sorts quad keys and expands them to
per-tile lists; its sorted arrays, ranges, key count and image against the
per-stage calls, which sort per-tile keys.

Keys and ranges are integers and must be equal; pairs of equal key may come in
any order, so values are compared as sets per key, and images within 2/255 (the
blend order of equal keys).  Frames whose sides leave partial tiles and partial
quads, a single tile, an empty view, and key buffers that are too small.
"""
import numpy as np
import pytest
import torch

from polysplat_gb300 import Camera, Rasterizer, Scene, ops, scenes
from polysplat_gb300 import _lib as R
from polysplat_gb300._lib import GsrError

pytestmark = pytest.mark.gpu

BG = torch.tensor([0.1, 0.2, 0.3])


@pytest.fixture(scope="module")
def scene(cuda_device):
    return Scene.from_raw(scenes.scene_clustered(60_000, seed=5), cuda_device)


def _camera(w, h, az=0.7):
    return Camera.from_spec(scenes.orbit_camera(8.0, az, 0.3, w, h, scenes.focal_for(w)))


def _fused(scene, r, cam, variant, ranges, flag=R.EXPAND_QUADS):
    out = torch.zeros((cam.height, cam.width, 3), dtype=torch.uint8, device=r.device)
    n = ops._forward(variant | flag, True, scene.position, scene.shs_half, scene.opacity, scene.cov3d, cam.width,
                     cam.height, 16, 16, cam.position, cam.rotation, cam.focal_x, cam.focal_y, cam.zFar, cam.zNear,
                     r.curr_offset, r.list_sorting_space, r.gaussian_keys_unsorted, r.gaussian_values_unsorted,
                     r.gaussian_keys_sorted, r.gaussian_values_sorted, r.points_xy, r.rgb_depth, r.conic_opacity,
                     ranges, BG, out)
    return out, n


@pytest.mark.parametrize("w,h", [(16, 16), (1, 1), (33, 17), (48, 80), (250, 131), (641, 359), (1920, 1080),
                                 (3839, 2161)])
def test_expanded_lists_match_the_per_tile_sort(scene, w, h):
    cam = _camera(w, h)
    cap, tiles = 6_000_000, -(-w // 16) * -(-h // 16)
    a, b = Rasterizer(scene, cap, 1 << 16), Rasterizer(scene, cap, 1 << 16)
    img, m = _fused(scene, a, cam, R.RENDER_PERSISTENT_RANGES, a.tile_ranges_buf)
    ref, sr = b.forward(scene, cam, BG, render_variant="preranges_smem", return_stats=True, use_es=False)
    n = sr["num_rendered"]
    assert m == n
    ka, kb = a.gaussian_keys_sorted[:n], b.gaussian_keys_sorted[:n]
    assert torch.equal(ka, kb)
    va, vb = (r.gaussian_values_sorted[:n] for r in (a, b))
    k, na, nb = (t.cpu().numpy() for t in (ka, va, vb))
    assert np.array_equal(na[np.lexsort((na, k))], nb[np.lexsort((nb, k))])
    assert torch.equal(a.tile_ranges_buf[:tiles], b.tile_ranges_buf[:tiles])
    assert int((img.int() - ref.int()).abs().max()) <= 2
    # without the caller's ranges; the fused variant's exit test on the per-tile lists
    ops._render(R.RENDER_PERSISTENT_FUSED, n, w, h, b.points_xy, b.rgb_depth, b.conic_opacity, kb, vb, None, BG, ref,
                16, 16)
    img2, m2 = _fused(scene, a, cam, R.RENDER_PERSISTENT_FUSED, None)
    assert m2 == n and int((img2.int() - ref.int()).abs().max()) <= 2


def test_empty_view_and_small_buffers(scene):
    away = _camera(320, 200)
    away.position = away.position * -1000.0  # everything lies behind it
    r = Rasterizer(scene, 1_000_000, 1 << 16)
    img, m = _fused(scene, r, away, R.RENDER_PERSISTENT_FUSED, None)
    ref, m0 = _fused(scene, r, away, R.RENDER_PERSISTENT_FUSED, None, flag=0)
    assert m == m0 == 0 and torch.equal(img, ref)
    cam = _camera(1920, 1080)
    n = _fused(scene, Rasterizer(scene, 6_000_000, 1 << 16), cam, R.RENDER_PERSISTENT_FUSED, None, flag=0)[1]
    # the count is the per-tile one, whether or not the quad keys fit too, and
    # where the buffer does not even hold the expansion's own words
    for cap in (n - 1, n // 2, n // 8, 1000):
        with pytest.raises(GsrError) as ei:
            _fused(scene, Rasterizer(scene, cap, 1 << 16), cam, R.RENDER_PERSISTENT_FUSED, None)
        assert ei.value.status == R.GSR_OVERFLOW and ei.value.num == n
    assert _fused(scene, Rasterizer(scene, n, 1 << 16), cam, R.RENDER_PERSISTENT_FUSED, None)[1] == n


def _depth_first(scene, cam, cap, dev, flag):
    r = Rasterizer(scene, cap, 1 << 16)
    r._expand_quads = lambda _: bool(flag)
    img, st = r.forward(scene, cam, BG, render_variant="preranges_smem_persistent_lite", use_es=True,
                        return_stats=True)
    assert st["used_es"]
    return r, img, st["num_rendered"]


@pytest.mark.parametrize("w,h", [(16, 16), (33, 17), (250, 131), (641, 359), (1920, 1080), (3839, 2161)])
def test_depth_first_expanded_lists_are_the_same(cuda_device, scene, w, h):
    """The depth-first order of equal keys is the Gaussians' index order, so the
    arrays and the image are equal, not only alike."""
    cam, cap, tiles = _camera(w, h), 6_000_000, -(-w // 16) * -(-h // 16)
    a, ia, na = _depth_first(scene, cam, cap, cuda_device, True)
    b, ib, nb = _depth_first(scene, cam, cap, cuda_device, False)
    assert na == nb and torch.equal(ia, ib)
    for x, y in ((a.gaussian_keys_sorted.view(torch.int32)[:na], b.gaussian_keys_sorted.view(torch.int32)[:na]),
                 (a.gaussian_values_sorted[:na], b.gaussian_values_sorted[:na]),
                 (a.tile_ranges_buf[:tiles], b.tile_ranges_buf[:tiles])):
        assert torch.equal(x, y)


def test_depth_first_expansion_reports_the_per_tile_count(cuda_device, scene):
    cam = _camera(1920, 1080)
    n = _depth_first(scene, cam, 6_000_000, cuda_device, False)[2]
    for cap in (n - 1, n // 2, n // 8):
        with pytest.raises(GsrError) as ei:
            _depth_first(scene, cam, cap, cuda_device, True)
        assert ei.value.status == R.GSR_OVERFLOW and ei.value.num == n
    assert _depth_first(scene, cam, n, cuda_device, True)[2] == n
