"""The expansion on either side of the line where the CTAs of k_quad_tiles take
the totals of k_quad_sums instead of adding up all earlier lists (32768 tiles),
with CTAs that end inside a row of quads: the depth-first arrays and images of
expanded and of per-tile lists are equal, and the fused forward's keys, ranges
and count too."""
import pytest
import torch

from polysplat_gb300 import Rasterizer
from polysplat_gb300 import _lib as R

from test_gpu_quad_expand import BG, _camera, _depth_first, _fused, scene  # noqa: F401

pytestmark = pytest.mark.gpu

SIZES = [(4096, 2048), (4097, 2048), (4111, 2300), (129, 70_001), (9001, 1700)]


@pytest.mark.parametrize("w,h", SIZES)
def test_depth_first(cuda_device, scene, w, h):  # noqa: F811
    cam, cap, tiles = _camera(w, h), 1 << 24, -(-w // 16) * -(-h // 16)
    a, ia, na = _depth_first(scene, cam, cap, cuda_device, True)
    b, ib, nb = _depth_first(scene, cam, cap, cuda_device, False)
    assert 0 < na == nb and torch.equal(ia, ib)
    for x, y in ((a.gaussian_keys_sorted.view(torch.int32)[:na], b.gaussian_keys_sorted.view(torch.int32)[:na]),
                 (a.gaussian_values_sorted[:na], b.gaussian_values_sorted[:na]),
                 (a.tile_ranges_buf[:tiles], b.tile_ranges_buf[:tiles])):
        assert torch.equal(x, y)


@pytest.mark.parametrize("w,h", SIZES)
def test_fused(cuda_device, scene, w, h):  # noqa: F811
    cam, cap, tiles = _camera(w, h), 1 << 24, -(-w // 16) * -(-h // 16)
    a, b = Rasterizer(scene, cap, 1 << 16), Rasterizer(scene, cap, 1 << 16)
    ia, na = _fused(scene, a, cam, R.RENDER_PERSISTENT_RANGES, a.tile_ranges_buf)
    ib, nb = _fused(scene, b, cam, R.RENDER_PERSISTENT_RANGES, b.tile_ranges_buf, flag=0)
    assert na == nb and torch.equal(a.gaussian_keys_sorted[:na], b.gaussian_keys_sorted[:na])
    assert torch.equal(a.tile_ranges_buf[:tiles], b.tile_ranges_buf[:tiles])
    assert int((ia.int() - ib.int()).abs().max()) <= 2
