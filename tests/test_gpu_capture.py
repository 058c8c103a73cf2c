"""The fused and the depth-first forward can be captured in a CUDA graph: a replay
gives the image, the key count and the sorted keys of the direct call, with
per-tile keys, quad keys and expanded quads, and after the scene was changed in
place between replays."""
import ctypes

import pytest
import torch

from polysplat_gb300 import Camera, Rasterizer, Scene, ops, scenes
from polysplat_gb300 import _lib as R
from polysplat_gb300._lib import lib

pytestmark = pytest.mark.gpu

CAP, TILES = 1 << 22, 1 << 13


def _floats(t):
    v = [float(x) for x in t.reshape(-1).tolist()]
    return (ctypes.c_float * len(v))(*v)


@pytest.mark.parametrize("flag", [0, R.QUAD_KEYS, R.EXPAND_QUADS], ids=["tiles", "quads", "expanded"])
@pytest.mark.parametrize("depth_first", [False, True], ids=["fused", "depth_first"])
def test_replay_gives_the_direct_call(cuda_device, depth_first, flag):
    dev = cuda_device
    scene = Scene.from_raw(scenes.subsample(scenes.scene_clustered(600_000, seed=1), 40_000, seed=2), dev)
    cam = Camera.from_spec(scenes.orbit_camera(8.0, 0.5, 0.1, 641, 359, scenes.focal_for(641)))
    r, P = Rasterizer(scene, CAP, TILES), scene.num_vertex
    scratch = torch.zeros(ops.depth_first_scratch_size(P), dtype=torch.int8, device=dev)
    out = torch.zeros((359, 641, 3), dtype=torch.uint8, device=dev)
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    pos, rot, bg = _floats(cam.position), _floats(cam.rotation), _floats(torch.tensor([0.1, 0.2, 0.3]))

    def call(stream):
        scene_args = (P, p(scene.position), p(scene.shs_half), 1, p(scene.opacity), p(scene.cov3d), 641, 359, 16, 16,
                      pos, rot, cam.focal_x, cam.focal_y, cam.zFar, cam.zNear, p(r.curr_offset),
                      p(r.list_sorting_space), r.list_sorting_space.numel())
        rest = (p(r.gaussian_keys_unsorted), p(r.gaussian_values_unsorted), p(r.gaussian_keys_sorted),
                p(r.gaussian_values_sorted), CAP, p(r.points_xy), p(r.rgb_depth), p(r.conic_opacity),
                p(r.tile_ranges_buf), bg, p(out), ctypes.c_void_p(stream))
        if depth_first:
            return lib().gsr_forward_depth_first(R.RENDER_PERSISTENT_FUSED | flag, *scene_args, p(scratch),
                                                 scratch.numel(), *rest)
        return lib().gsr_forward(R.RENDER_PERSISTENT_FUSED | flag, *scene_args, *rest)

    side = torch.cuda.Stream(dev)
    with torch.cuda.stream(side):
        assert call(side.cuda_stream) == 0
    side.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        assert call(torch.cuda.current_stream(dev).cuda_stream) == 0
    for k in range(3):
        scene.opacity.mul_(0.8)  # another frame each time
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            assert call(side.cuda_stream) == 0
        side.synchronize()
        n, image = int(r.curr_offset.item()), out.clone()
        keys = r.gaussian_keys_sorted.view(torch.int32)[:n] if depth_first else r.gaussian_keys_sorted[:n]
        keys = keys.clone()
        for _ in range(2):
            out.zero_()
            r.curr_offset.fill_(-1)
            r.gaussian_keys_sorted.zero_()
            torch.cuda.synchronize()
            graph.replay()
            torch.cuda.synchronize()
            assert int(r.curr_offset.item()) == n > 0
            again = r.gaussian_keys_sorted.view(torch.int32)[:n] if depth_first else r.gaussian_keys_sorted[:n]
            assert torch.equal(again, keys)
            far = (out.int() - image.int()).abs()
            assert far.max() == 0 if depth_first else far.max() <= 2
