"""The preprocess without the large-Gaussian queue (no workspace, and the ES
operators): large rectangles are swept by the Gaussian's own warp.  Same keys
and same feature rows as with the queue, rows of Gaussians whose large
rectangle hits no tile among them; the ES pass counts the same tiles per
Gaussian.  Needles (conics of every kind) and clustered Gaussians, ragged image
sizes, rectangles from one tile to the whole frame."""
import ctypes

import numpy as np
import pytest
import torch

from polysplat_gb300 import Camera, Scene, ops, scenes
from polysplat_gb300._lib import lib

pytestmark = pytest.mark.gpu


def _preprocess(scene, cam, half, queue):
    dev, P, cap = scene.position.device, scene.num_vertex, 1 << 23
    feats = [torch.full((P, k), -7.0, device=dev) for k in (2, 4, 4)]
    keys, vals = torch.zeros(cap, dtype=torch.int64, device=dev), torch.zeros(cap, dtype=torch.int32, device=dev)
    off = torch.zeros(1, dtype=torch.int32, device=dev)
    ws = torch.zeros(int(lib().gsr_render_workspace_size()), dtype=torch.uint8, device=dev)
    p = lambda t: t.data_ptr()  # noqa: E731
    pos, rot = (ctypes.c_float * 3)(*cam.position.tolist()), (ctypes.c_float * 9)(*cam.rotation.reshape(-1).tolist())
    st = lib().gsr_preprocess(P, p(scene.position), p(scene.shs_half if half else scene.shs), int(half),
                              p(scene.opacity), p(scene.cov3d), cam.width, cam.height, 16, 16, pos, rot, cam.focal_x,
                              cam.focal_y, cam.zFar, cam.zNear, *[p(t) for t in feats], p(keys), p(vals), cap, p(off),
                              p(ws) if queue else None, ws.numel() if queue else 0,
                              torch.cuda.current_stream(dev).cuda_stream)
    assert st == 0
    n = int(off.item())
    assert n <= cap
    k, v = keys[:n].cpu().numpy(), vals[:n].cpu().numpy()
    order = np.lexsort((v, k))
    return k[order], v[order], [t.cpu().numpy() for t in feats]


@pytest.mark.parametrize("half", [False, True], ids=["fp32", "fp16"])
@pytest.mark.parametrize("size", [(1271, 717), (333, 250)])
@pytest.mark.parametrize("name", ["clustered", "needles"])
def test_same_keys_and_features_without_the_queue(cuda_device, name, size, half):
    raw = scenes.scene_needles(20_000) if name == "needles" else scenes.subsample(
        scenes.scene_clustered(600_000, seed=1), 60_000, seed=2)
    scene = Scene.from_raw(raw, cuda_device)
    cam = Camera.from_spec(scenes.orbit_camera(8.0, 0.4, 0.1, *size, scenes.focal_for(size[0])))
    k0, v0, f0 = _preprocess(scene, cam, half, True)
    k1, v1, f1 = _preprocess(scene, cam, half, False)
    assert np.array_equal(k0, k1) and np.array_equal(v0, v1)
    for a, b in zip(f0, f1):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    written = (f0[2] != -7.0).any(1)
    counts = np.bincount(v0, minlength=scene.num_vertex)
    assert written[counts > 0].all()
    if name == "needles":
        assert (written & (counts == 0)).any(), "large rectangles without a hit"

    P, dev = scene.num_vertex, cuda_device
    tiles, rect = (torch.zeros((P, k), dtype=torch.int32, device=dev) for k in (1, 2))
    raw_con, depth = torch.zeros((P, 4), device=dev), torch.zeros(P, device=dev)
    feats = [torch.zeros((P, k), device=dev) for k in (2, 4, 4)]
    es = ops.preprocess_es_pass_a_half_sh if half else ops.preprocess_es_pass_a
    es(scene.position, scene.shs_half if half else scene.shs, scene.opacity, scene.cov3d, cam.width, cam.height, 16,
       16, cam.position, cam.rotation, cam.focal_x, cam.focal_y, cam.zFar, cam.zNear, *feats, tiles.view(-1), raw_con,
       depth, rect)
    assert np.array_equal(tiles.view(-1).cpu().numpy(), counts)
    r = rect.cpu().numpy().astype(np.int64)
    area = ((r[:, 1] & 0xFFFF) - (r[:, 0] & 0xFFFF)) * ((r[:, 1] >> 16) - (r[:, 0] >> 16))
    assert (area[counts > 0] >= 128).sum() > 10 and (area[counts > 0] == 1).sum() > 10
