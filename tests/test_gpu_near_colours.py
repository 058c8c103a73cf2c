"""The render backward against 64 bits where the Gaussians along a ray have
nearly one colour, as in a converged scene: the gradient of a Gaussian's opacity
is a product with (c - R), its colour less the colour behind it, and must keep
the accuracy it has where colours differ.

Lists of 100 Gaussians over four tiles, every one of them in every list, no
early exit; the reference takes the forward's own features, so that what is
measured is the walk: alpha's ex2 and the restored transmittance (about 1e-6
over such lists) and the rounding of (c - R) . G.  A difference of products that
are as large as the colours would be off by 2^-24 / spread, 2e-5 and 2e-4 here."""
import ctypes

import numpy as np
import pytest
import torch

from polysplat_gb300 import Camera, scenes
from polysplat_gb300._lib import lib
from polysplat_gb300.ops import get_sort_buffer_size

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spread", [0.3, 3e-3, 3e-4])
@pytest.mark.parametrize("bg", [(0.0, 0.0, 0.0), (0.6, 0.5, 0.4)])
def test_opacity_gradients(cuda_device, spread, bg):
    dev, P, W, H = cuda_device, 100, 32, 32
    rng = np.random.default_rng(11)
    cam = Camera.from_spec(scenes.camera_front(W, H, 32.0))
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float32)).to(dev)  # noqa: E731
    means = np.stack([rng.normal(0, 0.8, P), rng.normal(0, 0.8, P), rng.permutation(np.linspace(-1, 1, P))], 1)
    shs = np.zeros((P, 16, 3))
    shs[:, 0] = (np.array([0.6, 0.5, 0.4]) + spread * rng.uniform(-1, 1, (P, 3)) - 0.5) / 0.28209479177387814
    opacity = rng.uniform(0.02, 0.08, P)
    params = [t(means), t(np.log(rng.uniform(4.0, 6.0, (P, 3)))), t(rng.normal(size=(P, 4))),
              t(np.log(opacity / (1 - opacity))), t(shs.reshape(P, 48))]
    grad = t(rng.normal(size=(H, W, 3)))
    cap, f32, i32 = 4096, torch.float32, torch.int32
    z = lambda n, dt=f32: torch.zeros(n, dtype=dt, device=dev)  # noqa: E731
    p = lambda x: ctypes.c_void_p(x.data_ptr())  # noqa: E731
    op, cov, cnt, ws = z(P), z(6 * P), z(1, i32), z(get_sort_buffer_size(cap), torch.uint8)
    ku, vu, ks, vs = z(cap, torch.int64), z(cap, i32), z(cap, torch.int64), z(cap, i32)
    xy, rgbd, con, ranges, n_tile = z(2 * P), z(4 * P), z(4 * P), z(8, i32), z(4, i32)
    T, img, gxy, gcon, grgb = z(H * W), z(H * W * 3), z(2 * P), z(4 * P), z(3 * P)
    outs = [torch.zeros_like(x) for x in params]
    pos, rot = (ctypes.c_float * 3)(*cam.position.tolist()), (ctypes.c_float * 9)(*cam.rotation.reshape(-1).tolist())
    view = (W, H, pos, rot, cam.focal_x, cam.focal_y, cam.zFar, cam.zNear, (ctypes.c_float * 3)(*bg))
    s = ctypes.c_void_p(torch.cuda.current_stream(dev).cuda_stream)
    assert lib().gsr_train_forward(P, *[p(x) for x in params], *view, p(op), p(cov), p(cnt), p(ws), ws.numel(), p(ku),
                                   p(vu), p(ks), p(vs), cap, p(xy), p(rgbd), p(con), p(ranges), p(n_tile), p(T),
                                   p(img), s) == 0
    assert lib().gsr_train_backward(P, *[p(x) for x in params], *view, p(cnt), cap, p(vs), p(ranges), p(n_tile), p(T),
                                    p(xy), p(rgbd), p(con), p(grad), p(gxy), p(gcon), p(grgb),
                                    *[p(x) for x in outs], 0, s) == 0
    assert n_tile.tolist() == [P] * 4, "every Gaussian in every list, none left out"
    xy, con, rgbd = (x.cpu().double().reshape(P, -1) for x in (xy, con, rgbd))
    order = torch.argsort(rgbd[:, 3])
    xy, con, col = xy[order], con[order], rgbd[order, :3]
    py, px = torch.meshgrid(torch.arange(H).double(), torch.arange(W).double(), indexing="ij")
    dx, dy = xy[:, 0, None] - px.reshape(-1), xy[:, 1, None] - py.reshape(-1)
    alpha = torch.exp2(con[:, 3, None] + con[:, 0, None] * dx * dx + con[:, 2, None] * dy * dy + con[:, 1, None] * dx * dy)
    before = torch.cat([torch.ones(1, H * W).double(), torch.cumprod(1 - alpha, 0)[:-1]])
    assert (before[-1].min() > 1e-3), "no pixel saturates"
    G = grad.cpu().double().reshape(-1, 3)
    R, want = torch.tensor(bg).double().expand(H * W, 3).float().double().clone(), torch.zeros(P).double()
    for k in range(P - 1, -1, -1):
        d = ((col[k] - R) * G).sum(1)
        want[k] = (d * alpha[k] * before[k]).sum() * np.log(2.0)
        R = R + alpha[k][:, None] * (col[k] - R)
    got = gcon.cpu().double().reshape(P, 4)[order, 3]
    off = ((got - want).norm() / want.norm()).item()
    assert off < 5e-6, off
