"""Pairs of equal (tile, depth) keys are blended in the order in which the
preprocess's CTAs reserve their place in the key buffer, so that order decides
pixels.  A CTA reserves once its Gaussians' features are written.  Here every
other CTA tests two steps of tiles for two Gaussians and loads two colours; the
CTAs between them test one tile for each of 256 Gaussians and load 256 colours
from DRAM.  With the reservation behind the colours most of the former come
first, with the reservation in front of them most of the latter."""
import numpy as np
import pytest
import torch

from polysplat_gb300 import ops, scenes

pytestmark = pytest.mark.gpu

CTA = 256


def test_a_cta_reserves_after_its_features(cuda_device):
    dev, ctas = cuda_device, 300  # one wave: every CTA is resident from the start
    P = ctas * CTA
    W, H, f = 800, 592, 600.0
    cam = scenes.camera_front(W, H, f)
    rot = np.asarray(cam.rotation, np.float32).reshape(3, 3)
    at = np.asarray(cam.position, np.float32)
    rng = np.random.default_rng(3)
    cta, lane = np.arange(P) // CTA, np.arange(P) % CTA
    depth = 10.0
    # image position: the middle of a tile away from the border
    px = np.stack([16.0 * rng.integers(8, W // 16 - 8, P) + 8.0, 16.0 * rng.integers(8, H // 16 - 8, P) + 8.0], 1)
    view = np.concatenate([(px - [W / 2, H / 2]) / f * depth, np.full((P, 1), depth)], 1)
    large = (cta % 2 == 1) & (lane < 2)
    outside = (cta % 2 == 1) & (lane >= 2)
    view[outside, 0] += 100.0  # in front of the camera, projected, beside the image
    pos = torch.from_numpy((at + view @ rot.T).astype(np.float32)).to(dev)
    # 34 and 2 pixels of reach at an opacity of 0.9
    var = np.where(large, 106.0, 0.05) * (depth / f) ** 2
    cov = np.zeros((P, 6), np.float32)
    cov[:, 0] = cov[:, 3] = cov[:, 5] = var
    cov = torch.from_numpy(cov).to(dev)
    op = torch.full((P,), 0.9, device=dev)
    sh = torch.zeros((P, 48), device=dev)
    feats = (torch.zeros((P, 2), device=dev), torch.zeros((P, 4), device=dev), torch.zeros((P, 4), device=dev))
    cap = 8 * P
    ku, vu = torch.zeros(cap, dtype=torch.int64, device=dev), torch.zeros(cap, dtype=torch.int32, device=dev)
    off = torch.zeros(1, dtype=torch.int32, device=dev)
    flush = torch.empty(1 << 28, dtype=torch.uint8, device=dev)
    first = total = 0
    for k in range(12):
        off.zero_()
        flush.fill_(1)  # the colours come from DRAM
        ops.preprocess(pos, sh, op, cov, W, H, 16, 16, torch.from_numpy(at), torch.from_numpy(rot), f, f, 100.0, 0.01,
                       *feats, ku, vu, off)
        n = int(off.item())
        where = np.full(ctas, -1)
        np.maximum.at(where, vu[:n].cpu().numpy() // CTA, np.arange(n))
        assert (where >= 0).all(), "every CTA has keys"
        keys = np.bincount(vu[:n].cpu().numpy() // CTA, minlength=ctas)
        assert (keys[0::2] == CTA).all(), "one tile for each of a CTA's 256 Gaussians"
        assert (keys[1::2] > 32).all() and (keys[1::2] <= 64).all(), "two Gaussians of many tiles"
        if k >= 2:
            first += int((where[1::2] < where[0::2]).sum())
            total += ctas // 2
    assert first > total // 2, "%d of %d" % (first, total)
