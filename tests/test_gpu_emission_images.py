"""Whichever scheme tests a rectangle's tiles (the dispatch thresholds of a
batch), the images are the same bytes: no scheme swaps one tile for another.
Clustered and needle Gaussians whose depths are all different, so that every
list has one order, at ragged image sizes and for both key layouts, against the
single views' depth-first renders.  Thresholds above 128 tiles act as 128: a
batch always has its queue, and test_gpu_no_queue.py covers the sweeps without
one."""
import numpy as np
import pytest
import torch

from polysplat_gb300 import Camera, Rasterizer, Scene, scenes
from polysplat_gb300 import _lib as R
from polysplat_gb300.batch import Batcher, View

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("quad", [0, R.QUAD_KEYS], ids=["tiles", "quads"])
@pytest.mark.parametrize("name", ["clustered", "needles"])
def test_thresholds_do_not_change_the_images(cuda_device, name, quad):
    raw = scenes.scene_needles(20_000) if name == "needles" else scenes.subsample(
        scenes.scene_clustered(600_000, seed=1), 60_000, seed=2)
    P = raw.num
    raw.means[:, 2] = np.random.default_rng(4).permutation(np.linspace(-6.0, 9.0, P)).astype(np.float32)
    scene = Scene.from_raw(raw, cuda_device)
    cams = [Camera.from_spec(scenes.camera_front(w, h, scenes.focal_for(w)))
            for w, h in [(1271, 717), (333, 250), (2560, 1440)]]
    assert np.unique((raw.means[:, 2] - cams[0].position[2].item()).astype(np.float32)).size == P
    b = Batcher(3, 1 << 24, 3 * P, 1 << 16, cuda_device)
    stream, first = torch.cuda.Stream(cuda_device), None
    for massive, huge in [(32, 2048), (2, 2), (2, 1 << 30), (64, 64), (127, 200), (1 << 30, 1 << 30)]:
        b.set_thresholds(massive, huge)
        views = [View(0, c) for c in cams]
        torch.cuda.synchronize()
        b.render([scene], views, variant=R.RENDER_PERSISTENT_RANGES | quad, stream=stream)
        b.finish(stream)
        images = [v.out.cpu() for v in views]
        first = first or images
        for x, y in zip(images, first):
            assert torch.equal(x, y), (massive, huge)
    for c, x in zip(cams, first):
        r = Rasterizer(scene, 1 << 24, 1 << 16)
        one = r.forward(scene, c, torch.zeros(3), render_variant="preranges_smem_persistent_lite", use_es=True)
        assert torch.equal(one.cpu(), x)
