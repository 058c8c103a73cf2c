"""The emission's dispatch thresholds decide which scheme tests a rectangle's
tiles, never which keys come out: one tile per thread, the warp's pool, the
warp's and the CTA's large-rectangle sweeps.  Key counts of a batch are equal
for every threshold, down to everything queued (2 tiles) and up to nothing
queued (a threshold above every area), on a clustered and on a needle scene
(conics of every kind), at ragged image sizes, for both key layouts, and equal
the sum of the single views' counts for per-tile keys."""
import pytest
import torch

from polysplat_gb300 import Camera, Rasterizer, Scene, scenes
from polysplat_gb300 import _lib as R
from polysplat_gb300.batch import Batcher, View

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("quad", [0, R.QUAD_KEYS])
@pytest.mark.parametrize("raw", [scenes.subsample(scenes.scene_clustered(600_000, seed=1), 60_000, seed=2),
                                 scenes.scene_needles(20_000)], ids=["clustered", "needles"])
def test_thresholds_do_not_change_the_keys(cuda_device, raw, quad):
    scene = Scene.from_raw(raw, cuda_device)
    cams = [Camera.from_spec(scenes.orbit_camera(8.0, 0.4 + k, 0.1, w, h, scenes.focal_for(w)))
            for k, (w, h) in enumerate([(1271, 717), (333, 250), (2560, 1440)])]
    b = Batcher(3, 1 << 24, 3 * scene.num_vertex, 1 << 16, cuda_device)
    stream = torch.cuda.Stream(cuda_device)
    counts = []
    for massive, huge in [(32, 2048), (2, 2), (2, 1 << 30), (64, 64), (127, 200), (129, 1 << 30), (1 << 30, 1 << 30)]:
        b.set_thresholds(massive, huge)
        views = [View(0, c) for c in cams]
        b.render([scene], views, variant=R.RENDER_PERSISTENT_FUSED | quad, stream=stream)
        counts.append(b.finish(stream))
    assert len(set(counts)) == 1, counts
    if not quad:
        total = 0
        for c in cams:
            r = Rasterizer(scene, 1 << 23, 1 << 15)
            total += r.forward(scene, c, torch.zeros(3), render_variant="preranges_smem_persistent_lite_e2e",
                               return_stats=True)[1]["num_rendered"]
        assert counts[0] == total
