"""A scene without Gaussians is refused by the training renders: the parts of
their one allocation have no address where they are empty."""
import pytest
import torch

from polysplat_gb300 import diff


def test_an_empty_part_has_no_address():
    sizes = (0, 4, 300, 0, 8)
    parts = diff._parts(diff._slab("cpu", sizes), sizes)
    assert [p.value is None for p in parts] == [True, False, False, True, False]
    at = [p.value for p in parts if p.value]
    assert at[1] - at[0] == 256 and at[2] - at[1] == 512


@pytest.mark.gpu
@pytest.mark.parametrize("views", [1, 2])
def test_a_scene_without_gaussians_is_refused(cuda_device, views):
    from polysplat_gb300 import Camera, scenes
    from polysplat_gb300._lib import GsrError

    z = lambda *s: torch.zeros(*s, device=cuda_device)  # noqa: E731
    args = (z(0, 3), z(0, 3), z(0, 4), z(0), z(0, 48))
    cam = Camera.from_spec(scenes.camera_front(64, 48, 48.0))
    with pytest.raises(GsrError):
        if views == 1:
            diff.render(*args, cam)
        else:
            diff.render_views(*args, [cam] * views)
