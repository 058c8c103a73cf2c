"""When a frame sorts quad keys and expands them: the measured frames of
Rasterizer._expand_quads, by the last frame's key count, the Gaussians and the
tiles."""
import types

import pytest

from polysplat_gb300 import Rasterizer


@pytest.mark.parametrize("M,P,tiles,expand", [
    (None, 3_000_000, 8160, False),
    (9_500_000, 3_000_000, 8160, True),
    (5_200_000, 3_000_000, 8160, True),
    (2_000_000, 1_000_000, 4056, True),
    (1_500_000, 480_000, 4056, True),
    (1_400_000, 100_000, 4056, False),
    (26_117_280, 20_000_000, 129_600, False),
    (7_370_089, 100_000, 129_600, True),
    (7_605_908, 5_000_000, 291_600, False),
    (8_853_910, 5_000_000, 518_400, False),
    (35_387_098, 20_000_000, 518_400, True),
    (26_251_503, 100_000, 518_400, True),
])
def test_expand_rule(M, P, tiles, expand):
    r = object.__new__(Rasterizer)
    r._es_last_M, r._frame_tiles = M, tiles
    assert r._expand_quads(types.SimpleNamespace(num_vertex=P)) is expand
