"""The digit passes at the edges of their 3584-key tiles: counts one below, at
and above a tile, a single key, more tiles than one look-back window, with
keys spread over all digits, all equal, and in runs; bit widths that end
inside, at and across the depth word.  Exact against numpy's stable sort."""
import numpy as np
import pytest
import torch

from polysplat_gb300 import ops

pytestmark = pytest.mark.gpu
TILE = 3584


@pytest.mark.parametrize("end_bit", [5, 32, 37, 45, 64])
@pytest.mark.parametrize("n", [1, 31, 33, TILE - 1, TILE, TILE + 1, 2 * TILE, 11 * TILE + 5, 40 * TILE - 3])
def test_sort_at_tile_edges(cuda_device, n, end_bit):
    rng = np.random.default_rng(n + end_bit)
    spread = rng.integers(0, 1 << 63, n, dtype=np.uint64)
    runs = np.repeat(rng.integers(0, 1 << 63, n // 5 + 1, dtype=np.uint64), 5)[:n]
    for keys in (spread, runs, np.full(n, spread[0])):
        vals = rng.permutation(n).astype(np.uint32)
        ku = torch.from_numpy(keys.view(np.int64).copy()).to(cuda_device)
        vu = torch.from_numpy(vals.view(np.int32).copy()).to(cuda_device)
        ks, vs = torch.zeros_like(ku), torch.zeros_like(vu)
        ws = torch.zeros(ops.get_sort_buffer_size(n), dtype=torch.int8, device=cuda_device)
        ops.sort_pairs_bits(n, end_bit, ws, ku, vu, ks, vs)
        mask = np.uint64((1 << end_bit) - 1)
        order = np.argsort(keys & mask, kind="stable")
        np.testing.assert_array_equal(ks.cpu().numpy().view(np.uint64), keys[order])
        np.testing.assert_array_equal(vs.cpu().numpy().view(np.uint32), vals[order])
