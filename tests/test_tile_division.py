"""The candidate tiles hold every tile that passes the exact test when the
divisions behind them are off by the 2 ulp that the device's fast-math division
may be off, in either direction, for every tile width the preprocess takes.  A
width of 24 is no power of two, so a centre on a multiple of it may get a
quotient below the whole number: conics without a hit but the centre's tile
(NaN, infinite) have that one tile to lose."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from test_tile_candidates import _conics

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module", params=[-2, 0, 2])
def shim(request, tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no host C++ compiler")
    out = str(tmp_path_factory.mktemp("tile") / "libtile.so")
    subprocess.check_call([gxx, "-O2", "-ffp-contract=off", "-std=c++17", "-shared", "-fPIC",
                           "-DGSR_TT_ULPS=%d" % request.param, os.path.join(HERE, "tile_div_shim.cpp"), "-o", out])
    return ctypes.CDLL(out)


@pytest.mark.parametrize("bx,by", [(16, 16), (24, 16), (32, 32)])
@pytest.mark.parametrize("spread", [400.0, 3000.0])
def test_no_hit_tile_is_lost_to_a_quotient(shim, spread, bx, by):
    rng = np.random.default_rng(int(spread) + bx + by)
    n, W, H = 3000, 1296, 720
    con, power = _conics(rng, n)
    con[1::7] = np.nan
    ctr = np.stack([W / 2 + rng.normal(0, spread, n), H / 2 + rng.normal(0, spread, n)], 1).astype(np.float32)
    ctr[::2, 0] = bx * rng.integers(0, W // bx, n // 2)  # first and last pixels of a tile
    ctr[::4, 0] += bx - 1
    ctr[::3, 1] = by * rng.integers(0, H // by, n // 3)
    kind = np.empty(n, np.int32)
    hits, lost, cand = (np.empty(n, np.int64) for _ in range(3))
    p = lambda x: x.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    shim.tile_candidates(n, p(ctr), p(con), p(power), bx, by, 0, (W + bx - 1) // bx, 0, (H + by - 1) // by, p(kind),
                         p(hits), p(lost), p(cand))
    centre = kind == 3
    assert (hits[centre] > 0).sum() > 100
    assert lost.sum() == 0, "%d tiles of %d Gaussians, kinds %s" % (lost.sum(), (lost > 0).sum(),
                                                                  np.unique(kind[lost > 0]))
