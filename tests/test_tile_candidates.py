"""The candidate tiles of the large-Gaussian sweep (csrc/tile_test.h) hold
every tile that passes the exact test, over all tiles of a grid: conics
inverted in FP32 from random 2D covariances with axis ratios up to 10^7 (so
that the determinant cancels, vanishes or turns negative), in every
orientation and next to the axes, centres on the screen, near it and far off;
conics with NaN, infinities and zeros; powers from negative to 6.  Exact: no
tile may be lost."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no host C++ compiler")
    out = str(tmp_path_factory.mktemp("tile") / "libtile.so")
    subprocess.check_call([gxx, "-O2", "-ffp-contract=off", "-std=c++17", "-shared", "-fPIC",
                           os.path.join(HERE, "tile_shim.cpp"), "-o", out])
    return ctypes.CDLL(out)


def _conics(rng, n):
    f4 = np.float32
    ang = rng.uniform(0, np.pi, n)
    ang[: n // 8] = rng.choice([0.0, np.pi / 2, np.pi / 4], n // 8) + rng.normal(0, 1e-4, n // 8)
    minor = 10.0 ** rng.uniform(-0.5, 2.0, n)
    major = minor * 10.0 ** rng.uniform(0.0, 3.5, n)
    ca, sa = np.cos(ang), np.sin(ang)
    with np.errstate(all="ignore"):
        a = (ca * ca * major ** 2 + sa * sa * minor ** 2 + 0.3).astype(f4)
        b = (ca * sa * (major ** 2 - minor ** 2)).astype(f4)
        c = (sa * sa * major ** 2 + ca * ca * minor ** 2 + 0.3).astype(f4)
        det = (a * c - b * b).astype(f4)
        con = np.stack([c / det, -b / det, a / det], 1).astype(f4)
    power = rng.uniform(0.05, 6.0, n).astype(f4)
    k = n // 50  # special values
    con[:k, rng.integers(0, 3)] = np.nan
    con[k:2 * k, 0] = np.inf
    con[2 * k:3 * k, 1] = 0.0
    con[3 * k:4 * k] = 0.0
    con[5 * k:6 * k] *= np.float32(-1.0)  # both diagonal entries negative
    con[6 * k:7 * k, 0] *= np.float32(-1.0)  # of different signs
    con[7 * k:8 * k] = rng.choice([np.inf, -np.inf], (k, 3))
    power[4 * k:5 * k] = rng.choice([0.0, -1.0, np.nan], k)
    return con, power


@pytest.mark.parametrize("bx,by", [(16, 16), (32, 16), (32, 32)])
@pytest.mark.parametrize("spread", [400.0, 3000.0, 2e5])
def test_no_hit_tile_is_lost(shim, spread, bx, by):
    rng = np.random.default_rng(int(spread) + bx + by)
    n, W, H = 4000, 1280, 720
    con, power = _conics(rng, n)
    ctr = np.stack([W / 2 + rng.normal(0, spread, n), H / 2 + rng.normal(0, spread, n)], 1).astype(np.float32)
    ctr[::3] = np.round(ctr[::3])  # on pixel and tile edges
    kind = np.empty(n, np.int32)
    hits, lost, cand = (np.empty(n, np.int64) for _ in range(3))
    p = lambda x: x.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    shim.tile_candidates(n, p(ctr), p(con), p(power), bx, by, 0, (W + bx - 1) // bx, 0, (H + by - 1) // by, p(kind),
                         p(hits), p(lost), p(cand))
    assert lost.sum() == 0, (np.flatnonzero(lost)[:5], kind[lost > 0][:5])
    assert set(kind) == {0, 1, 2, 3}
    # the needles' bands are worth having: a small part of the grid
    tiles = ((W + bx - 1) // bx) * ((H + by - 1) // by)
    needles = kind == 2
    assert cand[needles].mean() < 0.35 * tiles
