"""The preprocess's float form of the pixel coordinate (csrc/ndc.h) against
its double form, bit for bit: random values, values whose exact result lies
at the midpoint of two floats and their neighbours, the edges of the float
form's range, and infinities and NaN."""
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
    out = str(tmp_path_factory.mktemp("ndc") / "libndc.so")
    subprocess.check_call([gxx, "-O2", "-ffp-contract=off", "-std=c++17", "-shared", "-fPIC",
                           os.path.join(HERE, "ndc_shim.cpp"), "-o", out])
    return ctypes.CDLL(out)


@pytest.mark.parametrize("S", [1, 2, 3, 16, 717, 1080, 1237, 4320, 7680, 16383, 16384, 16385, 65535])
def test_pixel_coordinate_is_the_double_forms(shim, S):
    rng = np.random.default_rng(S)
    mid = (rng.integers(0, 2 ** 24, 200_000) + 0.5) * 2.0 ** rng.integers(-30, -8, 200_000)
    at_mid = ((2 * mid + 1) / S - 1).astype(np.float32)
    with np.errstate(over="ignore"):
        v = np.concatenate([
            rng.uniform(-2, 2, 400_000), rng.choice([-1.0, 1.0], 400_000) * 2.0 ** rng.uniform(-40, 100, 400_000),
            at_mid, -at_mid, np.nextafter(at_mid, np.float32(np.inf)), np.nextafter(at_mid, np.float32(-np.inf)),
            [0.0, -0.0, 1.0, -1.0, 2.0 ** -10, -2.0 ** -10, 2.0 ** 20, np.nextafter(np.float32(2.0 ** -10), np.float32(0)),
             np.inf, -np.inf, np.nan, 1e-45, 3e38]]).astype(np.float32)
    fast, ref = np.empty_like(v), np.empty_like(v)
    shim.ndc_both(v.size, v.ctypes.data_as(ctypes.c_void_p), S, fast.ctypes.data_as(ctypes.c_void_p),
                  ref.ctypes.data_as(ctypes.c_void_p))
    np.testing.assert_array_equal(fast.view(np.uint32), ref.view(np.uint32))
