"""gsr_read_status takes its host words from one block of the process: more
threads at once than the block has places, threads that live for one call, and
calls after a device reset all read their own words."""
import ctypes
import subprocess
import sys
import threading

import pytest
import torch

from polysplat_gb300 import _lib as R
from polysplat_gb300._lib import lib

pytestmark = pytest.mark.gpu


def _read(ws, num, cap, stream):
    n = ctypes.c_int32(-1)
    st = lib().gsr_read_status(ws, num, cap, ctypes.byref(n), ctypes.c_void_p(stream))
    return st, n.value


@pytest.mark.parametrize("threads,calls", [(100, 40), (200, 1)])
def test_threads_read_their_own_words(cuda_device, threads, calls):
    ws = torch.zeros(threads, dtype=torch.int32, device=cuda_device)
    num = torch.arange(threads, dtype=torch.int32, device=cuda_device) * 3
    streams = [torch.cuda.Stream(cuda_device).cuda_stream for _ in range(threads)]
    torch.cuda.synchronize()
    go, bad = threading.Barrier(threads), []

    def work(k):
        torch.cuda.set_device(cuda_device)
        go.wait()
        for _ in range(calls):
            got = _read(ctypes.c_void_p(ws.data_ptr() + 4 * k), ctypes.c_void_p(num.data_ptr() + 4 * k), 1 << 20,
                        streams[k])
            if got != (R.GSR_OK, 3 * k):
                bad.append((k, got))

    ts = [threading.Thread(target=work, args=(k,)) for k in range(threads)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad, bad[:3]


RESET = """
import ctypes, sys
sys.path.insert(0, %r)
from polysplat_gb300._lib import lib
rt = ctypes.CDLL("libcudart.so.13")
for value in (5, 9):
    p = ctypes.c_void_p()
    assert rt.cudaMalloc(ctypes.byref(p), 8) == 0
    word = ctypes.c_int32(value)
    assert rt.cudaMemset(p, 0, 8) == 0
    assert rt.cudaMemcpy(p, ctypes.byref(word), 4, 1) == 0
    n = ctypes.c_int32(-1)
    for _ in range(3):
        assert lib().gsr_read_status(ctypes.c_void_p(p.value + 4), p, 100, ctypes.byref(n), None) == 0
        assert n.value == value, n.value
    assert rt.cudaDeviceReset() == 0
print("ok")
"""


def test_the_block_is_made_again_after_a_device_reset(cuda_device):
    import os

    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", RESET % root], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stderr[-2000:]
