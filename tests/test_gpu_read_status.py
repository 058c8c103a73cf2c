"""gsr_read_status: the words a kernel writes to host memory and the copies it
falls back to give the same result, on several host threads and streams at once;
host arguments read in place equal converted ones."""
import ctypes
import threading

import pytest
import torch

from polysplat_gb300 import _lib as R
from polysplat_gb300 import ops
from polysplat_gb300._lib import lib

pytestmark = pytest.mark.gpu


def _read(ws, num, cap, stream):
    n = ctypes.c_int32(-1)
    st = lib().gsr_read_status(ws, num, cap, ctypes.byref(n), ctypes.c_void_p(stream.cuda_stream))
    return st, n.value


@pytest.mark.parametrize("num,cap,expect", [(0, 0, R.GSR_OK), (7, 7, R.GSR_OK), (8, 7, R.GSR_OVERFLOW)])
@pytest.mark.parametrize("shift", [0, 2])  # 2: not on a word boundary, so copied
def test_count_and_status(cuda_device, num, cap, expect, shift):
    s = torch.cuda.Stream(cuda_device)
    b = torch.zeros(64, dtype=torch.uint8, device=cuda_device)
    b[16 + shift] = num
    torch.cuda.synchronize()
    ws, cnt = ctypes.c_void_p(b.data_ptr() + 32 + shift), ctypes.c_void_p(b.data_ptr() + 16 + shift)
    assert _read(ws, cnt, cap, s) == (expect, num)
    assert _read(None, cnt, cap, s) == (expect, num)
    assert _read(ws, None, cap, s) == (R.GSR_OK, 0)


def test_threads_read_their_own_words(cuda_device):
    bad = []

    def work(k):
        s = torch.cuda.Stream(cuda_device)
        with torch.cuda.stream(s):
            ws = torch.zeros(4, dtype=torch.int32, device=cuda_device)
            num = torch.zeros(1, dtype=torch.int32, device=cuda_device)
            for i in range(200):
                num.fill_(1000 * k + i)
                got = _read(ctypes.c_void_p(ws.data_ptr()), ctypes.c_void_p(num.data_ptr()), 1 << 20, s)
                if got != (R.GSR_OK, 1000 * k + i):
                    bad.append((k, i, got))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad[:3]


@pytest.mark.parametrize("t", [torch.arange(9.0), torch.arange(9.0).double(), torch.arange(18.0)[::2] / 2,
                               list(range(9))])
def test_host_floats(t):
    p = ops._host_floats(t, 9, "x")
    assert list(ctypes.cast(p, ctypes.POINTER(ctypes.c_float))[:9]) == [float(k) for k in range(9)]
    with pytest.raises(ValueError):
        ops._host_floats(t[:5], 9, "x")
