"""gv_mtx_parse keeps a block of device memory per thread between calls.  A
device reset takes that block away; the next parse makes its own, also where
the old address belongs to someone else by then."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

CHILD = r"""
import ctypes as C
import glob, os, threading
import numpy as np
from gv_b200 import _lib

L = _lib.lib()
rt = C.CDLL("libcudart.so.12") if not glob.glob("/usr/local/cuda/lib64/libcudart.so") \
    else C.CDLL("/usr/local/cuda/lib64/libcudart.so")

def text(k):
    return b"%%MatrixMarket matrix coordinate pattern general\n" + b"%d %d %d\n" % (k, k, k) + \
        b"".join(b"%d %d\n" % (i + 1, k - i) for i in range(k))

def parse(k):
    t = text(k)
    info, count = _lib.gv_mtx_info(), C.c_uint64()
    s, d = np.empty(k, np.uint32), np.empty(k, np.uint32)
    st = L.gv_mtx_parse(t, len(t), 0, C.byref(info), s.ctypes.data, d.ctypes.data, None, k, C.byref(count), None)
    assert st == 0, (st, L.gv_last_error_string())
    assert count.value == k and np.array_equal(s, np.arange(k)) and np.array_equal(d, np.arange(k)[::-1])

def others():
    # small blocks of a known pattern, where the kept one was among them
    ps = []
    for _ in range(64):
        p = C.c_void_p()
        assert rt.cudaMalloc(C.byref(p), C.c_size_t(4096)) == 0
        assert rt.cudaMemset(p, 0x5A, C.c_size_t(4096)) == 0
        ps.append(p)
    return ps

def untouched(ps):
    for p in ps:
        b = np.zeros(4096, np.uint8)
        assert rt.cudaMemcpy(C.c_void_p(b.ctypes.data), p, C.c_size_t(4096), 2) == 0
        assert np.all(b == 0x5A)

parse(1000)
parse(1000)
assert rt.cudaDeviceReset() == 0
ps = others()
parse(1000)          # the same size: the old block would do
parse(200000)        # a larger one: the old block would be given back
untouched(ps)
# a thread that ends after a reset gives nothing back that is not its own
go, ready = threading.Event(), threading.Event()
def one():
    parse(500)
    ready.set()
    go.wait()
t = threading.Thread(target=one)
t.start()
ready.wait()
assert rt.cudaDeviceReset() == 0
ps = others()
go.set()
t.join()
untouched(ps)
parse(1000)
untouched(ps)
print("fine")
"""


def test_parse_after_device_reset():
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "fine", r.stdout + r.stderr
