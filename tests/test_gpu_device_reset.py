"""The per-kernel entry points' scratch after the device's context has been reset by its owner
(cudaDeviceReset, in a process of its own): calls before and after give the same results."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import ctypes as C
import numpy as np
L = C.CDLL({so!r})
R = C.CDLL(next(l.split()[-1] for l in open("/proc/self/maps") if "libcudart" in l))


def dev(a):
    p = C.c_void_p()
    assert R.cudaMalloc(C.byref(p), C.c_size_t(a.nbytes)) == 0
    assert R.cudaMemcpy(p, a.ctypes.data_as(C.c_void_p), C.c_size_t(a.nbytes), 1) == 0
    return p


n = 2000
start = (4 * np.arange(n + 1)).astype(np.int64)
xy = np.random.default_rng(0).integers(0, 10000, (4 * n, 2)).astype(np.int32)
q = xy.reshape(n, 4, 2).astype(np.int64)
want = int((q.max(1) - q.min(1)).sum())
L.gpl_kernel_hpwl.argtypes = [C.c_int64, C.c_void_p, C.c_void_p, C.c_int32, C.c_void_p, C.c_void_p]
for turn in range(3):
    for fused in (0, 1, 1):
        h = C.c_int64()
        assert L.gpl_kernel_hpwl(n, dev(start), dev(xy), fused, C.byref(h), None) == 0 and h.value == want
    assert R.cudaDeviceReset() == 0
print("ok")
"""


def test_calls_after_a_reset():
    from gpl_b200 import build
    r = subprocess.run([sys.executable, "-c", CHILD.format(so=build.SO)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stderr[-2000:]
    assert os.path.exists(build.SO)
