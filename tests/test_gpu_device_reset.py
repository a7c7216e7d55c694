"""The per-kernel entry points after the device's context has been reset by its owner
(cudaDeviceReset, in a process of its own): calls before and after give the same results. The HPWL
takes scratch from the library's pool; the density solve on the tensor cores asks for its kernels'
shared memory, whose tiles are of another width on each of its grids."""
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
L.gpl_kernel_poisson.argtypes = [C.c_int32, C.c_int32] + [C.c_void_p] * 5 + [C.c_int, C.c_void_p]
sides = (512, 768, 1024)  # tiles 32, 64 and 128 wide for the pairs
density = {{m: np.random.default_rng(m).random(m * m).astype(np.float32) for m in sides}}
fields = {{}}


def solve(m):
    w = (np.pi * np.arange(m) / m).astype(np.float32)
    d, gx, gy, out = dev(density[m]), dev(density[m]), dev(density[m]), np.empty(m * m, np.float32)
    assert L.gpl_kernel_poisson(m, m, w.ctypes.data, w.ctypes.data, d, gx, gy, 1, None) == 0
    assert R.cudaMemcpy(out.ctypes.data_as(C.c_void_p), gx, C.c_size_t(out.nbytes), 2) == 0
    return out


for turn in range(3):
    for m in sides:
        got = solve(m)
        assert np.abs(got).max() > 0 and (fields.setdefault(m, got) == got).all()
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
