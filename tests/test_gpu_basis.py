"""The density solve's basis matrices as the device makes them, against the host library's cosine
and sine (the same double arguments, rounded once to float), bit for bit: small, odd, rectangular
and large grids; every entry of the small ones, a sample of the large."""
import ctypes as C
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def entry(which, r, c, n):
    k, j = (r, c) if which < 2 else (c, r)
    a = math.pi * float(k) * (float(j) + 0.5) / float(n)
    if which in (3, 4):
        return (-1.0 if j & 1 else 1.0) if k == 0 else math.sin(a)
    return ((0.5 if r == 0 else 1.0) * 2.0 / float(n)) * math.cos(a) if which < 2 else math.cos(a)


@pytest.mark.parametrize("nx,ny", [(1, 1), (5, 64), (96, 37), (257, 300), (1024, 1024), (3001, 640)])
def test_device_basis_equals_the_host_library(nx, ny):
    from gpl_b200 import engine
    L = engine.lib()
    L.gpl_rules_basis.argtypes = [C.c_int32, C.c_int32, C.c_void_p]
    sides = (ny, nx, ny, ny, nx, nx)
    out = np.zeros(sum(s * s for s in sides), np.float32)
    assert L.gpl_rules_basis(nx, ny, out.ctypes.data) == 0
    rng = np.random.default_rng(nx + ny)
    at = 0
    for which, n in enumerate(sides):
        got = out[at:at + n * n]
        at += n * n
        idx = np.arange(n * n) if n * n <= 20_000 else rng.integers(0, n * n, 60_000)
        want = np.array([entry(which, int(i) // n, int(i) % n, n) for i in idx], np.float64).astype(np.float32)
        assert np.array_equal(got[idx].view(np.uint32), want.view(np.uint32)), (which, n)
