"""The FP32 density solve's GEMM tiles at the edges of their shapes, against the double solve
(`gpl_kernel_poisson_fp64`, itself checked against the oracle): sides that end inside a tile or
inside a run of four, one chunk and several, both tile sizes, and density and field arrays off a
16-byte boundary. The FP32 form's bound is 1e-4 of the field's largest value."""
import ctypes as C

import numpy as np
import pytest

from tests.gpu_util import dev, ptr, stream, sync

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,shift", [(2, 3, 0), (5, 32, 0), (31, 33, 0), (64, 96, 0), (64, 64, 1), (130, 67, 3), (257, 129, 0), (1024, 1024, 0), (1030, 1025, 1)])
def test_fp32_solve_at_tile_edges(nx, ny, shift):
    import torch
    from gpl_b200 import engine
    L = engine.lib()
    L.gpl_kernel_poisson_fp64.argtypes = [C.c_int32, C.c_int32] + [C.c_void_p] * 6
    rng = np.random.default_rng(nx * 11 + ny)
    n = nx * ny
    wx = (np.pi * np.arange(nx) / nx).astype(np.float32)
    wy = (np.pi * np.arange(ny) / ny * 1.4).astype(np.float32)
    hold = [torch.zeros(n + 8, dtype=torch.float32, device="cuda") for _ in range(3)]
    d, gx, gy = (t[shift:shift + n] for t in hold)
    d.copy_(dev((rng.random(n) * 1.5).astype(np.float32)))
    assert L.gpl_kernel_poisson(nx, ny, wx.ctypes.data, wy.ctypes.data, ptr(d), ptr(gx), ptr(gy), 0, stream()) == 0
    ex, ey = dev(np.zeros(n)), dev(np.zeros(n))
    d0 = d.clone()
    assert L.gpl_kernel_poisson_fp64(nx, ny, wx.ctypes.data, wy.ctypes.data, ptr(d0), ptr(ex), ptr(ey), stream()) == 0
    sync()
    for got, want in ((gx, ex), (gy, ey)):
        g, w = got.cpu().numpy().astype(np.float64), want.cpu().numpy()
        assert np.max(np.abs(g - w)) <= 1e-4 * np.max(np.abs(w))
    # nothing outside the fields is written
    for t in hold[1:]:
        assert not t[:shift].any() and not t[shift + n:].any()
