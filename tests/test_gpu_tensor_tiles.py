"""The split-BF16 density solve at the grid sizes where its output tiles' widths change (32, 64
or 128 columns, the single products and the pairs each by their own rule), on square and oblong
grids and with K shorter than its ring of stages, against the FP64 solve. Tolerance: 5e-4 of the
field's maximum, the form's bound everywhere else (three products of 8-bit mantissa halves)."""
import ctypes as C

import numpy as np
import pytest

from gpl_b200 import engine
from gpu_util import dev, ptr, stream, sync

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(128, 128), (128, 640), (640, 512), (512, 640), (768, 768), (896, 896), (1152, 512)])
def test_tensor_tiles(nx, ny):
    L = engine.lib()
    L.gpl_kernel_poisson.argtypes = [C.c_int32, C.c_int32] + [C.c_void_p] * 5 + [C.c_int32, C.c_void_p]
    L.gpl_kernel_poisson_fp64.argtypes = [C.c_int32, C.c_int32] + [C.c_void_p] * 6
    rng = np.random.default_rng(nx * 7 + ny)
    wx = (np.pi * np.arange(nx) / nx).astype(np.float32)
    wy = (np.pi * np.arange(ny) / ny * 1.5).astype(np.float32)
    d = dev((rng.random(nx * ny) * 1.5).astype(np.float32))
    ex, ey = dev(np.zeros(nx * ny)), dev(np.zeros(nx * ny))
    assert L.gpl_kernel_poisson_fp64(nx, ny, wx.ctypes.data, wy.ctypes.data, ptr(d), ptr(ex), ptr(ey), stream()) == 0
    gx, gy = dev(np.full(nx * ny, np.nan, np.float32)), dev(np.full(nx * ny, np.nan, np.float32))
    assert L.gpl_kernel_poisson(nx, ny, wx.ctypes.data, wy.ctypes.data, ptr(d), ptr(gx), ptr(gy), 1, stream()) == 0
    sync()
    for g, e in ((gx, ex), (gy, ey)):
        g, e = g.cpu().numpy(), e.cpu().numpy()
        assert np.max(np.abs(g - e)) <= 5e-4 * np.max(np.abs(e))
