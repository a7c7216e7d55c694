"""The two objectives' kernels at the edges of their shapes. The wirelength (value and gradient)
against the same formula in torch double precision: nets without pins, one pin, block runs that
fit the staged pins exactly and that do not, one net alone, off weights. The double GEMM (under
the density objective and the FP64 solve) at sides that end inside its tiles, chunks and pairs,
against the separate double solve, within float rounding of the fields."""
import ctypes as C

import numpy as np
import pytest

from tests.gpu_util import dev, ptr, stream, sync

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degrees", [[1], [0, 0, 3], [2] * 127, [8] * 128, [8] * 127 + [9] + [2] * 5, [3000], [0, 1, 2, 40, 700] * 60])
@pytest.mark.parametrize("weights", [True, False])
def test_wirelength_value_and_gradient(degrees, weights):
    import torch
    from gpl_b200 import engine, functions
    functions._lib()
    rng = np.random.default_rng(len(degrees))
    deg = np.array(degrees)
    start = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
    xy = torch.from_numpy(rng.uniform(-20000, 20000, (int(start[-1]), 2))).cuda()
    w = torch.from_numpy(rng.uniform(0.5, 2.0, len(deg)).astype(np.float32)).cuda() if weights else None
    cx, cy = 4e-4, 7e-4
    L, d = engine.lib(), dev(start)
    v, g = C.c_double(), torch.zeros_like(xy)
    pw = ptr(w) if weights else None
    assert L.gpl_fn_wa_forward(len(deg), ptr(d), ptr(xy), pw, cx, cy, C.byref(v), stream()) == 0
    assert L.gpl_fn_wa_backward(len(deg), ptr(d), ptr(xy), pw, cx, cy, 1.7, ptr(g), stream()) == 0
    x = xy.clone().requires_grad_(True)
    total = torch.zeros((), dtype=torch.float64, device="cuda")
    for n in np.flatnonzero(deg):
        p = x[start[n]:start[n + 1]]
        for a, c in enumerate((cx, cy)):
            q = p[:, a]
            ep, em = torch.exp(c * (q - q.max().detach())), torch.exp(c * (q.min().detach() - q))
            total = total + (float(w[n]) if weights else 1.0) * ((q * ep).sum() / ep.sum() - (q * em).sum() / em.sum())
    total.backward()
    # sums of at most 3000 positive terms in double: a few thousand roundings of 1.1e-16
    scale = float(x.grad.abs().max())
    assert abs(v.value - float(total.detach())) <= 1e-11 * max(1.0, float(xy.abs().max()) * len(deg))
    assert float((g - 1.7 * x.grad).abs().max()) <= 1e-11 * max(scale, 1.0)


@pytest.mark.parametrize("nx,ny", [(1, 2), (3, 5), (16, 64), (37, 91), (65, 33), (130, 258)])
def test_double_gemm_at_tile_edges(nx, ny):
    from gpl_b200 import engine
    L = engine.lib()
    L.gpl_kernel_poisson_fp64.argtypes = [C.c_int32, C.c_int32] + [C.c_void_p] * 6
    rng = np.random.default_rng(nx * 5 + ny)
    n = nx * ny
    wx = (np.pi * np.arange(nx) / nx).astype(np.float32)
    wy = (np.pi * np.arange(ny) / ny * 1.4).astype(np.float32)
    d = dev((rng.random(n) * 1.5).astype(np.float32))
    g = [dev(np.zeros(n, np.float32)) for _ in range(2)]
    h = [dev(np.zeros(n)) for _ in range(2)]
    assert L.gpl_kernel_poisson(nx, ny, wx.ctypes.data, wy.ctypes.data, ptr(d), ptr(g[0]), ptr(g[1]), 2, stream()) == 0
    assert L.gpl_kernel_poisson_fp64(nx, ny, wx.ctypes.data, wy.ctypes.data, ptr(d), ptr(h[0]), ptr(h[1]), stream()) == 0
    sync()
    for a, b in zip(g, h):
        a, b = a.cpu().numpy().astype(np.float64), b.cpu().numpy()
        assert np.max(np.abs(a - b)) <= 1e-6 * max(np.max(np.abs(b)), 1e-30)
