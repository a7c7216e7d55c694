"""The bin scatter where its block chooses another way, against the oracle's int64 sums: cells
piled on a few bins (the shared tile, 32- and 64-bit), spread evenly (straight to HBM), macros of
many bins among them (taken by their warps; also alone, and narrower than a warp), cells past
the grid's edges, and a clump whose cells straddle its corner."""
import ctypes as C

import numpy as np
import pytest

import oracle
from tests.gpu_util import dev, ptr, stream, sync

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,clump,macros", [(64, 64, 0.02, 0.0), (64, 64, 0.02, 0.02), (64, 64, 1.0, 0.02), (8, 8, 0.05, 0.0), (300, 7, 0.1, 0.1), (200, 150, 0.0, 1.0), (64, 64, -0.01, 0.01)])
@pytest.mark.parametrize("form", ["tiles", "global", "pooled"])
def test_clumped_scatter_bit_exact(nx, ny, clump, macros, form, monkeypatch):
    from gpl_b200 import engine
    monkeypatch.setenv("GPL_SCATTER", form)
    rng = np.random.default_rng(nx + ny + int(1000 * abs(clump)))
    n = 3001
    w, h = 1929.6 if nx > 8 else 15000.2, 1195.4 if ny > 8 else 9000.7
    bx = np.array([1000 + int(np.floor(i * w + 0.5)) for i in range(nx + 1)], np.int32)
    by = np.array([-500 + int(np.floor(j * h + 0.5)) for j in range(ny + 1)], np.int32)
    W, H = bx[-1] - bx[0], by[-1] - by[0]
    mid = (bx[0], by[0]) if clump < 0 else ((bx[0] + bx[-1]) // 2, (by[0] + by[-1]) // 2)
    cx = (mid[0] + rng.uniform(-0.5, 0.5, n) * W * abs(clump)).astype(np.int32)
    cy = (mid[1] + rng.uniform(-0.5, 0.5, n) * H * abs(clump)).astype(np.int32)
    hx, hy = rng.integers(100, int(0.8 * w), n).astype(np.int32), rng.integers(100, int(0.8 * h), n).astype(np.int32)
    kind = rng.choice([0, 2], n, p=[0.8, 0.2]).astype(np.uint8)
    big = rng.random(n) < macros
    kind[big] = 1
    hx[big] = rng.integers(int(2 * w), int(0.4 * W) + int(2 * w) + 1, big.sum())
    hy[big] = rng.integers(int(2 * h), int(0.4 * H) + int(2 * h) + 1, big.sum())
    sc = rng.uniform(0.2, 1.0, n).astype(np.float32)
    want = [np.zeros(nx * ny, np.int64) for _ in range(2)]
    vp = lambda a: a.ctypes.data_as(C.c_void_p)
    oracle.lib().oracle_density_scatter(C.c_int64(n), *[vp(a) for a in (cx, cy, hx, hy, sc, kind)], nx, ny, int(bx[0]), int(by[0]), vp(bx), vp(by), C.c_double(w), C.c_double(h), C.c_float(0.7), *[vp(a) for a in want])
    d = [dev(a) for a in (cx, cy, hx, hy, sc, kind, bx, by)]
    got = [dev(np.zeros(nx * ny, np.int64)) for _ in range(2)]
    assert engine.lib().gpl_kernel_density_scatter(n, *[ptr(t) for t in d[:6]], nx, ny, int(bx[0]), int(by[0]), ptr(d[6]), ptr(d[7]), w, h, 0.7, *[ptr(t) for t in got], stream()) == 0
    sync()
    for g, v in zip(got, want):
        np.testing.assert_array_equal(g.cpu().numpy(), v)
