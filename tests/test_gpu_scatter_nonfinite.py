"""The bin scatter with density scales (or a target density) that are not finite: such a cell may
give any value to the bins of its own span, but no other bin, nothing past the accumulators.
Every other bin holds the oracle's sums of the other cells, exactly. The bad cells lie in the
grid's far corner and inside it, one to three bins an axis, among cells spread evenly and piled
up (the shared tile), with 32- and 64-bit slots."""
import ctypes as C

import numpy as np
import pytest

import oracle
from tests.gpu_util import dev, ptr, stream, sync

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["tiles", "global", "pooled"])
@pytest.mark.parametrize("bad,macro", [(np.inf, False), (np.nan, False), (-np.inf, False), (np.nan, True)])
@pytest.mark.parametrize("nx,ny,clump", [(64, 64, 1.0), (64, 64, 0.05), (8, 8, 0.3)])
def test_nonfinite_scale_stays_in_its_bins(nx, ny, clump, bad, macro, form, monkeypatch):
    import torch
    from gpl_b200 import engine
    monkeypatch.setenv("GPL_SCATTER", form)
    rng = np.random.default_rng(nx + int(100 * clump))
    n = 2000
    w, h = (1929.6, 1195.4) if nx > 8 else (15000.2, 9000.7)
    bx = np.array([1000 + int(np.floor(i * w + 0.5)) for i in range(nx + 1)], np.int32)
    by = np.array([-500 + int(np.floor(j * h + 0.5)) for j in range(ny + 1)], np.int32)
    # piled up towards the far corner, so the bad cells share blocks and tiles with the others
    cx = (bx[-1] - rng.uniform(0, clump, n) * (bx[-1] - bx[0])).astype(np.int32)
    cy = (by[-1] - rng.uniform(0, clump, n) * (by[-1] - by[0])).astype(np.int32)
    hx, hy = rng.integers(100, int(0.8 * w), n).astype(np.int32), rng.integers(100, int(0.8 * h), n).astype(np.int32)
    kind = rng.choice([0, 2], n, p=[0.8, 0.2]).astype(np.uint8)
    sc = rng.uniform(0.2, 1.0, n).astype(np.float32)
    # the bad cells: the far corner's bin alone, its column, its row, and one inside; of both arrays
    at = [(0, 0, 0.4, 0.4), (0, 0, 0.4, 1.2), (0, 0, 1.2, 0.4), (2, 2, 0.9, 0.9), (2, 1, 0.3, 0.3), (0, 0, 0.4, 0.4)]
    ids = np.arange(0, n, n // len(at))[:len(at)]
    for i, (bxi, byi, fx, fy) in zip(ids, at):
        cx[i], cy[i] = bx[-1] - int((bxi + 0.5) * w), by[-1] - int((byi + 0.5) * h)
        hx[i], hy[i] = int(fx * w), int(fy * h)
    kind[ids] = 1 if macro else [0, 0, 2, 0, 2, 2]
    td = np.float32(np.nan if macro else 0.7)
    if not macro:
        sc[ids] = np.float32(bad)
    spans = np.zeros((nx, ny), bool)
    for i in ids:
        x0, x1 = int((cx[i] - hx[i] - bx[0]) / w), int(np.ceil((cx[i] + hx[i] - bx[0]) / w))
        y0, y1 = int((cy[i] - hy[i] - by[0]) / h), int(np.ceil((cy[i] + hy[i] - by[0]) / h))
        spans[max(x0, 0):min(x1, nx), max(y0, 0):min(y1, ny)] = True
    assert 1 <= spans.sum() < 40
    good = sc.copy()
    good[ids] = 0.0
    want = [np.zeros(nx * ny, np.int64) for _ in range(2)]
    vp = lambda a: a.ctypes.data_as(C.c_void_p)
    oracle.lib().oracle_density_scatter(C.c_int64(n), *[vp(a) for a in (cx, cy, hx, hy, good, kind)], nx, ny, int(bx[0]), int(by[0]), vp(bx), vp(by), C.c_double(w), C.c_double(h), C.c_float(0.7), *[vp(a) for a in want])
    d = [dev(a) for a in (cx, cy, hx, hy, sc, kind, bx, by)]
    pad = 4 * ny
    got = [torch.full((nx * ny + 2 * pad,), 7, dtype=torch.int64, device="cuda") for _ in range(2)]
    assert engine.lib().gpl_kernel_density_scatter(n, *[ptr(t) for t in d[:6]], nx, ny, int(bx[0]), int(by[0]), ptr(d[6]), ptr(d[7]), w, h, td, *[ptr(t[pad:]) for t in got], stream()) == 0
    sync()
    out = ~spans.reshape(-1)
    for g, v in zip(got, want):
        a = g.cpu().numpy()
        np.testing.assert_array_equal(a[pad:-pad][out], v[out])
        assert (a[:pad] == 7).all() and (a[-pad:] == 7).all()
