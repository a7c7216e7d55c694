"""The solver on row starts that do not ascend: row i is the window [start i, start i + 1) of the
entries, empty where it ends before it starts, and windows may share entries. Against the oracle
over three iterations (the rows are summed in the same order; the inner products' rounding moves
the third iterate by far less than the tolerance, the solver parity test's relative 1e-4)."""
import ctypes as C

import numpy as np
import pytest

import oracle
from tests.gpu_util import dev, ptr, stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,back", [(20, (5,)), (700, (5, 128, 256, 640)), (3000, (1, 512, 1024, 2998))])
def test_row_windows_in_any_order(n, back):
    from gpl_b200 import engine
    rng = np.random.default_rng(n)
    w = np.arange(-4, 5)
    cols = np.arange(n)[:, None] + w
    ok = (cols >= 0) & (cols < n)
    vals = np.where(w == 0, 9.0, rng.uniform(-1.0, -0.5, cols.shape))[ok].astype(np.float32)
    starts = np.concatenate([[0], np.cumsum(ok.sum(1))]).astype(np.int64)
    cols = cols[ok].astype(np.int32)
    for i in back:
        starts[i] = starts[i + 1] + 3  # row i - 1 reaches into the rows after it, row i is empty
    assert (np.diff(starts) < 0).sum() == len(back) and 0 <= starts.min() and starts.max() <= len(cols)
    rhs, x0 = rng.uniform(-1, 1, n).astype(np.float32), rng.uniform(-1, 1, n).astype(np.float32)
    want, err, conv = x0.copy(), C.c_float(), C.c_int()
    oracle.lib().oracle_bicgstab(n, starts.ctypes.data, cols.ctypes.data, vals.ctypes.data, rhs.ctypes.data, want.ctypes.data, 3, C.byref(err), C.byref(conv))
    d = [dev(a) for a in (starts, cols, vals, rhs)]
    x, it, gerr = dev(x0), C.c_int32(), C.c_float()
    assert engine.lib().gpl_kernel_bicgstab(n, *[ptr(t) for t in d], ptr(x), 3, C.byref(it), C.byref(gerr), stream()) == 0
    assert it.value == 3
    np.testing.assert_allclose(x.cpu().numpy(), want, rtol=1e-4, atol=1e-4 * np.max(np.abs(want)))
