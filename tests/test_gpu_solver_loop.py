"""The solver's persistent loop (`bicgstab`, src/bicgstab.rs:615-669) where its shape changes,
against the oracle: one block and several, rows that do not fill a run of four, the last blocks
partly or wholly idle, a start point off a 16-byte boundary (its vector steps then take one
element a thread), and a row longer than the products a block holds at once. The systems
converge, so the solution agrees within the tolerance of the solver's parity test (1e-4 of the
largest entry, relative 1e-4); the iteration counts may differ by the inner products' rounding."""
import ctypes as C

import numpy as np
import pytest

import oracle
from tests.gpu_util import dev, ptr, stream

pytestmark = pytest.mark.gpu


def system(n, seed, long_row):
    rng = np.random.default_rng(seed)
    a, b = rng.integers(0, n, 3 * n), rng.integers(0, n, 3 * n)
    if long_row:
        others = rng.choice(np.arange(1, n), long_row, replace=False)
        a, b = np.concatenate([a, np.zeros(long_row, np.int64)]), np.concatenate([b, others])
    keep = a != b
    a, b = a[keep], b[keep]
    w = rng.uniform(0.01, 0.5, len(a)).astype(np.float32)
    diag = np.zeros(n)
    np.add.at(diag, a, w)
    np.add.at(diag, b, w)
    rows = np.concatenate([a, b, np.arange(n)]).astype(np.int64)
    cols = np.concatenate([b, a, np.arange(n)]).astype(np.int64)
    vals = np.concatenate([-w, -w, (diag + rng.uniform(0.1, 0.3, n)).astype(np.float32)]).astype(np.float32)
    starts, oc, ov = np.zeros(n + 1, np.int64), np.zeros(len(rows), np.int32), np.zeros(len(rows), np.float32)
    nnz = oracle.lib().oracle_csr_from_triplets(n, len(rows), rows.ctypes.data, cols.ctypes.data, vals.ctypes.data, starts.ctypes.data, oc.ctypes.data, ov.ctypes.data)
    return starts, oc[:nnz].copy(), ov[:nnz].copy(), rng.uniform(-1e5, 1e5, n).astype(np.float32), rng.uniform(0, 1e4, n).astype(np.float32)


@pytest.mark.parametrize("n,shift,long_row", [(1, 0, 0), (3, 0, 0), (512, 0, 0), (513, 0, 0), (4099, 1, 0), (30001, 0, 24000), (151553, 0, 0), (310007, 1, 300)])
def test_solver_loop_matches_the_oracle(n, shift, long_row):
    import torch
    from gpl_b200 import engine
    starts, cols, vals, rhs, x0 = system(n, 100 + n, long_row)
    want, err, conv = x0.copy(), C.c_float(), C.c_int()
    oracle.lib().oracle_bicgstab(n, starts.ctypes.data, cols.ctypes.data, vals.ctypes.data, rhs.ctypes.data, want.ctypes.data, 100, C.byref(err), C.byref(conv))
    d = [dev(a) for a in (starts, cols, vals, rhs)]
    buf = torch.zeros(n + 8, dtype=torch.float32, device="cuda")
    x = buf[shift:shift + n]
    x.copy_(dev(x0))
    it, gerr = C.c_int32(), C.c_float()
    assert engine.lib().gpl_kernel_bicgstab(n, *[ptr(t) for t in d], ptr(x), 100, C.byref(it), C.byref(gerr), stream()) == 0
    assert 0 < it.value <= 100 and gerr.value < 1e-5
    np.testing.assert_allclose(x.cpu().numpy(), want, rtol=1e-4, atol=1e-4 * np.max(np.abs(want)))
    # nothing past the solution is written
    assert not buf[:shift].any() and not buf[shift + n:].any()
