"""The solver's bounded waits: a wait limit set to next to nothing on a system with one long row
(every block but its own waits at the barrier after each product) runs out, the call returns the
time-out error at once, and the next call on the same data solves as before. Also on a thread
that takes denormal numbers for zero, where the error word must still be seen. With the limit's
share for the matrix's entries alone, the same system solves: a long step is no lost block."""
import ctypes as C
import time

import numpy as np
import pytest

from tests.gpu_util import dev, ptr, stream

pytestmark = pytest.mark.gpu

LAUNCH_TIMEOUT = 702  # cudaErrorLaunchTimeout


def long_row_system(n):
    """Row 0 over every column with small weights, the other rows their diagonal and column 0."""
    starts = np.concatenate([[0], n + 2 * np.arange(n)]).astype(np.int64)
    cols = np.empty(n + 2 * (n - 1), np.int32)
    vals = np.empty(len(cols), np.float32)
    cols[:n], vals[:n] = np.arange(n), -0.1 / n
    vals[0] = 2.0
    cols[n::2], cols[n + 1::2] = 0, np.arange(1, n)
    vals[n::2], vals[n + 1::2] = -0.1, 2.0 + np.arange(n - 1) % 7
    rhs = np.random.default_rng(3).uniform(-1, 1, n).astype(np.float32)
    return starts, cols, vals, rhs


def calls(n):
    import torch
    from gpl_b200 import engine
    L = engine.lib()
    L.gpl_rules_bicgstab_wait.argtypes = [C.c_int64] + [C.c_void_p] * 5 + [C.c_int32] + [C.c_void_p] * 2 + [C.c_uint64, C.c_uint64, C.c_void_p]
    starts, cols, vals, rhs = long_row_system(n)
    assert starts[-1] == len(cols) and cols.min() == 0 and cols.max() == n - 1
    d = [dev(a) for a in (starts, cols, vals, rhs)]

    def solve(wait=None):
        x, it, err = torch.zeros(n, device="cuda"), C.c_int32(), C.c_float()
        args = [n] + [ptr(t) for t in d] + [ptr(x), 100, C.byref(it), C.byref(err)]
        rc = L.gpl_kernel_bicgstab(*args, stream()) if wait is None else L.gpl_rules_bicgstab_wait(*args, *wait, stream())
        return rc, it.value, err.value, x
    return solve


@pytest.mark.parametrize("flush", [False, True])
def test_a_wait_that_runs_out_is_an_error(flush):
    import torch
    solve = calls(1_000_003)
    want = solve()
    assert want[0] == 0 and 0 < want[1] < 100 and want[2] < 1e-5
    assert torch.set_flush_denormal(flush) or not flush
    try:
        t = time.time()
        assert solve((1, 0))[0] == LAUNCH_TIMEOUT
        assert time.time() - t < 1.0
    finally:
        torch.set_flush_denormal(False)
    again = solve()
    assert again[0] == 0 and again[1] == want[1] and torch.equal(again[3], want[3])


def test_the_limit_grows_with_the_entries():
    import torch
    solve = calls(1_000_003)
    want, got = solve(), solve((1, 200))
    assert want[0] == 0 and got[:3] == want[:3] and torch.equal(got[3], want[3])
