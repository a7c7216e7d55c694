"""The sliced loop's items (long rows, slices of 32 rows) taken by a block's warps as they end:
it takes more items than the block's sixteen warps, which each case here has by its row lengths
(asserted). Against the rows form: both axes' solutions and iterations bit for bit. One block with
one item too many and with many long rows, several blocks, blocks with one item more than others,
and a full grid; the last slice partly filled."""
import ctypes as C

import numpy as np
import pytest

from tests.gpu_util import dev, ptr, stream

pytestmark = pytest.mark.gpu

WARPS, ROWS, SLICE, LONG = 16, 512, 32, 64  # of the loop's kernel and the sliced copy


def system(n, n_long, seed):
    """Rows of up to seven entries, n_long of 65 to 400; each diagonally dominant, columns ascending."""
    rng = np.random.default_rng(seed)
    length = rng.integers(1, 8, n)
    at = rng.choice(n, n_long, replace=False)
    length[at] = rng.integers(LONG + 1, min(400, n // 2) + 1, n_long)
    starts = np.concatenate([[0], np.cumsum(length)]).astype(np.int64)
    cols = np.empty(starts[-1], np.int32)
    vals = rng.uniform(-1, 1, starts[-1]).astype(np.float32)
    for i in range(n):
        k = int(length[i])
        c = i + np.arange(k) * max(1, n // (k + 1))  # distinct modulo n: k steps of less than n / k
        c = np.sort(c % n)
        b = starts[i]
        cols[b:b + k] = c
        vals[b + int(np.flatnonzero(c == i)[0])] = 2.0 + k
    return length, starts, cols, vals, rng.uniform(-1, 1, n).astype(np.float32)


@pytest.mark.parametrize("n,n_long", [(512, 1), (500, 90), (2048, 5), (5000, 300), (5121, 20), (80_000, 40)])
def test_items_taken_match_rows(n, n_long):
    import torch
    from gpl_b200 import engine
    L = engine.lib()
    L.gpl_rules_bicgstab_pair.argtypes = [C.c_int64] + [C.c_void_p] * 6 + [C.c_int32] * 2 + [C.c_void_p] * 3
    length, starts, cols, vals, rhs = system(n, n_long, n)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    blocks = min(sms, -(-n // ROWS))  # a system's: two blocks an SM, two systems
    long_rows = int((length > LONG).sum())
    items = long_rows + -(-(n - long_rows) // SLICE)
    assert long_rows == n_long and -(-items // blocks) > WARPS
    d = [dev(a) for a in (starts, cols, vals, rhs)]
    runs = []
    for form in (0, 2):
        x = [torch.zeros(n, device="cuda"), torch.full((n,), 0.5, device="cuda")]
        it, err = (C.c_int32 * 2)(), (C.c_float * 2)()
        assert L.gpl_rules_bicgstab_pair(n, *[ptr(t) for t in d], ptr(x[0]), ptr(x[1]), 100, form, it, err, stream()) == 0
        runs.append((list(it), list(err), x))
    assert all(0 < k < 100 for k in runs[0][0]) and max(runs[0][1]) < 1e-5
    assert runs[0][:2] == runs[1][:2]
    assert all(torch.equal(a, b) for a, b in zip(runs[0][2], runs[1][2]))
