"""The wirelength forces of few nets, whose two kernels run in one launch, against the oracle bit
for bit: one part alone (small degrees, large degrees), both, partly filled warps and tiles, and
a net larger than a tile beside them; and the same nets' HPWL, alone and beside the forces."""
import ctypes as C

import numpy as np
import pytest

import oracle
from tests.gpu_util import dev, ptr, stream, sync

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 1])  # positions on an 8-byte boundary, or off it
@pytest.mark.parametrize("degrees", [[2], [4, 4, 4], [9], [512, 1, 0, 5], [2] * 129 + [3] * 81 + [4] * 65 + [5] * 40 + [16] * 33 + [600], list(range(0, 40)) * 50])
def test_few_nets_bit_exact(degrees, shift):
    import torch
    from gpl_b200 import engine
    rng = np.random.default_rng(len(degrees))
    deg = rng.permutation(degrees)
    start = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
    xy = rng.integers(-300000, 300000, (int(start[-1]), 2)).astype(np.int32)
    w = rng.uniform(1.0, 2.0, len(deg)).astype(np.float32)
    want = np.zeros(2 * len(xy), np.float32)
    oracle.lib().oracle_wa(C.c_int64(len(deg)), start.ctypes.data_as(C.c_void_p), xy.ctypes.data_as(C.c_void_p), w.ctypes.data_as(C.c_void_p), C.c_float(2.7e-4), C.c_float(3.1e-4), want.ctypes.data_as(C.c_void_p))
    hold = torch.zeros(2 * len(xy) + 4, dtype=torch.int32, device="cuda")
    pos = hold[shift:shift + 2 * len(xy)]
    pos.copy_(dev(xy).view(-1))
    d = [dev(start), pos, dev(w)]
    g = dev(np.zeros(2 * len(xy), np.float32))
    assert engine.lib().gpl_kernel_wa(len(deg), *[ptr(t) for t in d], 2.7e-4, 3.1e-4, ptr(g), stream()) == 0
    sync()
    np.testing.assert_array_equal(g.cpu().numpy().view(np.uint32), want.view(np.uint32))
    for fused in (0, 1):
        got = C.c_int64()
        assert engine.lib().gpl_kernel_hpwl(len(deg), ptr(d[0]), ptr(d[1]), fused, C.byref(got), stream()) == 0
        assert got.value == oracle.lib().oracle_hpwl(len(deg), start.ctypes.data_as(C.c_void_p), xy.ctypes.data_as(C.c_void_p))
