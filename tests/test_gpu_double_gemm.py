"""The double GEMM's products bit for bit: each output is the chain of fused multiply-adds over k
in order, from 0, which the C library's fma gives on the host. Sides and depths that end inside a
tile, a chunk, a matrix instruction and a pair; rows apart from one another; arrays off a 16-byte
boundary; values over thirty orders of magnitude, zeros of both signs, infinities and NaN."""
import ctypes as C
import ctypes.util

import numpy as np
import pytest

from tests.gpu_util import ptr, stream, sync

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,pad,shift,odd_values", [(1, 1, 1, 0, 0, False), (65, 33, 17, 0, 0, False), (64, 32, 64, 0, 0, False), (9, 40, 50, 2, 0, False), (70, 5, 35, 1, 1, False), (8, 8, 19, 0, 1, True), (33, 17, 48, 4, 0, True)])
def test_products_are_the_fma_chain(M, N, K, pad, shift, odd_values):
    import torch
    from gpl_b200 import engine
    L = engine.lib()
    L.gpl_rules_dgemm.argtypes = [C.c_int32] * 3 + [C.c_void_p, C.c_int32] * 3 + [C.c_void_p]
    fma = C.CDLL(ctypes.util.find_library("m") or "libm.so.6").fma
    fma.restype, fma.argtypes = C.c_double, [C.c_double] * 3
    rng = np.random.default_rng(M + 100 * K)
    ld = K + pad
    host = [rng.standard_normal((r, ld)) * 10.0 ** rng.integers(-15, 16, (r, ld)) for r in (M, N)]
    if odd_values:
        host[0][0, 0], host[0][1, :] = np.inf, -0.0
        host[1][2, K // 2], host[1][3, :] = np.nan, 0.0
    devs = []
    for h in host:
        buf = torch.zeros(h.size + 2, dtype=torch.float64, device="cuda")
        v = buf[shift:shift + h.size]
        v.copy_(torch.from_numpy(h.reshape(-1)))
        devs.append(v)
    out = torch.full((M * (N + pad) + 2,), 3.25, dtype=torch.float64, device="cuda")
    assert L.gpl_rules_dgemm(M, N, K, ptr(devs[0]), ld, ptr(devs[1]), ld, ptr(out[shift:]), N + pad, stream()) == 0
    sync()
    got = out.cpu().numpy()
    D = got[shift:shift + M * (N + pad)].reshape(M, N + pad)
    a, b = host[0].tolist(), host[1].tolist()
    for m in range(M):
        for n in range(N):
            acc = 0.0
            for k in range(K):
                acc = fma(a[m][k], b[n][k], acc)
            assert D[m, n] == acc or (np.isnan(D[m, n]) and np.isnan(acc)), (m, n)
            if acc == 0.0:
                assert np.signbit(D[m, n]) == np.signbit(acc), (m, n)
    # nothing between the rows or past them is written
    assert (D[:, N:] == 3.25).all() and (got[:shift] == 3.25).all() and (got[shift + M * (N + pad):] == 3.25).all()
