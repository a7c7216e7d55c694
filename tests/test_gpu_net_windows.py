"""Net starts that do not ascend: each net is its own window [start, next start) of the pins, one that
ends before it starts is empty, and windows may share pins or reach past the last start. The
wirelength objective's value and (where one net alone holds a pin) gradient against the same formula in torch
double precision, pins of no window keeping what the gradient array held; and the HPWL, with and
without the forces beside it, whose array is the call's own."""
import ctypes as C

import numpy as np
import pytest

from tests.gpu_util import dev, ptr, stream

pytestmark = pytest.mark.gpu

CASES = {
    "one_step_back": [0, 4, 9, 6, 12, 15],
    "past_the_last": [0, 900, 10],
    "backwards": [40, 30, 20, 10, 0],
    "far_back": [0] + list(range(5, 640, 5)) + [3, 8, 2000, 700],
    "second_block": list(range(0, 3 * 128 + 1, 3)) + [100, 400, 350, 500],
}


@pytest.mark.parametrize("case", CASES)
def test_windows_in_any_order(case):
    import torch
    from gpl_b200 import engine, functions
    functions._lib()
    start = np.array(CASES[case], np.int64)
    n, pins = len(start) - 1, int(start.max())
    rng = np.random.default_rng(n)
    xy = torch.from_numpy(rng.uniform(-20000, 20000, (pins, 2))).cuda()
    w = torch.from_numpy(rng.uniform(0.5, 2.0, n).astype(np.float32)).cuda()
    cx, cy = 4e-4, 7e-4
    L, d, v = engine.lib(), dev(start), C.c_double()
    g = torch.full_like(xy, 5.0)
    assert L.gpl_fn_wa_forward(n, ptr(d), ptr(xy), ptr(w), cx, cy, C.byref(v), stream()) == 0
    assert L.gpl_fn_wa_backward(n, ptr(d), ptr(xy), ptr(w), cx, cy, 1.7, ptr(g), stream()) == 0
    x = xy.clone().requires_grad_(True)
    total = torch.zeros((), dtype=torch.float64, device="cuda")
    holds = np.zeros(pins, int)
    for k in range(n):
        if start[k + 1] <= start[k]:
            continue
        holds[start[k]:start[k + 1]] += 1
        p = x[start[k]:start[k + 1]]
        for a, c in enumerate((cx, cy)):
            q = p[:, a]
            ep, em = torch.exp(c * (q - q.max().detach())), torch.exp(c * (q.min().detach() - q))
            total = total + float(w[k]) * ((q * ep).sum() / ep.sum() - (q * em).sum() / em.sum())
    if total.requires_grad:
        total.backward()
    want = torch.zeros_like(xy) if x.grad is None else x.grad
    # sums of at most 2000 positive terms in double, as in the objectives' other edge tests
    assert abs(v.value - float(total.detach())) <= 1e-11 * max(1.0, float(xy.abs().max()) * n)
    one, none = torch.from_numpy(holds == 1).cuda(), torch.from_numpy(holds == 0).cuda()
    assert float((g - 1.7 * want)[one].abs().max() if bool(one.any()) else 0.0) <= 1e-11 * max(float(want.abs().max()), 1.0)
    assert bool((g[none] == 5.0).all())


@pytest.mark.parametrize("fused", [0, 1])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("case", list(CASES) + ["all_past_the_last"])
def test_hpwl_of_windows_in_any_order(case, shift, fused):
    import torch
    from gpl_b200 import engine
    start = np.array(CASES.get(case, [0, 3000, 5000, 5004, 2]), np.int64)
    n, pins = len(start) - 1, int(start.max())
    xy = np.random.default_rng(n).integers(-20000, 20000, (pins, 2)).astype(np.int32)
    buf = torch.zeros(2 * pins + 1, dtype=torch.int32, device="cuda")
    p = buf[shift:shift + 2 * pins]  # on an 8-byte boundary or off one
    p.copy_(dev(xy.reshape(-1)))
    d, h = dev(start), C.c_int64()
    assert engine.lib().gpl_kernel_hpwl(n, ptr(d), ptr(p), fused, C.byref(h), stream()) == 0
    want = 0
    for a, b in zip(start, start[1:]):
        if b > a:
            w = xy[a:b].astype(np.int64)
            want += int((w.max(0) - w.min(0)).sum())
    assert h.value == want
