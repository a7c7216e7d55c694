"""The FP32 density solve of a grid with more points on a side than a launch has blocks on its
second axis (65535). The density is a sum of cosines of the long axis, so the field is known: each
cosine's sine over its wavenumber.

Tolerance: 4e-3 of the field's largest value. Two sums of 65600 terms by fused multiply-adds in
float, each rounding 2^-24 of a partial sum that stays below the result's scale: at most
65600 x 2^-24 = 3.9e-3 in all. The field past point 65535 comes from the
matrices' rows past it, so a row left out is off by the field itself there."""
import numpy as np
import pytest

from tests.gpu_util import dev, ptr, stream, sync

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("x_long", [True, False])
def test_a_side_past_65535_points(x_long):
    from gpl_b200 import engine
    n = 65600
    j = np.arange(n) + 0.5
    w = (np.pi * np.arange(n) / n).astype(np.float32)
    terms = ((1, 1.0), (4, 0.5))
    density = sum(a * np.cos(np.pi * k * j / n) for k, a in terms).astype(np.float32)
    want = sum(a / float(w[k]) * np.sin(np.pi * k * j / n) for k, a in terms)
    one = np.zeros(1, np.float32)
    d, gx, gy = dev(density), dev(np.zeros(n, np.float32)), dev(np.zeros(n, np.float32))
    nx, ny, wx, wy = (n, 1, w, one) if x_long else (1, n, one, w)
    assert engine.lib().gpl_kernel_poisson(nx, ny, wx.ctypes.data, wy.ctypes.data, ptr(d), ptr(gx), ptr(gy), 0, stream()) == 0
    sync()
    along, across = (gx, gy) if x_long else (gy, gx)
    got = along.cpu().numpy().astype(np.float64)
    assert np.max(np.abs(got - want)) <= 4e-3 * np.max(np.abs(want))
    assert not across.any()
