"""One round of the initial placement on designs that reach every branch of the net model's
per-pin emission: fixed pins (macros, ports) as the lower and the higher of a pair, two-pin
nets, nets wider than a warp, a fanout limit that drops most nets, counts that are no multiple
of a block.

Tolerance: 1e-3 of the core's longer side per coordinate. The matrix entries are the oracle's
to f32 rounding (6e-8) and both solves stop at a 1e-6 residual, so with the condition of these
few hundred rows the solutions agree to far better; a pair lost or counted twice moves its
cells by whole fractions of the net's extent."""
import numpy as np
import pytest

import oracle
from gpl_b200 import engine, synth

pytestmark = pytest.mark.gpu

SMALL = dict(w_min=2, w_max=12, util=0.55, n_io=16, macros=0, macro_frac=0.0, max_degree=16, seed=11)
CASES = {
    "macros": (dict(SMALL, cells=700, nets=801, macros=3, macro_frac=0.15), []),
    "one_port": (dict(SMALL, cells=300, nets=390, n_io=1), []),
    "wide_nets": (dict(SMALL, cells=500, nets=600, max_degree=150), []),
    "fanout_limit": (dict(SMALL, cells=500, nets=901), ["-initial_place_max_fanout", "4"]),
    "no_pairs": (dict(SMALL, cells=129, nets=140), ["-initial_place_max_fanout", "2"]),
}


@pytest.mark.parametrize("case", CASES)
def test_one_round_matches_the_oracle(case):
    params, extra = CASES[case]
    d = synth.generate(params)
    args = ["-density", "0.80", "-bin_grid_count", "32", "-skip_nesterov_place", "-initial_place_max_iter", "1"] + extra
    ref = oracle.global_placement(d, args)
    got = engine.global_placement(d, args)
    assert got["outcome"] == ref["outcome"] == "initially_placed"
    a, b = got["locations"][:, 1:].astype(float), ref["locations"][:, 1:].astype(float)
    np.testing.assert_array_equal(got["locations"][:, 0], ref["locations"][:, 0])
    assert np.isfinite(a).all()
    assert np.max(np.abs(a - b)) <= 1e-3 * max(np.ptp(b[:, 0]), np.ptp(b[:, 1]), 20000.0)
