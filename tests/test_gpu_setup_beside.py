"""The placer's set-up, prepared beside the initial placement's rounds (or, with no round, after
it): its report lines word for word and in the oracle's order and place, on one region and on
several, with a density the design cannot hold (the adjusting warning) and without rounds."""
import pytest

import oracle
from gpl_b200 import engine, synth

pytestmark = pytest.mark.gpu

SET_UP = tuple(f"GPL-{c:04d}]" for c in (33, 302, 306, 23, 24, 25, 26, 27, 28, 29, 30, 34))
CASES = {
    "one_region": ("cfg1", ["-density", "0.70", "-bin_grid_count", "32"]),
    "adjusted": ("cfg1", ["-density", "0.05", "-bin_grid_count", "32"]),
    "no_round": ("cfg1", ["-density", "0.70", "-bin_grid_count", "32", "-skip_initial_place"]),
    "regions": ("cfg4s", ["-density", "0.70", "-bin_grid_count", "32"]),
}


@pytest.mark.parametrize("case", CASES)
def test_set_up_lines(case):
    preset, args = CASES[case]
    d = synth.generate(preset)
    a, b = engine.global_placement(d, args)["lines"], oracle.global_placement(d, args)["lines"]
    pick = lambda lines: [l for l in lines if any(c in l for c in SET_UP)]
    assert len(pick(b)) >= 9
    assert pick(a) == pick(b)
    # the place: after the last initial placement row, before the loop's table
    rows = [k for k, l in enumerate(a) if l.startswith("[InitialPlace]")]
    first = next(k for k, l in enumerate(a) if "GPL-0033]" in l)
    assert (not rows) == (case == "no_round") and all(k < first for k in rows)
