"""The sliced solve with more items (long rows and slices) a block than warps, which its warps
then take as they come, against a thread per row: the products are the same bit for bit, so the
placed locations and the report are identical. Row counts a little past a block's sixteen
slices, with and without rows of over 64 entries, and past what one item a warp covers on every
SM."""
import numpy as np
import pytest

from gpl_b200 import engine, synth

pytestmark = pytest.mark.gpu

SMALL = dict(w_min=2, w_max=12, util=0.55, n_io=16, macros=0, macro_frac=0.0, seed=5)


@pytest.mark.parametrize("cells,max_degree", [(513, 150), (2049, 16), (9001, 120), (80_000, 64)])
def test_items_taken_match_rows(cells, max_degree, monkeypatch):
    d = synth.generate(dict(SMALL, cells=cells, nets=cells + cells // 20, max_degree=max_degree))
    args = ["-density", "0.80", "-bin_grid_count", "32", "-skip_nesterov_place", "-initial_place_max_iter", "3"]
    runs = []
    for form in ("0", "2"):
        monkeypatch.setenv("GPL_SPMV_FORM", form)
        runs.append(engine.global_placement(d, args))
    assert runs[0]["outcome"] == "initially_placed"
    assert np.array_equal(runs[0]["locations"], runs[1]["locations"])
    assert runs[0]["lines"] == runs[1]["lines"]
