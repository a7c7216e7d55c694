"""Contexts are independent: whole commands on two contexts from two threads at once, beside a
third thread's solves through the solver's entry point, each equal to its run alone, bit for bit
(the results do not depend on the order in which the device runs the launches). The designs are
large enough that each solver loop takes many blocks, which wait for one another."""
import ctypes as C
import threading

import numpy as np
import pytest

from gpl_b200 import engine, synth
from tests.gpu_util import dev, ptr

pytestmark = pytest.mark.gpu

SMALL = dict(w_min=2, w_max=12, util=0.55, n_io=16, macros=2, macro_frac=0.1, max_degree=40)
ARGS = ["-density", "0.80", "-bin_grid_count", "64"]


def solver():
    import torch
    n = 150_001
    w = np.arange(-5, 6)
    cols = np.arange(n)[:, None] + w
    ok = (cols >= 0) & (cols < n)
    vals = np.broadcast_to(np.where(w == 0, 12.0, -1.0), cols.shape)
    starts = np.concatenate([[0], np.cumsum(ok.sum(1))])
    d = [dev(a) for a in (starts.astype(np.int64), cols[ok].astype(np.int32), vals[ok].astype(np.float32), np.linspace(-1, 1, n).astype(np.float32))]
    s = torch.cuda.Stream()
    torch.cuda.synchronize()

    def run():
        with torch.cuda.stream(s):
            x, it, err = torch.zeros(n, device="cuda"), C.c_int32(), C.c_float()
            rc = engine.lib().gpl_kernel_bicgstab(n, *[ptr(t) for t in d], ptr(x), 100, C.byref(it), C.byref(err), C.c_void_p(s.cuda_stream))
            return rc, it.value, x.cpu().numpy()
    return run


def test_commands_at_once_equal_the_commands_alone():
    designs = [synth.generate(dict(SMALL, cells=n, nets=n + n // 20, seed=n)) for n in (20_000, 45_000)]
    alone = [engine.global_placement(d, ARGS) for d in designs]
    run = solver()
    solved = run()
    assert solved[0] == 0 and all(a["status"] == "placed" for a in alone)
    got, sols, raised = [[], []], [], []

    def command(k):
        try:
            p = engine.Placer(0)
            for _ in range(3):
                got[k].append(p.global_placement(designs[k], ARGS))
            p.close()
        except Exception as e:  # a thread's failure is the test's
            raised.append(e)

    def solves():
        try:
            for _ in range(40):
                sols.append(run())
        except Exception as e:
            raised.append(e)

    threads = [threading.Thread(target=command, args=(k,)) for k in range(2)] + [threading.Thread(target=solves)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not raised
    for k in range(2):
        assert len(got[k]) == 3
        for r in got[k]:
            assert r["status"] == "placed" and r["lines"] == alone[k]["lines"]
            np.testing.assert_array_equal(r["locations"], alone[k]["locations"])
    assert len(sols) == 40 and all(r[0] == 0 and r[1] == solved[1] and np.array_equal(r[2], solved[2]) for r in sols)
