"""The initial placement's assembled matrices, bit for bit: every row's columns and values and the
right-hand side of both axes against `updatePinInfo` and `createSparseMatrix`
(src/initial_place.rs:203-355) restated here in float32, each row's duplicates summed in the order
the triplets are appended (src/bicgstab.rs:501-541). Nets of one and two pins, wider than a warp
and over the fanout limit; pins that tie for an extreme, several pins of an instance in a net, ports, fixed and locked
instances, movable IO pins, and an instance in nearly every net (rows of thousands of triplets)."""
import ctypes as C

import numpy as np
import pytest

from tests.gpu_util import stream

pytestmark = pytest.mark.gpu

F = np.float32


def restated(box, locked, pin_e, pin_inst, mio, xy, start, max_fanout, min_diff, scale):
    """Per axis: {row: {column: sum}} and the right-hand side of the rows that move."""
    n = len(box)
    rows = [[dict() for _ in range(n)] for _ in range(2)]
    rhs = [[F(0)] * n for _ in range(2)]

    def add(a, r, c, v):
        d = rows[a][r]
        d[c] = F(d[c] + v) if c in d else v

    for e in np.flatnonzero(locked):
        for a in range(2):
            add(a, int(e), int(e), F(1))
    for k in range(len(start) - 1):
        pins = range(int(start[k]), int(start[k + 1]))
        if len(pins) <= 1 or len(pins) >= max_fanout:
            continue
        solve = [p for p in pins if not mio[p]]
        ext = []
        for a in range(2):
            c = [int(xy[p][a]) for p in solve]
            ext.append({solve[c.index(min(c))], solve[c.index(max(c))]} if solve else set())
        net_weight = F(F(scale) / F(len(pins) - 1))
        for i1 in range(1, len(solve)):
            for i2 in range(i1):
                p1, p2 = solve[i1], solve[i2]
                if pin_inst[p1] == pin_inst[p2]:
                    continue
                for a in range(2):
                    if p1 not in ext[a] and p2 not in ext[a]:
                        continue
                    c1, c2 = int(xy[p1][a]), int(xy[p2][a])
                    w = F(net_weight / F(max(abs(c1 - c2), min_diff)))
                    ea, eb = int(pin_e[p1]), int(pin_e[p2])
                    mid = lambda e: (int(box[e][a]) + int(box[e][a + 2])) // 2
                    fa, fb = ea >= 0 and not locked[ea], eb >= 0 and not locked[eb]
                    if fa and fb:
                        add(a, ea, ea, w), add(a, eb, eb, w), add(a, ea, eb, F(-w)), add(a, eb, ea, F(-w))
                        rhs[a][ea] = F(rhs[a][ea] + F(F(-w) * F((c1 - mid(ea)) - (c2 - mid(eb)))))
                        rhs[a][eb] = F(rhs[a][eb] + F(F(-w) * F((c2 - mid(eb)) - (c1 - mid(ea)))))
                    elif eb >= 0 and (ea < 0 or (locked[ea] and fb)):
                        add(a, eb, eb, w)
                        rhs[a][eb] = F(rhs[a][eb] + F(w * F(c1 - (c2 - mid(eb)))))
                    elif ea >= 0 and (eb < 0 or (locked[eb] and fa)):
                        add(a, ea, ea, w)
                        rhs[a][ea] = F(rhs[a][ea] + F(w * F(c2 - (c1 - mid(ea)))))
    return rows, rhs


@pytest.mark.parametrize("n,nets,wide,hub,max_fanout", [(40, 150, 60, 0.3, 200), (300, 500, 40, 0.9, 30), (1, 5, 4, 1.0, 200), (700, 1000, 150, 0.0, 200)])
def test_assembled_rows_bit_for_bit(n, nets, wide, hub, max_fanout):
    from gpl_b200 import engine
    L = engine.lib()
    L.gpl_rules_b2b.argtypes = [C.c_int64, C.c_void_p, C.c_void_p, C.c_int64] + [C.c_void_p] * 4 + [C.c_int32, C.c_void_p, C.c_int32, C.c_int32, C.c_float, C.c_int64] + [C.c_void_p] * 5
    rng = np.random.default_rng(n)
    lo = rng.integers(0, 40, (n, 2)) * 500
    box = np.concatenate([lo, lo + rng.integers(100, 900, (n, 2))], 1).astype(np.int32)
    locked = (rng.random(n) < 0.1).astype(np.uint8)
    degree = np.where(rng.random(nets) < 0.05, rng.integers(wide // 2, wide + 1, nets), rng.integers(1, 8, nets))
    start = np.concatenate([[0], np.cumsum(degree)]).astype(np.int64)
    m = int(start[-1])
    inst = rng.integers(0, n, m)
    inst[start[:-1][rng.random(nets) < hub]] = n - 1
    kind = rng.choice(4, m, p=[0.85, 0.05, 0.05, 0.05])  # of a placed instance, fixed, port, movable IO
    pin_e = np.where(kind == 0, inst, -1).astype(np.int32)
    pin_inst = np.where(kind == 0, inst, np.where(kind == 1, n + inst, -1)).astype(np.int32)
    mio = (kind == 3).astype(np.uint8)
    # on a coarse grid: ties for the extremes, and distances on both sides of the least
    xy = np.ascontiguousarray((box[inst, :2] + rng.integers(0, 4, (m, 2)) * 250).astype(np.int32))
    cap = 4 * m * 200
    rs, cols, vals, rhs = np.zeros((2, n + 1), np.int64), np.zeros((2, cap), np.int32), np.zeros((2, cap), np.float32), np.zeros((2, n), np.float32)
    vp = lambda a: a.ctypes.data_as(C.c_void_p)
    assert L.gpl_rules_b2b(n, vp(box), vp(locked), m, vp(pin_e), vp(pin_inst), vp(mio), vp(xy), nets, vp(start), max_fanout, 1500, 800.0, cap, vp(rs), vp(cols), vp(vals), vp(rhs), stream()) == 0
    want, want_rhs = restated(box, locked, pin_e, pin_inst, mio, xy, start, max_fanout, 1500, 800.0)
    for a in range(2):
        for e in range(n):
            c = sorted(want[a][e])
            b, t = rs[a][e], rs[a][e + 1]
            assert cols[a][b:t].tolist() == c
            assert vals[a][b:t].tobytes() == np.array([want[a][e][k] for k in c], np.float32).tobytes()
        free = locked == 0
        np.testing.assert_array_equal(rhs[a][free], np.array(want_rhs[a], np.float32)[free])
