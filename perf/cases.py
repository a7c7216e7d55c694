"""The engine's measured cases: what a program that uses this framework has it do.

A user runs the `global_placement` command (through `Placer.global_placement`, the C ABI's
`gpl_global_placement`), calls one of its stages on device arrays (`gpl_kernel_*`), or puts its
objectives into an autograd graph (`gpl_b200.functions`). The listed cases cover all three at
the sizes of the synthetic designs (`gpl_b200/synth.py`), the tests and the benchmark, from the
294-cell block to 1.1M cells on 1024 x 1024 bins; `draw` gives others of the same ranges.

Device inputs are made with torch generators on the GPU, designs by the seeded generator.
"""
import ctypes as C
import math

import numpy as np
import torch

from gpl_b200 import engine, functions, synth

DEV = "cuda:0"
WINDOW = 0.15  # a net's pins lie within this share of the core's side around its anchor


def listed():
    return [
        # the small block (294 cells, 64 x 64 bins) through the whole command: launches and
        # read-backs decide; what an interactive or a per-block hierarchical flow runs many times
        {"name": "command_300", "kind": "command", "cells": 294, "bins": 64, "groups": 0, "macros": 0, "form": "mixed"},
        # an ordinary block: 100k cells with macros, 512 x 512 bins
        {"name": "command_100k", "kind": "command", "cells": 100_000, "bins": 512, "groups": 0, "macros": 8, "form": "mixed"},
        # region groups beside the top level: every region has a grid of its own, packed launches
        {"name": "command_groups_120k", "kind": "command", "cells": 120_000, "bins": 0, "groups": 48, "macros": 0, "form": "mixed"},
        # a large block on the benchmark's grid, the whole command
        {"name": "command_400k", "kind": "command", "cells": 400_000, "bins": 1024, "groups": 0, "macros": 32, "form": "mixed"},
        # the stages of one trial of the 1M-cell design (1.1M cells with its fillers), as a
        # program with its own loop calls them: the step with the bin scatter ...
        {"name": "step_1m", "kind": "step", "cells": 1_100_000, "nx": 1024, "ny": 1024},
        # ... the gradient update with the preconditioner and the step length's sums ...
        {"name": "gradients_1m", "kind": "gradients", "cells": 1_100_000, "nx": 1024, "ny": 1024},
        # ... the wirelength forces of a 100k-cell design's nets ...
        {"name": "wa_forces_105k", "kind": "wa", "nets": 105_000},
        # ... and the density's field on the benchmark's grid, split-BF16
        {"name": "poisson_1024", "kind": "poisson", "nx": 1024, "ny": 1024, "form": "mixed"},
        # one axis of an initial-placement round's solve, to the solver's iteration cap
        {"name": "bicgstab_300k", "kind": "bicgstab", "rows": 300_000},
        # the congestion map of a routability pass at 1M nets
        {"name": "rudy_1m", "kind": "rudy", "nets": 1_050_000, "tx": 1024, "ty": 1024},
        # the objectives in an autograd graph, value and gradient: a gradient step of a caller's loop
        {"name": "wirelength_250k", "kind": "wirelength", "nets": 250_000},
        {"name": "density_512", "kind": "density", "cells": 400_000, "nx": 512, "ny": 512},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["command", "command", "groups", "step", "gradients", "wa", "poisson", "bicgstab", "rudy", "wirelength", "density"])
    if kind == "command":
        n = _log(rng, 250, 200_000)
        # the placer's own bin rule (0), or a grid about the cells' number, odd sides too
        bins = rng.choice([0, max(16, int(math.sqrt(n) * rng.uniform(0.7, 1.6))), 1 << max(5, round(math.log2(math.sqrt(n) * 1.4)))])
        return {"kind": "command", "cells": n, "bins": min(bins, 512), "groups": 0, "macros": 8 if n >= 20_000 and rng.random() < 0.5 else 0, "form": rng.choice(["mixed", "mixed", "fp32"])}
    if kind == "groups":
        n = _log(rng, 30_000, 90_000)
        return {"kind": "command", "cells": n, "bins": 0, "groups": rng.randint(3, min(48, n // 2500)), "macros": 0, "form": rng.choice(["mixed", "fp32"])}
    if kind in ("step", "gradients"):
        n = _log(rng, 500, 1_100_000)
        side = min(1024, max(16, int(math.sqrt(n) * rng.uniform(0.6, 1.6))))
        return {"kind": kind, "cells": n, "nx": side, "ny": min(1024, max(16, int(side * rng.uniform(0.5, 1.5))))}
    if kind == "wa":
        return {"kind": "wa", "nets": _log(rng, 300, 105_000)}
    if kind == "poisson":
        if rng.random() < 0.6:
            return {"kind": "poisson", "nx": 128 * rng.randint(1, 8), "ny": 128 * rng.randint(1, 8), "form": rng.choice(["mixed", "mixed", "fp32"])}
        return {"kind": "poisson", "nx": _log(rng, 16, 700), "ny": _log(rng, 16, 700), "form": "fp32"}
    if kind == "bicgstab":
        return {"kind": "bicgstab", "rows": _log(rng, 250, 300_000)}
    if kind == "rudy":
        return {"kind": "rudy", "nets": _log(rng, 300, 1_050_000), "tx": _log(rng, 15, 1024), "ty": _log(rng, 15, 1024)}
    if kind == "wirelength":
        return {"kind": "wirelength", "nets": _log(rng, 300, 250_000)}
    return {"kind": "density", "cells": _log(rng, 300, 400_000), "nx": _log(rng, 32, 512), "ny": _log(rng, 32, 512)}


# ---------------------------------------------------------------- inputs
def _p(t):
    return C.c_void_p(t.data_ptr())


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _uniform(g, shape, lo, hi, dtype=torch.float64):
    return torch.rand(shape, generator=g, device=DEV, dtype=dtype) * (hi - lo) + lo


def _design(case, seed):
    n, seed = case["cells"], int(seed) % (1 << 31)
    if n == 294:
        return synth.generate("cfg1", seed=seed)
    nets = n + n // 20
    if case["groups"]:
        k = case["groups"]
        # log-uniform counts over a factor of 16, about two thirds of the cells in all
        return synth.generate("cfg4", seed=seed, cells=n, nets=nets, region_cells=(k, n // (8 * k), 2 * n // k))
    small = n < 5_000
    return synth.generate("cfg2", seed=seed, cells=n, nets=nets, macros=case["macros"], macro_frac={0: 0.0, 8: 0.12, 32: 0.15}[case["macros"]],
                          n_io=24 if small else 256, w_max=12 if small else 24, max_degree=16 if small else 64)


def _grid(nx, ny):
    """Bins of 1234.5 x 1530.25 DBU with rounded edges, from (1000, -500)."""
    sx, sy, lx, ly = 1234.5, 1530.25, 1000, -500
    bx = torch.floor(torch.arange(nx + 1, device=DEV, dtype=torch.float64) * sx + 0.5).to(torch.int32) + lx
    by = torch.floor(torch.arange(ny + 1, device=DEV, dtype=torch.float64) * sy + 0.5).to(torch.int32) + ly
    return dict(nx=nx, ny=ny, lx=lx, ly=ly, sx=sx, sy=sy, bx=bx, by=by, ux=lx + int(math.floor(nx * sx + 0.5)), uy=ly + int(math.floor(ny * sy + 0.5)))


def _cells(g, n, grid):
    """Cells as the loop holds them: most widened to about sqrt(2) bins, one in twenty thousand a
    macro of many bins, an eighth fillers; centres spread over the grid and in strips, as a sorted
    device order leaves them."""
    u = torch.rand(n, generator=g, device=DEV)
    kind = torch.where(u < 5e-5, 1, torch.where(u < 0.13, 2, 0)).to(torch.uint8)
    big = kind == 1

    def half(s, count):
        h = _uniform(g, n, 0.71 * s, 1.1 * s)
        m = _uniform(g, n, min(4, count / 8) * s, min(20, count / 4) * s)
        return torch.where(big, m, h).to(torch.int32)
    hx, hy = half(grid["sx"], grid["nx"]), half(grid["sy"], grid["ny"])
    scale = torch.where(big, 1.0, _uniform(g, n, 0.3, 1.0)).to(torch.float32)
    strips = max(1, grid["nx"] // 16)
    x = torch.rand(n, generator=g, device=DEV, dtype=torch.float64)
    y = torch.rand(n, generator=g, device=DEV, dtype=torch.float64)
    order = torch.argsort(torch.floor(x * strips) + y)
    x, y = x[order], y[order]
    xy = torch.stack([grid["lx"] + x * (grid["ux"] - grid["lx"]), grid["ly"] + y * (grid["uy"] - grid["ly"])], 1)
    return kind, hx, hy, scale, xy


def _degrees(g, n, top):
    """The designs' net degrees: 55 % of 2, 20 % of 3, 10 % of 4, the rest 5..16, one in a hundred
    up to `top`; the seed decides which net has which, not how many have each."""
    u = (torch.arange(n, device=DEV, dtype=torch.float64) + 0.5) / n
    rest = 5 + torch.arange(n, device=DEV) % 12
    large = 17 + (torch.arange(n, device=DEV) * 7) % (top - 16)
    deg = torch.where(u < 0.55, 2, torch.where(u < 0.75, 3, torch.where(u < 0.85, 4, torch.where(u < 0.99, rest, large))))
    deg = deg[torch.randperm(n, generator=g, device=DEV)]
    start = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    start[1:] = torch.cumsum(deg, 0)
    return deg, start


def _pins(g, deg, side, spread):
    """Pin positions within +-spread of each net's anchor, folded back into [0, side]."""
    n = deg.numel()
    total = int(deg.sum())
    anchor = _uniform(g, (n, 2), 0, side)
    net = torch.repeat_interleave(torch.arange(n, device=DEV), deg)
    xy = (anchor[net] + _uniform(g, (total, 2), -spread, spread)).abs()
    return net, torch.where(xy > side, 2 * side - xy, xy)


def _waves(n, size):
    """The solver's wavenumbers: pi k / n, scaled by the bin's share of the x bin."""
    return (math.pi * np.arange(n) / n * size).astype(np.float32)


def _system(g, n):
    """A bound-to-bound system of n cells: each net ties its pins to its two bound pins with
    weights 1 / ((degree - 1) distance), nets local to a window of the core, cells numbered at
    random; one cell in fifty also tied to a fixed pin."""
    deg, _ = _degrees(g, n + n // 20, 32 if n > 2000 else 17)
    side = int(math.ceil(math.sqrt(n)))
    net, xy = _pins(g, deg, side - 1e-3, WINDOW * side)
    number = torch.randperm(n, generator=g, device=DEV)
    cell = number[torch.clamp(xy[:, 1].long() * side + xy[:, 0].long(), max=n - 1)]
    first = torch.zeros_like(deg)
    first[1:] = torch.cumsum(deg, 0)[:-1]
    at = torch.arange(net.numel(), device=DEV) - first[net]
    rows, cols, vals = [], [], []
    diag = torch.zeros(n, dtype=torch.float64, device=DEV)
    rhs = torch.zeros(n, dtype=torch.float64, device=DEV)
    pitch = 2000.0
    for bound in (0, 1):
        use = at > bound  # pin k to bound pin 0, pins past 1 to bound pin 1 too
        a, b = cell[use], cell[(first[net] + bound)[use]]
        d = (xy[use][:, 0] - xy[(first[net] + bound)[use]][:, 0]).abs() * pitch
        w = 1.0 / ((deg[net][use] - 1) * d.clamp(min=200.0))
        off = _uniform(g, a.numel(), -500, 500) * w
        keep = a != b
        a, b, w, off = a[keep], b[keep], w[keep], off[keep]
        rows += [a, b]
        cols += [b, a]
        vals += [-w, -w]
        diag.index_add_(0, torch.cat([a, b]), torch.cat([w, w]))
        rhs.index_add_(0, torch.cat([a, b]), torch.cat([off, -off]))
    pos = torch.empty(n, dtype=torch.float64, device=DEV)
    grid_x = torch.arange(n, device=DEV) % side
    pos[number[torch.arange(n, device=DEV)]] = (grid_x.double() + 0.5) * pitch
    tied = torch.rand(n, generator=g, device=DEV) < 0.02
    tied[0] = True
    w = torch.where(tied, _uniform(g, n, 1e-4, 1e-3), 0.0)
    diag += w + 1e-7
    rhs += w * pos + 1e-7 * pitch * side / 2
    rows.append(torch.arange(n, device=DEV))
    cols.append(torch.arange(n, device=DEV))
    vals.append(diag)
    m = torch.sparse_coo_tensor(torch.stack([torch.cat(rows), torch.cat(cols)]), torch.cat(vals), (n, n)).coalesce()
    r, c = m.indices()
    start = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    start[1:] = torch.cumsum(torch.bincount(r, minlength=n), 0)
    x0 = torch.full((n,), pitch * side / 2, dtype=torch.float32, device=DEV)
    return dict(n=n, start=start, cols=c.to(torch.int32).contiguous(), vals=m.values().to(torch.float32).contiguous(), rhs=rhs.to(torch.float32), x0=x0)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "command":
        # a program keeps its engine context and the design's host arrays
        args = ["-density", "0.70"] + (["-bin_grid_count", str(case["bins"])] if case["bins"] else [])
        return dict(kind=kind, placer=engine.Placer(0, case["form"]), design=_design(case, seed), args=args)
    L, g = engine.lib(), _gen(seed)
    s = dict(kind=kind, L=L)
    if kind in ("step", "gradients"):
        n, grid = case["cells"], _grid(case["nx"], case["ny"])
        cell_kind, hx, hy, scale, xy = _cells(g, n, grid)
        s.update(n=n, grid=grid, cell_kind=cell_kind, hx=hx, hy=hy, scale=scale)
        if kind == "step":
            slp = xy.to(torch.float32)
            s.update(slp=slp, cur=(slp + _uniform(g, (n, 2), -2000, 2000)).to(torch.float32),
                     grad=(torch.randn((n, 2), generator=g, device=DEV) * 3.0).to(torch.float32),
                     next=torch.empty((n, 2), dtype=torch.float32, device=DEV), next_slp=torch.empty((n, 2), dtype=torch.float32, device=DEV),
                     centre=torch.empty((n, 2), dtype=torch.int32, device=DEV),
                     inst=torch.empty((grid["nx"], grid["ny"]), dtype=torch.int64, device=DEV), fill=torch.empty((grid["nx"], grid["ny"]), dtype=torch.int64, device=DEV))
        else:
            pins = torch.where(cell_kind == 2, 0, torch.randint(1, 8, (n,), generator=g, device=DEV))
            start = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
            start[1:] = torch.cumsum(pins, 0)
            normal = lambda shape, sd: (torch.randn(shape, generator=g, device=DEV) * sd).to(torch.float32)
            s.update(centre=xy.to(torch.int32), start=start, force=normal((int(start[-1]), 2), 0.5), area=(4.0 * hx.double() * hy.double() * 0.5).to(torch.float32),
                     fx=normal((grid["nx"], grid["ny"]), 1e-3), fy=normal((grid["nx"], grid["ny"]), 1e-3), a1=normal((n, 2), 500.0), b1=normal((n, 2), 500.0),
                     b2=normal((n, 2), 1e-2), sum=torch.empty((n, 2), dtype=torch.float32, device=DEV), penalty=3.7e-5)
    elif kind == "wa":
        deg, start = _degrees(g, case["nets"], 64)
        # from a few hundred DBU (a placed local net) to the whole window
        _, xy = _pins(g, deg, 1.0, 0.0)
        side = 2000.0 * math.sqrt(case["nets"])
        reach = torch.exp(_uniform(g, deg.numel(), math.log(300.0), math.log(max(400.0, WINDOW * side))))
        net = torch.repeat_interleave(torch.arange(deg.numel(), device=DEV), deg)
        xy = xy * side + (torch.rand((xy.shape[0], 2), generator=g, device=DEV, dtype=torch.float64) * 2 - 1) * reach[net, None]
        s.update(n=deg.numel(), start=start, xy=xy.to(torch.int32).contiguous(), weight=_uniform(g, deg.numel(), 1.0, 1.5).to(torch.float32),
                 coef=(2.1e-4, 2.6e-4), force=torch.empty((xy.shape[0], 2), dtype=torch.float32, device=DEV), net=net)
    elif kind == "poisson":
        nx, ny = case["nx"], case["ny"]
        # a placement's density: smooth hills on a noisy floor
        x = torch.linspace(0, 1, nx, device=DEV)[:, None]
        y = torch.linspace(0, 1, ny, device=DEV)[None, :]
        c = torch.rand((6, 3), generator=g, device=DEV)
        dens = 0.6 * torch.rand((nx, ny), generator=g, device=DEV)
        for k in range(6):
            dens = dens + torch.exp(-((x - c[k, 0]) ** 2 + (y - c[k, 1]) ** 2) / (0.002 + 0.05 * c[k, 2]))
        s.update(nx=nx, ny=ny, wx=_waves(nx, 1.0), wy=_waves(ny, 1400.0 / 900.0), dens=dens.contiguous(), mode={"fp32": 0, "mixed": 1}[case["form"]],
                 fx=torch.empty((nx, ny), device=DEV), fy=torch.empty((nx, ny), device=DEV))
    elif kind == "bicgstab":
        s.update(_system(g, case["rows"]))
    elif kind == "rudy":
        tile = 700
        die = (0, 0, case["tx"] * tile + 321, case["ty"] * tile + 77)
        n = case["nets"]
        w = torch.tensor([die[2], die[3]], device=DEV, dtype=torch.float64)
        # a placed design's boxes: from a third of a tile to the locality window
        low = 0.3 * tile / w
        size = torch.exp(torch.log(low) + torch.rand((n, 2), generator=g, device=DEV, dtype=torch.float64) * torch.log(2 * WINDOW / low).clamp(min=0)) * w
        lo = torch.rand((n, 2), generator=g, device=DEV, dtype=torch.float64) * (w - size)
        s.update(n=n, die=die, tile=tile, tx=case["tx"], ty=case["ty"], wire=120, boxes=torch.cat([lo, lo + size], 1).to(torch.int32).contiguous(),
                 demand=torch.empty((case["tx"], case["ty"]), dtype=torch.float32, device=DEV))
    elif kind == "wirelength":
        deg, start = _degrees(g, case["nets"], 64)
        side = 2000.0 * math.sqrt(case["nets"])
        net, xy = _pins(g, deg, side, 3000.0)
        s.update(start=start, net=net, xy=xy.contiguous().requires_grad_(True), weight=_uniform(g, deg.numel(), 1.0, 1.5).to(torch.float32), coef=(7.5e-4, 9e-4))
    elif kind == "density":
        nx, ny, n = case["nx"], case["ny"], case["cells"]
        bw, bh = 1000.0, 1250.0
        size = torch.tensor([nx * bw, ny * bh], device=DEV, dtype=torch.float64)
        s.update(nx=nx, ny=ny, bw=bw, bh=bh, xy=(torch.rand((n, 2), generator=g, device=DEV, dtype=torch.float64) * size).requires_grad_(True),
                 half=_uniform(g, (n, 2), 300, 1400), scale=_uniform(g, n, 0.5, 1.0), energy=functions.DensityEnergy(nx, ny, 0.0, 0.0, bw, bh))
    else:
        raise ValueError(kind)
    return s


# ---------------------------------------------------------------- one pass
def _ok(rc, what):
    if rc != 0:
        raise RuntimeError(f"{what}: error {rc}")


def run(s):
    kind = s["kind"]
    if kind == "command":
        r = s["placer"].global_placement(s["design"], s["args"])
        if r["status"] != "placed":
            raise RuntimeError(f"global_placement: {r['status']} {r['code']} {r['reason']}")
        return {"locations": r["locations"], "final_hpwl": r["final_hpwl"], "final_overflow": float(r["final_overflow"]), "iterations": r["nesterov_iterations"]}
    L = s["L"]
    if kind == "step":
        d = s["grid"]
        _ok(L.gpl_kernel_nesterov_step(s["n"], _p(s["slp"]), _p(s["grad"]), _p(s["cur"]), _p(s["hx"]), _p(s["hy"]), _p(s["scale"]), _p(s["cell_kind"]), None,
                                       d["nx"], d["ny"], d["lx"], d["ly"], _p(d["bx"]), _p(d["by"]), d["sx"], d["sy"], 0.7, 731.25, 0.8713,
                                       _p(s["next"]), _p(s["next_slp"]), _p(s["centre"]), _p(s["inst"]), _p(s["fill"]), _stream()), "step")
        return {"next": s["next"], "next_slp": s["next_slp"], "centre": s["centre"], "inst": s["inst"], "fill": s["fill"]}
    if kind == "gradients":
        d = s["grid"]
        sums = np.zeros(4)
        _ok(L.gpl_kernel_gradients(s["n"], _p(s["centre"]), _p(s["hx"]), _p(s["hy"]), _p(s["scale"]), _p(s["area"]), _p(s["start"]), _p(s["force"]),
                                   d["nx"], d["ny"], d["lx"], d["ly"], _p(d["bx"]), _p(d["by"]), d["sx"], d["sy"], _p(s["fx"]), _p(s["fy"]), s["penalty"],
                                   _p(s["sum"]), _p(s["a1"]), _p(s["b1"]), _p(s["b2"]), sums.ctypes.data_as(C.c_void_p), _stream()), "gradients")
        return {"sum": s["sum"], "sums": sums}
    if kind == "wa":
        _ok(L.gpl_kernel_wa(s["n"], _p(s["start"]), _p(s["xy"]), _p(s["weight"]), s["coef"][0], s["coef"][1], _p(s["force"]), _stream()), "wa")
        return s["force"]
    if kind == "poisson":
        _ok(L.gpl_kernel_poisson(s["nx"], s["ny"], s["wx"].ctypes.data_as(C.c_void_p), s["wy"].ctypes.data_as(C.c_void_p), _p(s["dens"]), _p(s["fx"]), _p(s["fy"]), s["mode"], _stream()), "poisson")
        return {"fx": s["fx"], "fy": s["fy"]}
    if kind == "bicgstab":
        x = s["x0"].clone()
        it, err = C.c_int32(), C.c_float()
        _ok(L.gpl_kernel_bicgstab(s["n"], _p(s["start"]), _p(s["cols"]), _p(s["vals"]), _p(s["rhs"]), _p(x), 100, C.byref(it), C.byref(err), _stream()), "bicgstab")
        return {"x": x, "iterations": it.value}
    if kind == "rudy":
        _ok(L.gpl_kernel_rudy(s["n"], _p(s["boxes"]), *s["die"], s["tx"], s["ty"], s["tile"], s["wire"], _p(s["demand"]), _stream()), "rudy")
        return s["demand"]
    if kind == "wirelength":
        s["xy"].grad = None
        w = functions.wirelength(s["xy"], s["start"], s["weight"], *s["coef"])
        w.backward()
        return {"value": w.detach(), "grad": s["xy"].grad}
    s["xy"].grad = None
    e = s["energy"](s["xy"], s["half"], s["scale"])
    e.backward()
    return {"value": e.detach(), "grad": s["xy"].grad}


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind == "command":
        # the design's arrays in (an instance's box, flags, group, pins, orientation and master: 41
        # bytes; a terminal's instance, shape, flag and order: 25), the written placement out
        n = case["cells"]
        pins = 4.0 * 1.05 * n
        return {"bytes": n * (41.0 + 12.0) + pins * 25.0 + 1.05 * n * 17.0, "flops": 0.0}
    if kind == "step":
        n, b = case["cells"], case["nx"] * case["ny"]
        return {"bytes": n * (24.0 + 13.0 + 24.0) + 16.0 * b, "flops": 60.0 * n}
    if kind == "gradients":
        n, b = case["cells"], case["nx"] * case["ny"]
        return {"bytes": n * (8.0 + 8.0 + 8.0 + 8.0 + 3.5 * 8.0 + 8.0 + 24.0) + 8.0 * b, "flops": 80.0 * n}
    if kind == "wa":
        pins = 4.0 * case["nets"]
        return {"bytes": 12.0 * case["nets"] + 16.0 * pins, "flops": 140.0 * pins}
    if kind == "poisson":
        nx, ny = case["nx"], case["ny"]
        return {"bytes": 12.0 * nx * ny, "flops": 2.5 * 3 * 2 * nx * ny * math.log2(nx * ny)}
    if kind == "bicgstab":
        # the matrix (about 13 entries a row) and the vectors once
        n = case["rows"]
        return {"bytes": n * (13.0 * 8.0 + 8.0 + 4.0 * 3), "flops": 100.0 * n * (2 * 2 * 13.0 + 20.0)}
    if kind == "rudy":
        return {"bytes": 16.0 * case["nets"] + 4.0 * case["tx"] * case["ty"], "flops": 30.0 * case["nets"]}
    if kind == "wirelength":
        pins = 4.0 * case["nets"]
        return {"bytes": 12.0 * case["nets"] + 32.0 * pins, "flops": 200.0 * pins}
    n, nx, ny = case["cells"], case["nx"], case["ny"]
    return {"bytes": 56.0 * n, "flops": 80.0 * n + 2 * 2 * 2.5 * nx * ny * math.log2(nx * ny)}


# ---------------------------------------------------------------- the same in 64 bits
def _box_sums(table, edges_x, edges_y, x0, x1, y0, y1):
    """Integrals of a piecewise-constant field over boxes, from its cumulated corner table."""
    def at(px, py):
        i = torch.clamp(torch.searchsorted(edges_x, px, right=True) - 1, 0, edges_x.numel() - 2)
        j = torch.clamp(torch.searchsorted(edges_y, py, right=True) - 1, 0, edges_y.numel() - 2)
        a = (px - edges_x[i]) / (edges_x[i + 1] - edges_x[i])
        b = (py - edges_y[j]) / (edges_y[j + 1] - edges_y[j])
        return (1 - a) * ((1 - b) * table[i, j] + b * table[i, j + 1]) + a * ((1 - b) * table[i + 1, j] + b * table[i + 1, j + 1])
    cx = lambda v: torch.minimum(torch.maximum(v, edges_x[0]), edges_x[-1]).contiguous()
    cy = lambda v: torch.minimum(torch.maximum(v, edges_y[0]), edges_y[-1]).contiguous()
    x0, x1, y0, y1 = cx(x0), cx(x1), cy(y0), cy(y1)
    return at(x1, y1) - at(x0, y1) - at(x1, y0) + at(x0, y0)


def _net_max(v, net, n, c):
    """Per net, the smooth maximum's shifted exponentials and their sums, per axis (c signed)."""
    top = torch.full((n, 2), -math.inf, dtype=torch.float64, device=DEV).scatter_reduce_(0, net[:, None].expand(-1, 2), v * c, "amax")
    e = torch.exp(v * c - top[net])
    s = torch.zeros((n, 2), dtype=torch.float64, device=DEV).index_add_(0, net, e)
    a = torch.zeros((n, 2), dtype=torch.float64, device=DEV).index_add_(0, net, v * e)
    return e, s, a


def _bases(n):
    k = torch.arange(n, device=DEV, dtype=torch.float64)
    t = math.pi * k[:, None] * (k[None, :] + 0.5) / n
    return torch.cos(t), torch.sin(t)  # [k][x]


def exact(case, seed):
    kind = case["kind"]
    if kind == "command":
        return None  # a whole run's course follows every rounding
    s = prepare(case, seed)
    if kind == "step":
        d = s["grid"]
        slp, grad, cur = s["slp"].double(), s["grad"].double(), s["cur"].double()
        half = torch.stack([s["hx"], s["hy"]], 1).double()
        lo = torch.tensor([d["lx"], d["ly"]], device=DEV, dtype=torch.float64) + half
        hi = torch.tensor([d["ux"], d["uy"]], device=DEV, dtype=torch.float64) - half
        nxt = slp + 731.25 * grad
        nslp = nxt + float(np.float32(0.8713)) * (nxt - cur)
        clamp = lambda v: torch.minimum(torch.maximum(v, lo), hi)
        return {"next": clamp(nxt), "next_slp": clamp(nslp), "centre": None, "inst": None, "fill": None}
    if kind == "gradients":
        d = s["grid"]
        n, start = s["n"], s["start"]
        wl = torch.zeros((n, 2), dtype=torch.float64, device=DEV)
        wl.index_add_(0, torch.repeat_interleave(torch.arange(n, device=DEV), start[1:] - start[:-1]), s["force"].double())
        ex, ey = d["bx"].double(), d["by"].double()
        area = (ex[1:] - ex[:-1])[:, None] * (ey[1:] - ey[:-1])[None, :]
        c, hx, hy = s["centre"].double(), s["hx"].double(), s["hy"].double()
        den = []
        for f in (s["fx"], s["fy"]):
            table = torch.zeros((d["nx"] + 1, d["ny"] + 1), dtype=torch.float64, device=DEV)
            table[1:, 1:] = torch.cumsum(torch.cumsum(f.double() * area, 0), 1)
            den.append(_box_sums(table, ex, ey, c[:, 0] - hx, c[:, 0] + hx, c[:, 1] - hy, c[:, 1] + hy) * s["scale"].double())
        den = torch.stack(den, 1)
        penalty = float(np.float32(s["penalty"]))
        pre = torch.clamp((start[1:] - start[:-1]).double() + penalty * s["area"].double(), min=1.0)
        out = (wl + penalty * den) / pre[:, None]
        sq = lambda a, b: float(((a.double() - b.double()) ** 2).sum())
        return {"sum": out, "sums": np.array([float(wl.abs().sum()), float(den.abs().sum()), sq(s["a1"], s["b1"]), sq(out, s["b2"])])}
    if kind == "wa":
        xy, net, n = s["xy"].double(), s["net"], s["n"]
        c = torch.tensor([float(np.float32(v)) for v in s["coef"]], dtype=torch.float64, device=DEV)
        e, t, a = _net_max(xy, net, n, c)
        gmax = e * ((1 + c * xy) * t[net] - c * a[net]) / t[net] ** 2
        e, t, a = _net_max(xy, net, n, -c)
        gmin = e * ((1 - c * xy) * t[net] + c * a[net]) / t[net] ** 2
        return (gmin - gmax) * s["weight"].double()[net, None]
    if kind == "poisson":
        nx, ny, rho = s["nx"], s["ny"], s["dens"].double()
        (cx, sx), (cy, sy) = _bases(nx), _bases(ny)
        wx, wy = (torch.from_numpy(v.astype(np.float64)).to(DEV) for v in (s["wx"], s["wy"]))
        a = cx @ rho @ cy.T * (4.0 / (nx * ny))
        a[0] *= 0.5
        a[:, 0] *= 0.5
        q = wx[:, None] ** 2 + wy[None, :] ** 2
        q[0, 0] = 1.0
        p = a / q
        p[0, 0] = 0.0
        return {"fx": sx.T @ (p * wx[:, None]) @ cy, "fy": cx.T @ (p * wy[None, :]) @ sy}
    if kind == "bicgstab":
        return None  # stopped at the cap, on its way: the iterate follows every rounding
    if kind == "rudy":
        b = s["boxes"].double()
        t, (lx, ly, ux, uy) = s["tile"], s["die"]
        hpwl, area = (b[:, 2] - b[:, 0]) + (b[:, 3] - b[:, 1]), (b[:, 2] - b[:, 0]) * (b[:, 3] - b[:, 1])
        # a box that begins past the last whole column or row (in the stretch) is on no tile
        ok = (area > 0) & (b[:, 0] < s["tx"] * t) & (b[:, 1] < s["ty"] * t)
        c = torch.where(ok, 100.0 * hpwl * s["wire"] / area.clamp(min=1.0), 0.0)
        edges = lambda n, end: torch.cat([torch.arange(n, device=DEV, dtype=torch.float64) * t, torch.tensor([float(end)], device=DEV, dtype=torch.float64)])
        gx, gy = edges(s["tx"], ux), edges(s["ty"], uy)
        # a net's cover of the columns rises at its lower edge and falls at its upper one: two
        # deposits an edge and axis, whose cumulated sums along both axes are the map
        diff = torch.zeros(((s["tx"] + 1) * (s["ty"] + 1),), dtype=torch.float64, device=DEV)

        def deposits(lo, hi, g):
            out = []
            for v, sign in ((lo, 1.0), (hi, -1.0)):
                i = torch.clamp(torch.searchsorted(g, v.contiguous(), right=True) - 1, 0, g.numel() - 2)
                share = (g[i + 1] - v) / (g[i + 1] - g[i])
                out += [(i, sign * share), (i + 1, sign * (1 - share))]
            return out
        for i, fi in deposits(b[:, 0], b[:, 2], gx):
            for j, fj in deposits(b[:, 1], b[:, 3], gy):
                diff.index_add_(0, i * (s["ty"] + 1) + j, c * fi * fj)
        full = torch.cumsum(torch.cumsum(diff.view(s["tx"] + 1, s["ty"] + 1), 0), 1)
        return full[:-1, :-1].contiguous()
    if kind == "wirelength":
        xy, net, n = s["xy"].detach(), s["net"], s["weight"].numel()
        w = s["weight"].double()
        c = torch.tensor(s["coef"], dtype=torch.float64, device=DEV)
        e, t, a = _net_max(xy, net, n, c)
        grad = e * ((1 + c * xy) * t[net] - c * a[net]) / t[net] ** 2
        value = a / t
        e, t, a = _net_max(xy, net, n, -c)
        grad = grad - e * ((1 - c * xy) * t[net] + c * a[net]) / t[net] ** 2
        value = value - a / t
        return {"value": (value.sum(1) * w).sum(), "grad": grad * w[net, None]}
    nx, ny, bw, bh = s["nx"], s["ny"], s["bw"], s["bh"]
    xy = s["xy"].detach()
    lo, hi = xy - s["half"], xy + s["half"]
    rho = torch.zeros(nx * ny, dtype=torch.float64, device=DEV)
    first = torch.floor(lo / torch.tensor([bw, bh], device=DEV, dtype=torch.float64)).long()
    span = 4  # a cell's half size is below 1.4 bins

    def over(k, axis, size, count):
        b = first[:, axis] + k
        o = (torch.minimum(hi[:, axis], (b + 1) * size) - torch.maximum(lo[:, axis], b * size)).clamp(min=0)
        return b.clamp(0, count - 1), torch.where((b >= 0) & (b < count), o, 0.0)
    for i in range(span):
        bx, ox = over(i, 0, bw, nx)
        for j in range(span):
            by, oy = over(j, 1, bh, ny)
            rho.index_add_(0, bx * ny + by, s["scale"] * ox * oy)
    rho = rho.view(nx, ny)
    (cx, _), (cy, _) = _bases(nx), _bases(ny)
    u = math.pi * torch.arange(nx, device=DEV, dtype=torch.float64) / nx
    v = math.pi * torch.arange(ny, device=DEV, dtype=torch.float64) / ny * (bh / bw)
    a = cx @ rho @ cy.T * (4.0 / (nx * ny))
    a[0] *= 0.5
    a[:, 0] *= 0.5
    q = u[:, None] ** 2 + v[None, :] ** 2
    q[0, 0] = 1.0
    a = a / q
    a[0, 0] = 0.0
    phi = cx.T @ a @ cy
    value = 0.5 * (rho * phi).sum()
    flat = phi.reshape(-1)
    grad = torch.zeros_like(xy)
    for axis, (size, count, osize, ocount) in enumerate(((bw, nx, bh, ny), (bh, ny, bw, nx))):
        for edge, sign in ((hi, 1.0), (lo, -1.0)):
            f = edge[:, axis] / size
            inside = (f > 0) & (f < count)
            b = torch.floor(f).long().clamp(0, count - 1)
            for j in range(span):
                ob, oo = over(j, 1 - axis, osize, ocount)
                k = ob * ny + b if axis else b * ny + ob
                grad[:, axis] += sign * torch.where(inside, oo, 0.0) * flat[k]
    return {"value": value, "grad": grad * s["scale"][:, None]}
