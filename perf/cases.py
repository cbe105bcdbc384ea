"""The workloads this package's speed is measured on.

A case is a dict of plain values.  ``prepare`` builds what a host program
holds before the call (a loaded context, pinned transfer buffers, state
blocks), ``run`` makes one pass through the public Python entry points,
``work`` states the bytes and operations a pass cannot do without and
``exact`` evaluates the same pass in 64-bit torch, written from the
formulas of the reference and without this package's kernels.

Kinds of pass:

* ``step``     what the GPU does between two Stokes solves of the host: the
               solution goes up (pinned), the node routines that follow the
               solve, nodes2markers + move, the next marker2nodes, the node
               routines that precede the next solve, and the solve's inputs
               come back (asynchronously under the node kernels, then the
               three that depend on them).
* ``cycle``    eight seismic-cycle steps (graph replays), each followed by
               calc_timestep, then the accumulated slips and the node fields.
* ``newton``   the per-marker VEP + RSF Newton on a block of states.
* ``sort``     the allocation-free cell sort on device positions.
* ``stokes``   the Stokes matrix into host CSR arrays.
* ``restart``  the marker part of the temperature solve, then every marker
               array to the host (what saving a restart file needs).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from velo2cycles_gb300 import abi, cellsort, mic, newton, synth

F64 = torch.float64


def _pick(cond, a: float, b: float):
    """a where cond, else b, in 64 bits"""
    return torch.where(cond, torch.tensor(a, dtype=F64, device=cond.device),
                       torch.tensor(b, dtype=F64, device=cond.device))

# what the host solver hands over, and what it needs for the next solve:
# UP and the DOWN list of the benchmark's end-to-end loop, and the three
# fields the node routines before the solve add
UP = ["VX", "VY", "PR", "SXX", "SXY", "EXX", "EXY", "ESP"]
DOWN = ["NU_M2C", "GG", "ND_M2C", "GD", "RO", "MRX", "MRY", "MVX", "MVY", "SPPE",
        "SXXE", "SXYE", "EXXE", "EXYE", "PHIS", "TK"]
DOWN_LATE = ["NU", "ND", "PHIS_IT"]
MARKER_FIELDS = ["X", "Y", "K", "E", "P", "EXX", "EXY", "XX", "XY", "VX", "VY", "PHI", "SLIPV"]


def nf(name: str) -> int:
    return getattr(abi, "NF_" + name)


def mf(name: str) -> int:
    return getattr(abi, "MF_" + name)


# ------------------------------------------------------------------ cases

def _step(xn, yn, per_x, per_y, **kw):
    c = dict(kind="step", xn=xn, yn=yn, per_x=per_x, per_y=per_y, dx=2000.0, refine=False,
             keep=1.0, random_fields=False, mode=2, antidiff=1, densimod=0, stoksmod=1,
             guess=abi.GUESS_PLAIN, dt_lo=1e8, dt_hi=1e8)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest model anyone steps (the tests' small grid): launches
        # and host latency
        dict(_step(51, 21, 4, 4), name="step_51x21"),
        # the 600 x 200 km megathrust model at 2 km, interseismic time step
        dict(_step(301, 101, 4, 4), name="step_301x101"),
        # the refined megathrust grid, scattered stresses and strain rates,
        # adaptive time steps from coseismic to interseismic
        dict(_step(1001, 401, 4, 4, dx=600.0, refine=True, random_fields=True,
                   dt_lo=1e-3, dt_hi=1e10), name="step_refined_1001x401"),
        # the benchmark's large model: 80 M markers, adaptive time steps,
        # Newton from the network's start
        dict(_step(4001, 1001, 5, 4, dx=500.0, guess=abi.GUESS_LEARNED, dt_lo=1e-3, dt_hi=1e10),
             name="step_4001x1001"),
        # the 13-node stencil (interpolationmod 1) on an odd grid whose
        # markers have thinned out unevenly
        dict(_step(433, 187, 4, 3, dx=1500.0, keep=0.87, mode=1), name="step_13node_433x187"),
        # no antidiffusion, temperature-dependent density, no marker Newton,
        # Jaumann rotation, odd grid, uneven marker density
        dict(_step(811, 309, 4, 5, dx=1000.0, keep=0.9, antidiff=0, densimod=1, stoksmod=2,
                   guess=abi.GUESS_OFF), name="step_plain_811x309"),
        # the seismic cycle on the 600 x 200 km model
        dict(kind="cycle", xn=301, yn=101, per_x=4, per_y=4, dx=2000.0, steps=8, dt=1e8,
             name="cycle_301x101"),
        # the Newton benchmark: 4 M seeded states, plain start
        dict(kind="newton", n=4_000_000, guess=abi.GUESS_PLAIN, fp64=0, name="newton_4M"),
        # an odd block with the network's start
        dict(kind="newton", n=300_007, guess=abi.GUESS_LEARNED, fp64=0,
             name="newton_learned_300k"),
        # cell sort of a model's markers, array order scattered within 64
        # neighbouring cells
        dict(kind="sort", xn=1501, yn=401, n=9_000_017, name="sort_1501x401"),
        # the Stokes matrix of the 600 x 200 km model
        dict(kind="stokes", xn=301, yn=101, per_x=4, per_y=4, dx=2000.0, name="stokes_301x101"),
        # temperature update and a restart file's marker arrays
        dict(kind="restart", xn=301, yn=101, per_x=4, per_y=4, dx=2000.0, keep=0.95,
             name="restart_301x101"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "cycle", "newton", "sort", "stokes",
                       "restart"])
    if kind == "newton":
        return dict(kind=kind, n=_log_int(rng, 1_000, 4_000_000),
                    guess=rng.choice([abi.GUESS_PLAIN, abi.GUESS_LEARNED]),
                    fp64=1 if rng.random() < 0.2 else 0)
    xn, yn = _log_int(rng, 24, 1600), _log_int(rng, 14, 700)
    if kind == "sort":
        return dict(kind=kind, xn=xn, yn=yn,
                    n=min(10_000_000, int((xn - 1) * (yn - 1) * rng.uniform(4, 24)) + 1))
    if kind != "step":
        xn, yn = min(xn, 600), min(yn, 240)
    per_x, per_y = rng.choice([(3, 3), (4, 3), (4, 4), (4, 4), (5, 4), (5, 5)])
    geo = dict(xn=xn, yn=yn, per_x=per_x, per_y=per_y, dx=rng.choice([500.0, 1000.0, 2000.0]))
    if kind == "cycle":
        return dict(kind=kind, steps=8, dt=10.0 ** rng.uniform(0, 9), **geo)
    if kind == "stokes":
        return dict(kind=kind, **geo)
    if kind == "restart":
        return dict(kind=kind, keep=rng.uniform(0.8, 1.0), **geo)
    dt = rng.choice([(1e8, 1e8), (1e8, 1e8), (1e-3, 1e10), (1e3, 1e3)])
    return _step(xn, yn, per_x, per_y, dx=geo["dx"], refine=rng.random() < 0.4,
                 keep=rng.choice([1.0, rng.uniform(0.8, 1.0)]),
                 random_fields=rng.random() < 0.4, mode=rng.choice([2, 2, 2, 1]),
                 antidiff=rng.choice([1, 1, 1, 0]), densimod=rng.choice([0, 0, 1]),
                 stoksmod=rng.choice([1, 1, 2]),
                 guess=rng.choice([abi.GUESS_PLAIN, abi.GUESS_PLAIN, abi.GUESS_LEARNED,
                                   abi.GUESS_OFF]),
                 dt_lo=dt[0], dt_hi=dt[1])


# ----------------------------------------------------------- model states
# The fields of synth.make_case, drawn on the GPU.

def _grid(case):
    xn, yn, dx = case["xn"], case["yn"], case["dx"]

    def lines(n, centre):
        w = np.ones(n - 1)
        if case.get("refine"):  # fine zone around `centre`, five times coarser at the far end
            w += 4.0 * np.abs((np.arange(n - 1) + 0.5) / (n - 1) - centre)
        w *= (n - 1) * dx / w.sum()
        return np.concatenate([[0.0], np.cumsum(w)])

    return lines(xn, 0.35), lines(yn, 0.1)


def _temperature(y):
    return 273.0 + 1350.0 * torch.erf(y / (2.0 * math.sqrt(1e-6 * 60e6 * 3.15576e7)))


def _stream(x, y, xs, ys):
    """velocity, strain rates and spin of a convection cell plus a Gaussian
    shear band along the slab top"""
    A, kx, ky = synth.V_PLATE * ys / math.pi, math.pi / xs, math.pi / ys
    sx, cx, sy, cy = torch.sin(kx * x), torch.cos(kx * x), torch.sin(ky * y), torch.cos(ky * y)
    t0, t1 = math.cos(synth.DIP), math.sin(synth.DIP)
    x0 = synth.SLAB_X0 * xs
    d = (y - math.tan(synth.DIP) * (x - x0)) * t0
    g = synth.V_PLATE * torch.exp(-0.5 * (d / 1e3) ** 2) * (x > x0)
    dg = -g * d / 1e6
    vx, vy = A * ky * sx * cy + g * t0, -A * kx * cx * sy + g * t1
    exx = A * ky * kx * cx * cy - t0 * t1 * dg
    dvxdy, dvydx = -A * ky * ky * sx * sy + t0 * t0 * dg, A * kx * kx * sx * sy - t1 * t1 * dg
    return vx, vy, exx, 0.5 * (dvxdy + dvydx), 0.5 * (dvydx - dvxdy)


def _model(case, seed):
    """(params, gx, gy, rock table, nodes, markers, types, bonds); nodes and
    markers as 64-bit device tensors"""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    dev = dict(device="cuda", dtype=F64)

    def uni(n, lo=0.0, hi=1.0):
        return torch.rand(n, generator=gen, **dev) * (hi - lo) + lo

    def nrm(n, s=1.0):
        return torch.randn(n, generator=gen, **dev) * s

    gx, gy = _grid(case)
    xn, yn = gx.size, gy.size
    xs, ys, nn = float(gx[-1]), float(gy[-1]), xn * yn
    p = synth.default_params(
        xnumx=xn, ynumy=yn, xsize=xs, ysize=ys, xstpx=xs / (xn - 1), ystpy=ys / (yn - 1),
        timestep=case.get("dt", case.get("dt_lo", 1e8)), interpolationmod=case.get("mode", 2),
        antidiffinter=case.get("antidiff", 1), densimod=case.get("densimod", 0),
        stoksmod=case.get("stoksmod", 1), newton_guess=case.get("guess", abi.GUESS_PLAIN))
    GX, GY = torch.tensor(gx, **dev), torch.tensor(gy, **dev)

    per = case["per_x"] * case["per_y"]
    ids = torch.arange((xn - 1) * (yn - 1) * per, device="cuda")
    if case.get("keep", 1.0) < 1.0:
        few = torch.randperm(ids.numel(), generator=gen, device="cuda")
        ids = few[:int(case["keep"] * ids.numel())].sort()[0]
    n = ids.numel()
    cell, sub = ids // per, ids % per
    ci, cj = cell // (yn - 1), cell % (yn - 1)
    fx = ((sub // case["per_y"]).to(F64) + uni(n)) / case["per_x"]
    fy = ((sub % case["per_y"]).to(F64) + uni(n)) / case["per_y"]
    x = GX[ci] + fx * (GX[ci + 1] - GX[ci])
    y = GY[cj] + fy * (GY[cj + 1] - GY[cj])
    del ids, cell, sub, ci, cj, fx, fy
    top = math.tan(synth.DIP) * (x - synth.SLAB_X0 * xs)
    t = torch.full((n,), 5, device="cuda", dtype=torch.int8)
    t[y < 35e3], t[y < 15e3], t[y < 2e3] = 4, 3, 2
    t[(x > synth.SLAB_X0 * xs) & (y > top) & (y < top + 8e3 / math.cos(synth.DIP))] = 6
    vx, vy, exx, exy, _ = _stream(x, y, xs, ys)
    M = {"X": x, "Y": y, "K": _temperature(y) + nrm(n, 5.0)}
    if case.get("random_fields"):
        M["XX"], M["XY"] = nrm(n, 5e6), nrm(n, 5e6)
        mag, ang = 10.0 ** uni(n, -18, -10), uni(n, 0, 2 * math.pi)
        M["EXX"], M["EXY"] = mag * torch.cos(ang), mag * torch.sin(ang)
    else:
        eta = 10.0 ** uni(n, 20.0, 22.0)
        M["EXX"], M["EXY"] = exx * (1 + nrm(n, 0.05)), exy * (1 + nrm(n, 0.05))
        M["XX"] = 2 * eta * M["EXX"] + nrm(n, 1e5)
        M["XY"] = 2 * eta * M["EXY"] + nrm(n, 1e5)
    M["P"] = 3000.0 * 9.81 * y + nrm(n, 1e5)
    M["E"] = nrm(n, 0.01).abs()
    M["VX"], M["VY"] = vx * (1 + nrm(n, 0.01)), vy * (1 + nrm(n, 0.01))
    M["PHI"] = _pick((y - 10e3).abs() <= 250.0, 8.0, 10.0) + nrm(n, 0.1)
    M["SLIPV"] = 10.0 ** uni(n, -12, -8)

    I = torch.arange(xn, device="cuda").repeat_interleave(yn)
    J = torch.arange(yn, device="cuda").repeat(xn)
    xb, yb = GX[I], GY[J]
    xr, yd = GX[(I + 1).clamp(max=xn - 1)], GY[(J + 1).clamp(max=yn - 1)]
    xl, yu = GX[(I - 1).clamp(min=0)], GY[(J - 1).clamp(min=0)]
    xc, yc = 0.5 * (xl + xb), 0.5 * (yu + yb)
    N = {k[3:]: torch.zeros(nn, **dev) for k in vars(abi) if k.startswith("NF_") and k != "NF_N"}
    N["VX"] = _stream(xb, 0.5 * (yb + yd), xs, ys)[0]
    N["VY"] = _stream(0.5 * (xb + xr), yb, xs, ys)[1]
    for k in ("MVX", "MVXE"):
        N[k] = N["VX"] * (1 + nrm(nn, 1e-3))
    for k in ("MVY", "MVYE"):
        N[k] = N["VY"] * (1 + nrm(nn, 1e-3))
    N["EXX"] = _stream(xc, yc, xs, ys)[2]
    _, _, _, N["EXY"], N["ESP"] = _stream(xb, yb, xs, ys)
    N["SXX"] = 2e21 * N["EXX"] + nrm(nn, 1e4)
    N["SXY"] = 2e21 * N["EXY"] + nrm(nn, 1e4)
    N["PR"] = 3000.0 * 9.81 * yc + 10e6 + nrm(nn, 1e4)
    for k, b, s in (("EXXE", "EXX", 1e-2), ("EXXEE", "EXX", 1e-2), ("EXYE", "EXY", 1e-2),
                    ("EXYEE", "EXY", 1e-2), ("SXXE", "SXX", 1e-2), ("SXXEE", "SXX", 1e-2),
                    ("SXYE", "SXY", 1e-2), ("SXYEE", "SXY", 1e-2), ("SXXS", "SXX", 1e-2),
                    ("SPPE", "PR", 1e-4), ("SPPEE", "PR", 1e-4), ("SPPES", "PR", 1e-4)):
        N[k] = N[b] * (1 + nrm(nn, s))
    band = (yb - 10e3).abs() <= 100.0
    for k in ("PHIS", "PHIS_IT", "PHIE"):
        N[k] = _pick(band, 8.0, 50.0) + nrm(nn, 0.05)
    N["PE"] = nrm(nn, 0.01).abs()
    N["PES"], N["PEE"] = N["PE"] + 1e-4, N["PE"] * (1 + nrm(nn, 1e-2))
    N["RK_SLIPRS_FINAL"] = 10.0 ** uni(nn, -11, -8)
    N["RK_PHIDTS_FINAL"] = nrm(nn, 1e-9)
    N["RK_SLIPRS_SOLVED"] = N["RK_SLIPRS_FINAL"] * 1.1
    N["RK_PHIDTS_SOLVED"] = N["RK_PHIDTS_FINAL"] * 0.9
    N["NU_M2C"] = 10.0 ** uni(nn, 20, 23)
    N["NU"], N["ND_M2C"], N["ND"] = N["NU_M2C"].clone(), 10.0 ** uni(nn, 20, 23), N["NU_M2C"].clone()
    N["GG"], N["GD"] = torch.full((nn,), 3.0e10, **dev), torch.full((nn,), 3.0e10, **dev)
    N["BM"] = 5.0e10 * (1 + uni(nn, 0, 0.1))
    N["TK"] = _temperature(yb)
    N["TK2"] = N["TK"] + nrm(nn, 1e-4)
    N["RO"], N["CP"], N["KT"] = 3000.0 + uni(nn, 0, 300), 1000.0 + uni(nn), 2.0 + uni(nn)
    N["PRS"] = 3000.0 * 9.81 * yb + 10e6 + nrm(nn, 1e4)
    N["MUS_S"] = _pick(band, 0.2, 0.6)
    N["SYIELDS"] = 6e6 * (1 + uni(nn, 0, 0.1))
    for k, f in (("a", "AS"), ("b", "BS"), ("L", "LS")):
        N[f] = _pick(band, p[k + "_vw"], p[k + "_hr"]) * (1 + uni(nn, 0, 0.01))
    N["V0S"] = _pick(band, p["V0_vw"], p["V0_hr"])
    return p, gx, gy, synth.rock_table(), N, M, t, synth._bonds(xn, yn)


_PINNED: dict = {}  # pinned staging of the marker arrays, one block per field, reused


def _host_marks(M):
    """the marker arrays in pinned host memory, as numpy (valid until the
    next call)"""
    out = {}
    for k, v in M.items():
        b = _PINNED.get(k)
        if b is None or b.numel() < v.numel():
            b = _PINNED[k] = torch.empty(v.numel(), dtype=F64, pin_memory=True)
        b[:v.numel()].copy_(v)
        out[mf(k)] = b[:v.numel()].numpy()
    return out


def _pinned_like(names, nn):
    return {nf(k): torch.zeros(nn, dtype=F64, pin_memory=True).numpy() for k in names}


def _context(case, seed):
    p, gx, gy, rt, N, M, t, bonds = _model(case, seed)
    m = mic.MarkerInCell(p, t.numel())
    m.set_grid(gx, gy)
    m.set_rock_table(rt)
    m.set_bonds(*bonds)
    m.upload_markers(_host_marks(M), t.cpu().numpy())
    m.upload_nodes({nf(k): v.cpu().numpy() for k, v in N.items() if bool(v.any())})
    m.synchronize()
    return m, N


def _network(seed):
    """packed network parameters, normalised to the range of Newton states"""
    X = np.array([[-8, -2, 0.9, -0.8, 0.2, 5, -8, -9], [3, 8, 2.0, 1.0, 0.6, 50, 11, -8]], float)
    Y = np.array([[-40.0, 5.0], [-10.0, 50.0]])
    return newton.random_params(seed, X, Y)


def _dts(case, seed):
    r = np.random.default_rng(seed)
    return (10.0 ** r.uniform(math.log10(case["dt_lo"]), math.log10(case["dt_hi"]), 5)).tolist()


def _states(n, seed):
    """newton.rsf_states' distributions, drawn on the GPU"""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))

    def uni(lo, hi):
        return torch.rand(n, generator=gen, device="cuda", dtype=F64) * (hi - lo) + lo

    S = torch.zeros((abi.RS_N, n), device="cuda", dtype=F64)
    b = torch.full((n,), 0.015, device="cuda", dtype=F64)
    a, V, sn, V0 = b + uni(-0.01, 0.015), 10.0 ** uni(-15, 1), uni(5e6, 100e6), 10.0 ** uni(-9, -6)
    phi = torch.log(V0 / V) + torch.randn(n, generator=gen, device="cuda", dtype=F64)
    w = torch.log(V / (2 * V0)) + (0.6 + b * phi) / a
    A = torch.where(w > 20, w + math.log(2.0), torch.asinh(torch.exp(w.clamp(max=20))))
    for k, v in ((abi.RS_VOLD, V), (abi.RS_PHIOLD, phi), (abi.RS_A, a), (abi.RS_B, b),
                 (abi.RS_L, 10.0 ** uni(-3, -1)), (abi.RS_V0, V0), (abi.RS_SN, sn),
                 (abi.RS_DT, 10.0 ** uni(-3, 10)), (abi.RS_TAUOLD, sn * a * A * uni(0.8, 1.2)),
                 (abi.RS_EDOT, 10.0 ** uni(-18, -10)), (abi.RS_ETA, 10.0 ** uni(18, 25))):
        S[k] = v
    S[abi.RS_MU0], S[abi.RS_G] = 0.6, 3.0e10
    return S


# ---------------------------------------------------------------- prepare

def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "newton":
        p = synth.default_params(xnumx=8, ynumy=8, xsize=7.0, ysize=7.0, xstpx=1.0, ystpy=1.0,
                                 newton_precision=abi.NEWTON_FP64 if case["fp64"]
                                 else abi.NEWTON_SPLIT)
        s["mic"] = mic.MarkerInCell(p, 1)
        if case["guess"] == abi.GUESS_LEARNED:
            newton.load(s["mic"], _network(seed))
        s["states"] = _states(case["n"], seed)
        return s
    if kind == "sort":
        n, xn, yn = case["n"], case["xn"], case["yn"]
        gen = torch.Generator(device="cuda").manual_seed(int(seed))
        u = torch.rand((3, n), generator=gen, device="cuda", dtype=F64)
        ncell = (xn - 1) * (yn - 1)
        at = torch.arange(n, device="cuda").to(F64) / n * ncell + (u[0] - 0.5) * 64
        c = at.long().clamp(0, ncell - 1)
        s["gx"] = torch.arange(xn, device="cuda", dtype=F64) * 500.0
        s["gy"] = torch.arange(yn, device="cuda", dtype=F64) * 500.0
        s["x"] = ((c // (yn - 1)).to(F64) + u[1]) * 500.0
        s["y"] = ((c % (yn - 1)).to(F64) + u[2]) * 500.0
        i32 = dict(device="cuda", dtype=torch.int32)
        s["cell"], s["perm"] = torch.empty(n, **i32), torch.empty(n, **i32)
        s["start"] = torch.empty(ncell + 1, **i32)
        return s
    m, N = _context(case, seed)
    s["mic"], nn = m, m.nn
    if kind == "step":
        if case["guess"] == abi.GUESS_LEARNED:
            newton.load(m, _network(seed))
        s["dts"], s["k"] = _dts(case, seed), 0
        s["up"], s["down"], s["late"] = (_pinned_like(k, nn) for k in (UP, DOWN, DOWN_LATE))
        for k in UP:
            s["up"][nf(k)][:] = N[k].cpu().numpy()
    elif kind == "cycle":
        v = [N[k].cpu().numpy() for k in ("VX", "VY")]
        m.cycle_set_velocity(0, *v)
        s["down"] = _pinned_like(DOWN + DOWN_LATE, nn)
    elif kind == "stokes":
        m.marker2nodes()
        m.compute_before_solve(m.params["timestep"], 0)
        m.interpolate_basic2center()
        m.synchronize()
    elif kind == "restart":
        s["solved"] = _pinned_like(["TK", "TK2"], nn)
        for k in ("TK", "TK2"):
            s["solved"][nf(k)][:] = N[k].cpu().numpy()
        s["out"] = {mf(k): torch.zeros(m.n, dtype=F64, pin_memory=True).numpy()
                    for k in MARKER_FIELDS}
    return s


# -------------------------------------------------------------------- run

def _names(arrays, names):
    return {k.lower(): arrays[nf(k)] for k in names}


def _run_step(s):
    m, dt = s["mic"], s["dts"][s["k"] % len(s["dts"])]
    s["k"] += 1
    m.set_params(timestep=dt)
    m.upload_nodes(s["up"])
    m.interpolate_center2basic(dt)
    deltas = m.compute_after_solve(dt, 0)
    m.copyarrays()
    m.nodes2markers_move()
    m.marker2nodes()
    m.download_nodes_async(s["down"])
    m.interpolate_center2basic_old()
    m.compute_before_solve(dt, 0)
    m.interpolate_basic2center()
    late = m.download_nodes(list(s["late"]), into=s["late"])
    m.wait_downloads()
    return dict(_names(s["down"], DOWN), **_names(late, DOWN_LATE), deltas=deltas)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        return _run_step(state)
    m = state.get("mic")
    if kind == "cycle":
        for _ in range(case["steps"]):
            m.cycle_step(0, case["dt"])
            info = m.calc_timestep(1)
        return dict(info={k: info[k] for k in ("dt_f", "maxvel", "maxVx", "dtnvp", "dtd", "dtphi",
                                               "dtL")},
                    slip=m.cycle_slip(), marker_slip=m.cycle_marker_slip(),
                    nodes=_names(m.download_nodes([nf(k) for k in DOWN + DOWN_LATE],
                                                  into=state["down"]), DOWN + DOWN_LATE))
    if kind == "newton":
        out, it = newton.solve(m, state["states"], case["guess"], on_device=True)
        return dict(V=out[abi.RO_V], phi=out[abi.RO_PHI], tau=out[abi.RO_TAU],
                    residual=out[abi.RO_RES], iterations=it)
    if kind == "sort":
        o = [state[k] for k in ("cell", "perm", "start")]
        cellsort.sort_cells_static(state["gx"], state["gy"], state["x"], state["y"], *o)
        return o
    if kind == "stokes":
        dt = m.params["timestep"]
        return m.stokes_assemble(mukoef=dt * 30e5, dt=dt)
    m.upload_nodes(state["solved"])
    m.marker_temperature(1.0)
    out = m.download_markers(list(state["out"]), into=dict(state["out"]))
    return dict({k.lower(): out[mf(k)] for k in MARKER_FIELDS}, markt=out["markt"])


# ------------------------------------------------------------------- work

def work(case):
    """Marker state: 53 B read and 48 B written per step (cell, offsets,
    type, temperature, stresses, strain rates, pressure, strain, state,
    velocities), node fields 94 x 4 B, the host transfers at 8 B.  Operations
    per marker and step: about 1200 for the creep iteration and the
    properties, 500 for the node sums, 300 for the interpolations and the
    move, 200 for the Newton."""
    kind = case["kind"]
    if kind == "newton":
        return dict(bytes=case["n"] * ((abi.RS_N + abi.RO_N) * 8 + 4), flops=case["n"] * 5 * 400)
    if kind == "sort":
        return dict(bytes=case["n"] * (16 + 4 + 4) + (case["xn"] - 1) * (case["yn"] - 1) * 4,
                    flops=case["n"] * 40)
    nn = case["xn"] * case["yn"]
    n = (case["xn"] - 1) * (case["yn"] - 1) * case["per_x"] * case["per_y"] * case.get("keep", 1.0)
    if kind == "stokes":
        return dict(bytes=nn * (11 * 4 + 3 * (13 * 12 + 12)), flops=nn * 3 * 150)
    if kind == "restart":
        return dict(bytes=n * (8 + 8 + len(MARKER_FIELDS) * (4 + 8) + 2) + nn * 2 * 8,
                    flops=n * 80)
    if kind == "cycle":
        return dict(bytes=case["steps"] * (n * 101 + nn * 94 * 4) + 8 * (n + nn),
                    flops=case["steps"] * (n * 2200 + nn * 1500))
    io = 8 * (len(UP) + len(DOWN) + len(DOWN_LATE))
    newton_ops = 0 if case["guess"] == abi.GUESS_OFF else 200
    return dict(bytes=n * 101 + nn * (94 * 4 + io), flops=n * (2000 + newton_ops) + nn * 1500)


# ------------------------------------------------------------------ exact
# One pass in 64 bits: the formulas of the reference (interpolation.c,
# moveandrotatemarkers.c, density_ductilevisc_calc.c, calc_RSF.c,
# plastic.c) on the inputs as drawn.

def exact(case, seed):
    if case["kind"] == "step":
        n = (case["xn"] - 1) * (case["yn"] - 1) * case["per_x"] * case["per_y"]
        return None if n > 20_000_000 else _Exact(case, seed).one_pass()
    if case["kind"] == "newton":
        return _exact_newton(_states(case["n"], seed))
    if case["kind"] == "restart":
        return _Exact(case, seed).temperature()
    return None


def _exact_newton(S):
    Vold, phio, a, b, L, V0, mu0, sn, dt, tau, edot, eta, G = S
    W, rad = 400.0, 4.3303e6
    Ts, c1 = tau + 2 * G * dt * edot, 1 + G * dt / eta
    klin = rad * c1 + 2 * G * dt / W

    def friction(u):
        """slip rate, state, asinh term A and dA/du at u = log V"""
        V, e = torch.exp(u), torch.exp(phio)
        x, r = V * dt / L, V0 / torch.exp(u)
        ex, slow = torch.exp(-x), x <= 1e-6
        g = torch.where(slow, e * (1 - x) + V0 * dt / L, r + (e - r) * ex)
        dg = torch.where(slow, -e * x, -r + r * ex - (e - r) * ex * x)
        phi = torch.log(g)
        w = u - torch.log(2 * V0) + (mu0 + b * phi) / a
        A = torch.where(w > 20, w + math.log(2.0) + 0.25 * torch.exp(-2 * w),
                        torch.asinh(torch.exp(w.clamp(max=20))))
        return V, phi, A, (1 + b / a * dg / g) / torch.sqrt(1 + torch.exp(-2 * w))

    # Newton in log V from the previous slip rate, kept inside the bracket
    # (a velocity-weakening state can have three roots: the one this descent
    # reaches is the solution)
    floor = math.log(1e-40)
    lo, hi = torch.full_like(Ts, floor), torch.log(Ts / klin)
    V, phi, A, _ = friction(lo)
    at_floor = ~(hi > lo) | (sn * a * c1 * A + klin * V >= Ts)
    tau_floor = sn * a * A + rad * V
    u = torch.log(Vold)
    u = torch.where(u > lo, u, lo + 0.5e-3 * (hi - lo))
    u = torch.where(u < hi, u, hi - 1e-3 * (hi - lo))
    lo_known = torch.zeros_like(at_floor)
    for _ in range(100):
        V, phi, A, dA = friction(u)
        F, dF = sn * a * c1 * A + klin * V - Ts, sn * a * c1 * dA + klin * V
        lo, hi = torch.where(F < 0, u, lo), torch.where(F < 0, hi, u)
        lo_known |= F < 0
        un = u - F / dF
        low = ~lo_known & (dF > 0) & ~(un > lo)
        ok = (dF > 0) & (un > lo) & (un < hi)
        done = F.abs() <= 1e-15 * (F + Ts)
        u = torch.where(done, u, torch.where(low, floor, torch.where(ok, un, 0.5 * (lo + hi))))
    V, phi, A, _ = friction(u)
    return dict(V=torch.where(at_floor, 1e-40, V), phi=torch.where(at_floor, phio, phi),
                tau=torch.where(at_floor, tau_floor, sn * a * A + rad * V), residual=None,
                iterations=None)


class _Exact:
    def __init__(self, case, seed):
        self.case = case
        self.p, gx, gy, rt, self.N, self.M, self.t, self.bonds = _model(case, seed)
        self.gx, self.gy = torch.tensor(gx, device="cuda"), torch.tensor(gy, device="cuda")
        self.rt = torch.tensor(rt, device="cuda")
        self.xn, self.yn = gx.size, gy.size
        self.nn = self.xn * self.yn
        i = torch.arange(self.nn, device="cuda")
        self.m1, self.m2 = i // self.yn, i % self.yn
        self.inner = (self.m1 >= 1) & (self.m2 >= 1) & (self.m1 < self.xn - 1) & \
            (self.m2 < self.yn - 1)
        self.dt = _dts(case, seed)[0] if "dt_lo" in case else self.p["timestep"]

    def one_pass(self):
        deltas = self.after_solve()
        self.nodes2markers()
        self.move()
        self.marker2nodes()
        out = {k.lower(): self.N[k].clone() for k in DOWN}
        self.before_solve()
        self.basic2center()
        out.update({k.lower(): self.N[k] for k in DOWN_LATE}, deltas=deltas)
        return out

    def temperature(self):
        """the marker part of solve_temperature (temperature_iterate.c), rock
        markers inside the model"""
        N, M, yn = self.N, self.M, self.yn
        x, y = M["X"], M["Y"]
        a, b = self.cell(x, y)
        wx, wy = self.gx[a + 1] - self.gx[a], self.gy[b + 1] - self.gy[b]
        at = (a, b, (x - self.gx[a]) / wx, (y - self.gy[b]) / wy)
        T, T2 = self.bil(N["TK"], *at), self.bil(N["TK2"], *at)
        # the device holds the node conductivity, heat capacity and density
        k, c = self.bil(N["KT"], *at), self.bil(N["CP"] * N["RO"], *at)
        d = (T2 - M["K"]) * -torch.expm1(-k / c * 2 * (1 / wx ** 2 + 1 / wy ** 2) * self.dt)
        w, node = (1 - at[2]) * (1 - at[3]), a * yn + b
        s = torch.zeros((2, self.nn), dtype=F64, device="cuda")
        s[0].index_add_(0, node, w / wx / wy)
        s[1].index_add_(0, node, w / wx / wy * d)
        M["K"] = M["K"] + d + (T - T2) - (s[1] / s[0])[node] * w
        return dict({k.lower(): M[k] for k in MARKER_FIELDS}, markt=None)

    # --- node routines
    def four(self, f):
        q, yn = torch.zeros_like(f), self.yn
        i = self.inner.nonzero()[:, 0]
        q[i] = 0.25 * (f[i] + f[i + 1] + f[i + yn] + f[i + yn + 1])
        return q

    def after_solve(self):
        """interpolate_center2basic, compute_after_solve, copyarrays"""
        N, p, k = self.N, self.p, self.inner
        pl = N["EXX"] - (N["SXX"] - N["SXXE"]) / (2 * N["GD"] * self.dt) - N["SXX"] / (2 * N["ND_M2C"])
        N["EXXPL"][k] = self.four(pl)[k]
        N["SXXS"][k] = self.four(N["SXX"])[k]
        sig = torch.sqrt(N["SXXS"] ** 2 + N["SXY"] ** 2)
        V = 2 * N["V0S"] * torch.sinh(sig / (N["AS"] * p["nstress"])) * \
            torch.exp(-(N["MUS_S"] + N["BS"] * N["PHIS_IT"]) / N["AS"])
        V = torch.minimum(V, torch.sqrt(N["EXXPL"] ** 2 + N["EXY"] ** 2) * p["faultwidth"])
        V = torch.where(sig > 0, V.clamp(min=1e-40), 0.0)
        N["RK_SLIPRS_FINAL"][k] = V[k]
        d = (N["SYIELDS"] - sig)[k & (V > 0)]
        return float(torch.sqrt((d * d).mean()))

    def before_solve(self):
        N, p, k, dt, W = self.N, self.p, self.inner, self.dt, self.p["faultwidth"]
        V, L, V0, ph = N["RK_SLIPRS_FINAL"], N["LS"], N["V0S"], N["PHIS"]
        a, b, mu, nm = N["AS"], N["BS"], N["MUS_S"], N["NU_M2C"]
        x = V * dt / L
        new = torch.where(x <= 1e-6, torch.log(torch.exp(ph) * (1 - x) + V0 * dt / L),
                          torch.log(V0 / V + (torch.exp(ph) - V0 / V) * torch.exp(-x)))
        sy = p["nstress"] * a * torch.asinh(V / (2 * V0) * torch.exp((mu + new * b) / a)) + 4.3303e6 * V
        vp = torch.where(sy > 0, nm * sy / (2 * nm * V / W + sy), nm)
        sig = torch.sqrt(N["SXXS"] ** 2 + N["SXY"] ** 2)
        q = k & (sig > 0)
        N["PHIS_IT"][q] = new[q]
        N["NU"][k] = torch.where(sig > 0, vp, nm)[k]

    def basic2center(self):
        i = ((self.m1 >= 1) & (self.m2 >= 1)).nonzero()[:, 0]
        x = 0.5 * (self.gx[self.m1[i]] + self.gx[self.m1[i] - 1])
        y = 0.5 * (self.gy[self.m2[i]] + self.gy[self.m2[i] - 1])
        a, b = self.cell(x, y)
        a, b = a.clamp(1, self.xn - 3), b.clamp(1, self.yn - 3)
        e = ((x - self.gx[a]) / (self.gx[a + 1] - self.gx[a])).clamp(0, 1)
        n = ((y - self.gy[b]) / (self.gy[b + 1] - self.gy[b])).clamp(0, 1)
        self.N["ND"][i] = 1 / self.bil(1 / self.N["NU"], a, b, e, n)

    # --- interpolation
    def cell(self, x, y):
        return ((torch.searchsorted(self.gx, x, right=True) - 1).clamp(0, self.xn - 2),
                (torch.searchsorted(self.gy, y, right=True) - 1).clamp(0, self.yn - 2))

    def bil(self, f, a, b, e, n):
        m, yn = a * self.yn + b, self.yn
        return (1 - e) * (1 - n) * f[m] + (1 - e) * n * f[m + 1] + e * (1 - n) * f[m + yn] + \
            e * n * f[m + yn + 1]

    def stencils(self, x, y):
        """(a, b, e, n) of a point on the basic, pressure, vx and vy nodes"""
        gx, gy, xn, yn = self.gx, self.gy, self.xn, self.yn
        x, y = x.clamp(0, self.p["xsize"]), y.clamp(0, self.p["ysize"])
        cx, cy = self.cell(x, y)
        hx, hy = 0.5 * (gx[cx] + gx[cx + 1]), 0.5 * (gy[cy] + gy[cy + 1])

        def at(a, b, sx, sy):
            if sx == 0:
                e = (x - gx[a]) / (gx[a + 1] - gx[a])
            else:
                q = a if sx > 0 else a - 1
                e = (x - 0.5 * (gx[q] + gx[q + 1])) / (0.5 * (gx[q + 2] - gx[q]))
            if sy == 0:
                n = (y - gy[b]) / (gy[b + 1] - gy[b])
            else:
                q = b if sy > 0 else b - 1
                n = (y - 0.5 * (gy[q] + gy[q + 1])) / (0.5 * (gy[q + 2] - gy[q]))
            return a, b, e, n

        return dict(
            basic=at(cx.clamp(1, xn - 3), cy.clamp(1, yn - 3), 0, 0),
            centre=at((cx + (x > hx)).clamp(1, xn - 2), (cy + (y > hy)).clamp(1, yn - 2), -1, -1),
            vx=at(cx, (cy - (y < hy).long()).clamp(0, yn - 3), 0, 1),
            vy=at((cx - (x < hx).long()).clamp(0, xn - 3), cy, 1, 0))

    # --- scatter
    def weights(self, kind, x, y):
        """(node, weight) pairs of the marker -> node stencil of one node kind"""
        yn, mode = self.yn, self.case["mode"]
        cx, cy = self.cell(x, y)
        wx, wy = self.gx[cx + 1] - self.gx[cx], self.gy[cy + 1] - self.gy[cy]
        u, v, s = (x - self.gx[cx]) / wx, (y - self.gy[cy]) / wy, 1 / wx / wy

        def lin(a, f):
            return f if a else 1 - f

        def half(k, f):
            return (0.5 - f).clamp(min=0) if k == 0 else (f - 0.5).clamp(min=0) if k == 2 \
                else 1 - (f - 0.5).abs()

        def side(a, f):  # the half of the cell next to the node only
            return (f > 0.5) if a else (f < 0.5)

        def tent(f):
            return 1 - 2 * (f - 0.5).abs()

        two = ((0, 0), (0, 1), (1, 0), (1, 1))
        if mode == 2:
            w = {"basic": [(a, b, side(a, u) * side(b, v) * (2 * u - 1).abs() * (2 * v - 1).abs())
                           for a, b in two],
                 "vx": [(a, 0, side(a, u) * lin(a, u) * half(1, v)) for a in (0, 1)],
                 "vy": [(0, b, side(b, v) * half(1, u) * lin(b, v)) for b in (0, 1)],
                 "centre": [(1, 1, tent(u) * tent(v))]}[kind]
        else:
            w = {"basic": [(a, b, lin(a, u) * lin(b, v)) for a, b in two],
                 "vx": [(a, b, lin(a, u) * half(b + 1, v)) for a in (0, 1) for b in (-1, 0, 1)],
                 "vy": [(a, b, half(a + 1, u) * lin(b, v)) for a in (-1, 0, 1) for b in (0, 1)],
                 "centre": [(a, b, half(a, u) * half(b, v)) for a in range(3) for b in range(3)],
                 }[kind]
        for a, b, f in w:
            f = f * s * ((cx + a >= 0) & (cx + a < self.xn) & (cy + b >= 0) & (cy + b < yn))
            yield ((cx + a) * yn + cy + b).clamp(0, self.nn - 1), f

    def sums(self, kind, x, y, vals):
        out = [torch.zeros(self.nn, dtype=F64, device="cuda") for _ in vals]
        for node, w in self.weights(kind, x, y):
            for o, q in zip(out, vals):
                o.index_add_(0, node, w * q)
        return out

    def density(self):
        return self.rt[abi.RT_RO][self.t.long()]

    # --- nodes2markers (all markers start inside the model)
    def nodes2markers(self):
        N, M = self.N, self.M
        st = self.stencils(M["X"], M["Y"])
        src = dict(EXY=("EXY", "EXYE", "basic"), XY=("SXY", "SXYE", "basic"),
                   E=("PES", "PE", "basic"), PHI=("PHIS_IT", "PHIS", "basic"),
                   EXX=("EXX", "EXXE", "centre"), XX=("SXX", "SXXE", "centre"),
                   P=("PR", "SPPE", "centre"), VX=("VX", "MVX", "vx"), VY=("VY", "MVY", "vy"))
        if not self.case["antidiff"]:
            for k, (f, g, s) in src.items():
                M[k] += self.bil(N[f] - N[g], *st[s])
            return
        for k, (f, _, s) in src.items():
            M[k] = self.bil(N[f], *st[s])
        x, y, one, ro = M["X"], M["Y"], torch.ones_like(M["X"]), self.density()
        *s, w = self.sums("basic", x, y, [M["PHI"], M["XY"], M["EXY"], M["E"], one])
        q = (w != 0) & self.inner
        for k, v in zip(("PHIE", "SXYEE", "EXYEE", "PEE"), s):
            N[k][q] = (v / w)[q]
        *s, w = self.sums("centre", x, y, [M["P"], M["XX"], M["EXX"], one])
        q = (w != 0) & (self.m1 >= 1) & (self.m2 >= 1)
        for k, v in zip(("SPPEE", "SXXEE", "EXXEE"), s):
            N[k][q] = (v / w)[q]
        if self.case["mode"] == 2:
            for k, e in (("vx", "MVXE"), ("vy", "MVYE")):
                v, mr, w = self.sums(k, x, y, [M[k.upper()] * ro, ro, one])
                N[e] = torch.where(w != 0, v / mr, N[e])

    # --- moveandrotatemarkers
    def velocity(self, x, y):
        N, yn = self.N, self.yn
        st = self.stencils(x, y)
        gx, gy = self.gx, self.gy
        xc, yc = x.clamp(0, self.p["xsize"]), y.clamp(0, self.p["ysize"])
        edge = (xc < 0.5 * (gx[0] + gx[1])) | (xc > 0.5 * (gx[-2] + gx[-1])) | \
            (yc < 0.5 * (gy[0] + gy[1])) | (yc > 0.5 * (gy[-2] + gy[-1]))
        r = _pick(edge, 1.0, 2.0 / 3.0)
        px = 0.5 * (torch.roll(N["VX"], 1) + torch.roll(N["VX"], yn + 1))
        py = 0.5 * (torch.roll(N["VY"], yn) + torch.roll(N["VY"], yn + 1))
        vx = self.bil(px, *st["centre"]) * (1 - r) + self.bil(N["VX"], *st["vx"]) * r
        vy = self.bil(py, *st["centre"]) * (1 - r) + self.bil(N["VY"], *st["vy"]) * r
        return vx, vy, self.bil(N["ESP"], *st["basic"])

    def move(self):
        M, p, dt = self.M, self.p, self.dt
        x, y = M["X"], M["Y"]
        k1 = self.velocity(x, y)
        k2 = self.velocity(x + k1[0] * dt / 2, y + k1[1] * dt / 2)
        k3 = self.velocity(x + k2[0] * dt / 2, y + k2[1] * dt / 2)
        k4 = self.velocity(x + k3[0] * dt, y + k3[1] * dt)
        vx, vy, sp = ((a + 2 * b + 2 * c + d) / 6 for a, b, c, d in zip(k1, k2, k3, k4))
        M["X"], M["Y"], sp = x + dt * vx, y + dt * vy, sp * dt
        xx, xy = M["XX"], M["XY"]
        if p["stoksmod"] == 1:
            M["XX"] = xx * torch.cos(2 * sp) + xy * torch.sin(2 * sp)
            M["XY"] = -xx * torch.sin(2 * sp) + xy * torch.cos(2 * sp)
        else:
            M["XX"], M["XY"] = xx + 2 * xy * sp, xy - 2 * xx * sp
        out = (M["X"] < 0) | (M["Y"] < 0) | (M["X"] > p["xsize"]) | (M["Y"] > p["ysize"])
        for k in ("K", "E"):
            M[k] = torch.where(out, 0.0, M[k])

    # --- marker2nodes
    def viscosity(self, t, T, mpb, xx, xy):
        p, R = self.p, self.rt
        nu, dh, dv = R[abi.RT_NU][t], R[abi.RT_DH][t], R[abi.RT_DV][t]
        ss, mm, gg = R[abi.RT_SS][t], R[abi.RT_MM][t], R[abi.RT_GG][t]
        eta = nu.clone()
        i = (((dh != 0) | (dv != 0)) & (ss != 0) & (mm != 1)).nonzero()[:, 0]
        nu, dh, dv, ss, mm, gdt = nu[i], dh[i], dv[i], ss[i], mm[i], gg[i] * self.dt
        sig = torch.sqrt(xx[i] ** 2 + xy[i] ** 2)
        e1 = torch.exp(((dh + dv * mpb[i]) / (8.314 * T[i])).clamp(max=150.0))
        diff = 0.5 * nu / ss ** (mm - 1) * e1
        disl = 0.5 * sig * nu * e1 / sig ** mm
        coeff, prev = disl ** (1 / mm), torch.zeros_like(disl)
        live = torch.arange(i.numel(), device="cuda")
        for k in range(1, 51):
            d, f, m, c = disl[live], diff[live], mm[live], coeff[live]
            mnu = 1 / (1 / f + 1 / d)
            base = (f + d) / f * (gdt[live] + mnu)
            f2 = d - c * base ** ((m - 1) / m)
            df = 1 - (m - 1) / (m * f) * c * base ** (-1 / m) * \
                ((gdt[live] + mnu) + f ** (2 / (f + d)))
            disl[live] = d - f2 / df
            if k > 3:
                go = ~(torch.log10(mnu / prev[live]).abs() < 1e-6)
                prev[live] = mnu
                live = live[go]
                if not live.numel():
                    break
            else:
                prev[live] = mnu
        v = (1 / (1 / diff + 1 / disl)).clamp(p["nubeg"], p["nuend"])
        v = torch.minimum(torch.maximum(v, R[abi.RT_N0][t[i]]), R[abi.RT_N1][t[i]])
        eta[i] = v
        return eta

    def marker2nodes(self):
        N, p, R, c = self.N, self.p, self.rt, self.case
        ins = (self.M["X"] > 0) & (self.M["Y"] > 0) & (self.M["X"] < p["xsize"]) & \
            (self.M["Y"] < p["ysize"])
        M, t = {k: v[ins] for k, v in self.M.items()}, self.t[ins].long()
        x, y, T, one = M["X"], M["Y"], M["K"], torch.ones_like(M["X"])
        mpb = 1e-5 * self.bil(N["PR"], *self.stencils(x, y)["centre"])
        bb, ro = R[abi.RT_BB][t], R[abi.RT_RO][t]
        if c["densimod"]:
            ro = ro * (1 - bb * (T - 298.15)) * (1 + R[abi.RT_AA][t] * (mpb - 1) * 1e-3)
        nu = self.viscosity(t, T, mpb, M["XX"], M["XY"])
        nug = nu / R[abi.RT_GG][t]
        r = (y - (p["fault_y"] + p["fault_slope"] * x)).abs()
        phi = torch.where(r <= p["fault_hw"], M["PHI"], 50.0)
        antid = c["antidiff"] == 1
        zero = torch.zeros(self.nn, dtype=F64, device="cuda")

        def node(q, avg, cur, prev):
            v = N[cur] + (avg - N[prev]) if antid else avg
            return torch.where(q, v, zero)

        snu, sg, sphi, sxy, sexy, ste, sro, stk, w = self.sums(
            "basic", x, y, [nu, nug, phi, M["XY"], M["EXY"], M["E"], ro, T, one])
        q = (w != 0) & self.inner
        N["PHIS"] = node(q, sphi / w, "PHIS_IT", "PHIE")
        N["SXYE"], N["EXYE"] = node(q, sxy / w, "SXY", "SXYEE"), node(q, sexy / w, "EXY", "EXYEE")
        N["PE"] = torch.where(q, node(q, ste / w, "PES", "PEE").clamp(min=0), N["PE"])
        N["NU_M2C"] = torch.where(q, snu / w, N["NU_M2C"])
        N["GG"] = torch.where(q, snu / sg, zero)
        N["RO"], N["TK"] = torch.where(w != 0, sro / w, zero), torch.where(w != 0, stk / w, zero)
        rb = (self.gy[self.m2] - (p["fault_y"] + p["fault_slope"] * self.gx[self.m1])).abs()
        self.friction(q, rb <= p["fault_hw"], self.gx[self.m1])
        N["NU"], N["ND"] = zero.clone(), zero.clone()
        snu, sg, sxx, sexx, sp, w = self.sums("centre", x, y,
                                              [nu, nug, M["XX"], M["EXX"], M["P"], one])
        q = (w != 0) & (self.m1 >= 1) & (self.m2 >= 1)
        N["SXXE"], N["EXXE"] = node(q, sxx / w, "SXX", "SXXEE"), node(q, sexx / w, "EXX", "EXXEE")
        N["SPPE"] = node(q, sp / w, "PR", "SPPEE")
        N["ND_M2C"] = torch.where(q, snu / w, N["ND_M2C"])
        N["GD"] = torch.where(q, snu / sg, zero)
        for k, V, MV, MVE, MR in (("vx", "VX", "MVX", "MVXE", "MRX"), ("vy", "VY", "MVY", "MVYE", "MRY")):
            s, mr, w = self.sums(k, x, y, [M[V] * ro, ro, one])
            N[MV], N[MR] = node(w != 0, s / mr, V, MVE), torch.where(w != 0, mr / w, zero)
        self.boundary()

    def friction(self, q, band, x):
        """calc_frictionpara_nodes on nodes q; zero elsewhere"""
        p, N = self.p, self.N
        h2 = 2 * p["half_range"]
        for k, f in (("a", "AS"), ("b", "BS"), ("L", "LS"), ("V0", "V0S")):
            vw, vs, hr = p[k + "_vw"], p[k + "_vs"], p[k + "_hr"]
            up = vs + (x - p["start_updip"]) / h2 * (vw - vs)
            dn = vw - (x - p["start_downdip"]) / h2 * (vw - vs)
            v = torch.where((x > p["end_updip"]) & (x < p["start_downdip"]), vw,
                            torch.where((x >= p["start_updip"]) & (x <= p["end_updip"]), up,
                                        torch.where((x >= p["start_downdip"]) & (x < p["end_downdip"]),
                                                    dn, vs)))
            N[f] = torch.where(q, torch.where(band, v, hr), 0.0)
        N["MUS_S"] = torch.where(q, _pick(band, 0.2, 0.6), 0.0)

    def boundary(self):
        """the boundary equations that end marker2nodes: a constant plus one
        reference each, followed through their references"""
        N, nn = self.N, self.nn
        bm, bn, bv = (torch.tensor(b, device="cuda") for b in self.bonds)
        bn, bv = bn.view(-1, 3), bv.view(-1, 4)
        N["MVX"] = torch.where(self.m2 < self.yn - 1, N["MVX"], 0.0)
        N["MVY"] = torch.where(self.m1 < self.xn - 1, N["MVY"], 0.0)
        for f, rows, off, step in (("MVX", bm[1:3 * nn:3], 2, 3), ("MVY", bm[2:3 * nn:3], 3, 3),
                                   ("SPPE", bm[0:3 * nn:3], 1, 3), ("TK", bm[3 * nn:], 1 + 3 * nn, 1)):
            k = (rows > 0)
            if f == "MVX":
                k = k & (self.m2 < self.yn - 1)
            if f == "MVY":
                k = k & (self.m1 < self.xn - 1)
            if f == "SPPE":
                k = k & (self.m1 >= 1) & (self.m2 >= 1)
            i = k.nonzero()[:, 0]
            r = rows[i]
            ref, has = ((bn[r, 0] - off) // step).clamp(0, nn - 1), bn[r, 0] != 0
            for _ in range(4):
                N[f][i] = bv[r, 0] + torch.where(has, bv[r, 1] * N[f][ref], 0.0)
