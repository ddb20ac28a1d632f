"""Timed workloads of the library's public entry points, with inputs, the work
each pass cannot do without, and the same results in plain 64-bit torch.

A case is a dict of plain values.  `kind` names the entry point:

  rhs      Context.rhs_regular_box      right-hand side of one regular box
  eb       Context.rhs_eb_box           right-hand side of one cut-cell box
  chem_rhs Context.rhs_chem_box         multispecies right-hand side of one box
  chem     Context.chem_advance_box     one implicit chemistry substep of a box
  level    Level.advance                whole RK steps of one level
  jet      Hierarchy.advance            coarse steps of a cut, refined hierarchy
  react    Reactor.advance              Strang steps of a reacting level
  mlp      Mlp.train_step               one training step of the surrogate network

The flow states are smooth waves of several lengths plus an oblique jump (box
calls) or a periodic blast (levels): sub- and supersonic parts, both sides of
every split, smooth and limited stencils.  The reacting states are H2/O2/N2
mixtures with products and radicals at 900-2400 K.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "opencfd-amr_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import ocfd  # noqa: E402
from ocfd import amr, cases, geometry, level, mlp, react  # noqa: E402

NG = 4
F64 = torch.float64
DEV = "cuda"


# ----------------------------------------------------------------- the cases
def listed():
    return [
        # per-box drop-in calls, as an application that keeps its own box loop makes them
        # the smallest: one 20 x 12 x 8 box (launch latency)
        dict(name="rhs_small", kind="rhs", nx=20, ny=12, nz=8, visc=True, fp32=False, flux=False, gravity=False),
        # an ordinary ragged box, viscous, face fluxes written for the caller's flux registers
        dict(name="rhs_visc_flux", kind="rhs", nx=61, ny=45, nz=37, visc=True, fp32=False, flux=True, gravity=False),
        # the mixed form of the same call on a box of the usual max_grid_size
        dict(name="rhs_f32_box", kind="rhs", nx=128, ny=96, nz=64, visc=False, fp32=True, flux=True, gravity=False),
        # a box cut by a cylinder, with the small-cell rescale
        dict(name="eb_box", kind="eb", nx=64, ny=48, nz=33, redistribute=True, flux=True),
        # multispecies box with mixture-averaged transport (a third of a 128 x 32 x 32 grid, ragged)
        dict(name="chem_rhs_visc", kind="chem_rhs", nx=43, ny=32, nz=29, visc=True, flux=True),
        # one implicit Li-Dryer substep of a 64^3 box
        dict(name="chem_box", kind="chem", nx=64, ny=64, nz=64, dt=1.25e-8),
        # whole levels, a step being one graph launch
        # 2D Sod tube as a thin slab, the reference's default Heun scheme
        dict(name="sod_rk2", kind="level", flow="sod", nx=512, ny=64, nz=4, box=512, steps=4, order=2, visc=False,
             fp32=False),
        # 3D periodic blast, plain FP64, SSP-RK3, boxes of 64
        dict(name="blast_f64", kind="level", flow="blast", nx=128, ny=128, nz=64, box=64, steps=1, order=3, visc=False,
             fp32=False),
        # ... and the mixed form at four times the size (larger than L2)
        dict(name="blast_f32", kind="level", flow="blast", nx=256, ny=256, nz=64, box=64, steps=2, order=3, visc=False,
             fp32=True),
        # Mach 2 jet past a cylinder, base grid + 2 refined levels, subcycled, plain FP64: two coarse
        # steps between two regrids
        dict(name="jet_amr", kind="jet", nx=64, ny=32, nz=32, levels=2, steps=2, fp32=False),
        # one Strang step of a reacting cube in the mixed form, chemistry binned by temperature
        dict(name="react_mixed", kind="react", n=64, box=32, visc=True, fp32=True, binned=True, substeps=4, dt=1e-8),
        # surrogate training, the usual batch
        dict(name="mlp_train", kind="mlp", batch=8192),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rhs", "rhs", "eb", "chem_rhs", "chem", "level", "level", "jet", "react", "mlp"])
    if kind == "rhs":
        nx, ny, nz = _log(rng, 8, 140), _log(rng, 4, 112), _log(rng, 4, 80)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, visc=rng.random() < 0.5, fp32=rng.random() < 0.5,
                    flux=rng.random() < 0.5, gravity=rng.random() < 0.2)
    if kind == "eb":
        return dict(kind=kind, nx=_log(rng, 12, 96), ny=_log(rng, 12, 72), nz=_log(rng, 4, 48),
                    redistribute=rng.random() < 0.5, flux=rng.random() < 0.5)
    if kind == "chem_rhs":
        return dict(kind=kind, nx=_log(rng, 8, 56), ny=_log(rng, 8, 40), nz=_log(rng, 4, 40),
                    visc=rng.random() < 0.6, flux=rng.random() < 0.5)
    if kind == "chem":
        return dict(kind=kind, nx=_log(rng, 8, 80), ny=_log(rng, 6, 72), nz=_log(rng, 4, 64),
                    dt=10.0 ** rng.uniform(-9.0, -7.5))
    if kind == "level":
        fp32 = rng.random() < 0.5
        if rng.random() < 0.35:
            return dict(kind=kind, flow="sod", nx=rng.randrange(96, 700), ny=rng.randrange(16, 80), nz=4,
                        box=rng.choice([64, 128, 512]), steps=rng.choice([1, 2, 4]), order=rng.choice([1, 2, 3]),
                        visc=rng.random() < 0.3, fp32=fp32)
        return dict(kind=kind, flow="blast", nx=_log(rng, 24, 192), ny=_log(rng, 24, 160), nz=_log(rng, 16, 72),
                    box=rng.choice([32, 48, 64]), steps=rng.choice([1, 2]), order=rng.choice([2, 3]),
                    visc=rng.random() < 0.3, fp32=fp32)
    if kind == "jet":
        return dict(kind=kind, nx=16 * rng.randrange(2, 5), ny=16 * rng.randrange(1, 3), nz=16 * rng.randrange(1, 3),
                    levels=rng.choice([1, 2]), steps=rng.choice([1, 2]), fp32=rng.random() < 0.5)
    if kind == "react":
        return dict(kind=kind, n=rng.randrange(20, 64), box=rng.choice([16, 24, 32]), visc=rng.random() < 0.6,
                    fp32=rng.random() < 0.5, binned=rng.random() < 0.5, substeps=rng.choice([1, 2, 4]),
                    dt=10.0 ** rng.uniform(-8.5, -7.5))
    return dict(kind=kind, batch=256 * rng.randrange(1, 33))


def work(case):
    k = case["kind"]
    if k in ("rhs", "eb", "chem_rhs", "chem"):
        n = (case["nx"], case["ny"], case["nz"])
        cells = n[0] * n[1] * n[2]
        faces = sum(cells // n[d] * (n[d] + 1) for d in range(3)) if case.get("flux") else 0
        grown = (n[0] + 6) * n[1] * n[2] + 6 * n[0] * n[2] + 6 * n[0] * n[1]  # the cells within 3 along x, y or z
        if k == "rhs":
            return {"bytes": 8.0 * 5 * (grown + cells + faces), "flops": cells * (2000.0 + 250.0 * case["visc"])}
        if k == "eb":
            cut = (n[0] + 4) * n[1] * n[2] + 4 * n[0] * n[2] + 4 * n[0] * n[1]
            return {"bytes": 8.0 * 5 * (cut + cells + faces) + 8.0 * 4.5 * cells, "flops": cells * 900.0}
        if k == "chem_rhs":
            return {"bytes": 8.0 * 14 * (grown + cells + faces), "flops": cells * (5500.0 + 2500.0 * case["visc"])}
        return {"bytes": 8.0 * (14 + 10) * cells, "flops": cells * 2500.0}
    if k == "level":
        cells = case["nx"] * case["ny"] * case["nz"]
        st = case["order"] * case["steps"]
        return {"bytes": 8.0 * 5 * cells * (2 + 3 * st), "flops": cells * st * (2050.0 + 250.0 * case["visc"])}
    if k == "jet":
        # level l refines about the shear layers and the body: a quarter to a third of the level below
        base = case["nx"] * case["ny"] * case["nz"]
        upd = base * sum((8 * 0.3) ** l * 2 ** l for l in range(case["levels"] + 1)) * case["steps"] * 3
        return {"bytes": upd * 120.0, "flops": upd * 1600.0}
    if k == "react":
        cells = case["n"] ** 3
        return {"bytes": cells * 8.0 * (14 * 2 * (2 + 2 * case["substeps"]) + 14 * 3 * 2),
                "flops": cells * (2 * case["substeps"] * 2500.0 + 2 * (5500.0 + 2500.0 * case["visc"]))}
    m = case["batch"]
    return {"bytes": 4.0 * (22 * m + 6 * mlp.WTOT), "flops": 6.0 * mlp.WTOT * m}


# -------------------------------------------------------------------- inputs
_CTX = []


def _ctx():
    """The program's one context (tables, scratch pool); a program keeps it for its whole run."""
    if not _CTX:
        _CTX.append(ocfd.Context())
    return _CTX[0]


def _coords(shape, off=0):
    return torch.meshgrid(*[torch.arange(s, dtype=F64, device=DEV) + (0.5 - off) for s in shape], indexing="ij")


def _waves(rng, zyx, period=None, nmode=5, shortest=10.0):
    """A sum of plane waves in [-1, 1]: lengths between the box and `shortest` cells, or integer
    wave numbers of the period (x, y, z)."""
    z, y, x = zyx
    out = torch.zeros_like(x)
    amp = 0.0
    for m in range(nmode):
        if period is None:
            kk = 2 * math.pi / math.exp(rng.uniform(math.log(shortest), math.log(16 * shortest)))
            d = rng.standard_normal(3)
            d *= kk / np.linalg.norm(d)
        else:
            d = [2 * math.pi / p * rng.integers(-min(4, p // 8) - 1, min(4, p // 8) + 2) for p in period]
        a = rng.uniform(0.3, 1.0)
        amp += a
        out += a * torch.sin(d[0] * x + d[1] * y + d[2] * z + rng.uniform(0, 2 * math.pi))
    return out / amp


def _ideal_box(rng, n):
    """Conserved state (5, nz+8, ny+8, nx+8): waves and an oblique jump of 8 : 1 in density, 10 : 1 in pressure."""
    zyx = _coords((n[2] + 8, n[1] + 8, n[0] + 8), NG)
    z, y, x = zyx
    rho = 1.0 + 0.35 * _waves(rng, zyx)
    p = 1.0 + 0.4 * _waves(rng, zyx)
    ph = rng.uniform(-0.6, 0.6, 2)
    cut = (x - 0.5 * n[0]) + ph[0] * (y - 0.5 * n[1]) + ph[1] * (z - 0.5 * n[2]) > 0
    rho = torch.where(cut, 0.125 * rho, rho)
    p = torch.where(cut, 0.1 * p, p)
    c = torch.sqrt(1.4 * p / rho)
    v = [c * (rng.uniform(-0.8, 0.8) + 1.1 * _waves(rng, zyx)) for _ in range(3)]
    return torch.stack([rho] + [rho * w for w in v] + [p / 0.4 + 0.5 * rho * sum(w * w for w in v)]).contiguous()


def _blast(rng, n, dx):
    """Periodic blast with waves in its surroundings: valid cells (5, nz, ny, nx)."""
    zyx = _coords((n[2], n[1], n[0]))
    z, y, x = zyx
    c = [rng.uniform(0.3, 0.7) * m for m in n]
    r2 = 0.0
    for q, c0, m in ((x, c[0], n[0]), (y, c[1], n[1]), (z, c[2], n[2])):
        d = torch.abs(q - c0)
        d = torch.minimum(d, m - d)
        r2 = r2 + d * d
    inside = r2 < (0.3 * min(n)) ** 2
    rho = torch.where(inside, 1.0, 0.125) * (1.0 + 0.1 * _waves(rng, zyx, n))
    p = torch.where(inside, 1.0, 0.1) * (1.0 + 0.1 * _waves(rng, zyx, n))
    v = [0.2 * _waves(rng, zyx, n) for _ in range(3)]
    return torch.stack([rho] + [rho * w for w in v] + [p / 0.4 + 0.5 * rho * sum(w * w for w in v)]).contiguous()


def _sod(rng, n):
    """Sod's states with a slight random ripple of the diaphragm and the pressure."""
    zyx = _coords((n[2], n[1], n[0]))
    z, y, x = zyx
    left = x + 2.0 * torch.sin(2 * math.pi * y / n[1] + rng.uniform(0, 6)) < 0.5 * n[0]
    rho = torch.where(left, 1.0, 0.125)
    p = torch.where(left, 1.0, 0.1) * (1.0 + 0.02 * _waves(rng, zyx))
    o = torch.zeros_like(x)
    return torch.stack([rho + o, o, o, o, p / 0.4]).contiguous()


def _reacting(rng, zyx, period=None):
    """(flow, partial densities) of H2/O2/N2 with products and radicals, 900-2400 K, 0.7-1.5 atm, moving."""
    T = 1650.0 + 750.0 * _waves(rng, zyx, period)
    p = 101325.0 * (1.1 + 0.4 * _waves(rng, zyx, period))
    u = [150.0 * _waves(rng, zyx, period) for _ in range(3)]
    X = [None] * 9
    for n, (lo, hi) in enumerate([(0.1, 0.3), (0.05, 0.16), (0.01, 0.2)] + [(1e-5, 8e-3)] * 3 + [(1e-7, 2e-4)] * 2):
        s = 0.5 + 0.5 * _waves(rng, zyx, period)
        X[n] = lo * (hi / lo) ** s if n >= 3 else lo + (hi - lo) * s
    X[8] = 1.0 - sum(X[:8])
    X = torch.stack(X)
    m = _Mech(_ctx().parm)
    mw = m.mw[:, None, None, None]
    W = (X * mw).sum(0)
    rho = p * W / (m.Ru * T)
    R = rho * X * mw / W
    E = (R / mw * m.u_rt(T)).sum(0) * m.Ru * T + 0.5 * rho * sum(w * w for w in u)
    return torch.stack([rho] + [rho * w for w in u] + [E]).contiguous(), R.contiguous()


def _flux_arrays(nc, n):
    return [torch.zeros((nc, n[2] + (d == 2), n[1] + (d == 1), n[0] + (d == 0)), dtype=F64, device=DEV)
            for d in range(3)]


def _flags(case):
    return ((ocfd.VISC if case.get("visc") else 0) | (ocfd.FLUX_FP32 if case.get("fp32") else 0)
            | (ocfd.GRAVITY if case.get("gravity") else 0) | (ocfd.REDISTRIBUTE if case.get("redistribute") else 0))


def _pack(boxes, U):
    return torch.cat([U[:, lo[2]:hi[2] + 1, lo[1]:hi[1] + 1, lo[0]:hi[0] + 1].reshape(-1) for lo, hi in boxes])


def _dx(case):
    """Cell sizes of a box call (slightly unequal, as a stretched domain has them)."""
    return (1.0 / 64, 1.1 / 64, 0.9 / 64)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    k = case["kind"]
    s = {"case": case, "ctx": _ctx(), "flags": _flags(case)}
    if k in ("rhs", "eb", "chem_rhs", "chem"):
        n = (case["nx"], case["ny"], case["nz"])
        s.update(lo=(0, 0, 0), hi=tuple(m - 1 for m in n))
        if k in ("rhs", "eb"):
            s["S"] = _ideal_box(rng, n)
            s["dS"] = torch.zeros((5,) + n[::-1], dtype=F64, device=DEV)
            s["flux"] = _flux_arrays(5, n) if case["flux"] else None
            s["dxinv"] = [1.0 / d for d in (_dx(case) if k == "rhs" else (1.0 / 64,) * 3)]
            if k == "eb":
                r = rng.uniform(0.2, 0.35) * min(n[0], n[1])
                g = geometry.box_geometry(geometry.cylinder_phi(rng.uniform(0.35, 0.65) * n[0],
                                                                rng.uniform(0.35, 0.65) * n[1], r),
                                          (0, 0, 0), n, (1.0, 1.0, 1.0))
                s["geom"] = {q: torch.from_numpy(np.ascontiguousarray(g[q]).view(np.int32) if q == "flag"
                                                 else np.ascontiguousarray(g[q])).to(DEV)
                             for q in ("flag", "vfrac", "apx", "apy", "apz")}
        elif k == "chem_rhs":
            s["S"], s["R"] = _reacting(rng, _coords(tuple(m + 8 for m in n[::-1]), NG))
            s["dS"] = torch.zeros((5,) + n[::-1], dtype=F64, device=DEV)
            s["dR"] = torch.zeros((9,) + n[::-1], dtype=F64, device=DEV)
            s["flux"] = (_flux_arrays(5, n), _flux_arrays(9, n)) if case["flux"] else (None, None)
            s["dxinv"] = [1.0 / (1e-2 * d) for d in _dx(case)]
        else:
            s["S0"], s["R0"] = _reacting(rng, _coords(n[::-1]))
            s["S"], s["R"] = torch.empty_like(s["S0"]), torch.empty_like(s["R0"])
        return s
    if k == "level":
        n = (case["nx"], case["ny"], case["nz"])
        boxes = level.chop_domain(n, case["box"])
        dx = 1.0 / n[0]
        sod = case["flow"] == "sod"
        L = level.Level(s["ctx"], boxes, tuple(m - 1 for m in n), (2, 4, 4) if sod else (0, 0, 0),
                        (2, 4, 4) if sod else (0, 0, 0), (dx, dx, dx))
        L.set_time_integration(case["order"])
        s["U"] = _sod(rng, n) if sod else _blast(rng, n, dx)
        s.update(level=L, boxes=boxes, flat=_pack(boxes, s["U"]), dx=dx)
        s["out"] = torch.empty_like(s["flat"])
        return s
    if k == "jet":
        c = cases.jet_eb_amr(case["nx"], case["ny"], case["nz"], max_level=case["levels"])
        H = amr.Hierarchy(s["ctx"], level.chop_domain(c["n"], 64), c["n"], c["lo_bc"], c["hi_bc"], c["dx"],
                          bc_case=c["bc_case"], case_params=c["case_params"], max_level=c["max_level"],
                          blocking_factor=c["blocking_factor"], max_grid_size=c["max_grid_size"],
                          n_error_buf=c["n_error_buf"], regrid_int=0, refine_dengrad=c["refine_dengrad"])
        H.set_eb(level.eb_desc(**c["eb"]))
        ext = tuple(m * d for m, d in zip(c["n"], c["dx"]))
        fab = lambda sd: lambda lo, hi, d: cases.jet_fab(lo, hi, d, L=ext, params=c["case_params"], seed=sd)  # noqa: E731
        # the flow meets the body: the grids that a regrid gives it after a few steps
        H.build(lambda lev, lo, hi, d: fab(c["seed"])(lo, hi, d))
        H.advance(4, 0.5)
        H.regrid(0)
        # on these grids, the jet with this seed's shear-layer perturbation, a few steps on
        for l in range(H.nlevels()):
            L = H.level(l)
            H.copy_in(l, L.pack_fabs(lambda lo, hi: fab(seed)(lo, hi, H.dx(l))))
            torch.cuda.synchronize()
        H.average_down()
        H.set_time(0.0)
        H.advance(2, 0.5)
        s["H"] = H
        s["in"] = [H.copy_valid_out(l, torch.empty(H.valid_elems(l), dtype=F64, device=DEV))
                   for l in range(H.nlevels())]
        s["out"] = [torch.empty_like(t) for t in s["in"]]
        return s
    if k == "react":
        n = (case["n"],) * 3
        dx = 0.01 / 128
        boxes = level.chop_domain(n, case["box"])
        U, R = _reacting(rng, _coords(n[::-1]), n)
        s["U"] = torch.cat([U, R])
        s["reactor"] = react.Reactor(s["ctx"], boxes, tuple(m - 1 for m in n), (dx, dx, dx), dt=case["dt"], rk_order=2,
                                     chem_substeps=case["substeps"], visc=case["visc"], binned=case["binned"],
                                     flux_fp32=case["fp32"])
        s.update(boxes=boxes, flat=_pack(boxes, s["U"]), dx=dx)
        s["out"] = torch.empty_like(s["flat"])
        return s
    net = mlp.Mlp(s["ctx"], case["batch"], int(rng.integers(1, 1 << 30)))
    g = torch.Generator(device="cpu").manual_seed(int(rng.integers(1, 1 << 30)))
    s["net"] = net
    s["X"] = torch.randn((case["batch"], 12), generator=g).to(DEV)
    s["T"] = torch.tanh(s["X"][:, :10] + 0.3 * s["X"][:, 2:12] ** 2).contiguous()
    return s


# ----------------------------------------------------------------- one pass
def run(s):
    case, ctx, k = s["case"], s["ctx"], s["case"]["kind"]
    if k == "rhs":
        ctx.rhs_regular_box(s["S"], s["dS"], s["lo"], s["hi"], s["dxinv"], s["flags"], flux=s["flux"])
        return [s["dS"]] + (s["flux"] or [])
    if k == "eb":
        ctx.rhs_eb_box(s["S"], s["dS"], s["geom"], s["lo"], s["hi"], s["dxinv"], s["flags"], flux=s["flux"])
        return [s["dS"]] + (s["flux"] or [])
    if k == "chem_rhs":
        ctx.rhs_chem_box(s["S"], s["R"], s["dS"], s["dR"], s["lo"], s["hi"], s["dxinv"], s["flags"], flux=s["flux"][0],
                         flux_spec=s["flux"][1])
        return [s["dS"], s["dR"]] + (s["flux"][0] or []) + (s["flux"][1] or [])
    if k == "chem":
        # the substep works in place on the state that the flow step left
        s["S"].copy_(s["S0"])
        s["R"].copy_(s["R0"])
        ctx.chem_advance_box(s["S"], s["R"], s["lo"], s["hi"], case["dt"])
        return [s["S"], s["R"]]
    if k == "level":
        s["level"].copy_valid_in(s["flat"])
        s["level"].advance(case["steps"], 0.5, s["flags"])
        s["level"].copy_valid_out(s["out"])
        return s["out"]
    if k == "jet":
        H = s["H"]
        for l, t in enumerate(s["in"]):
            H.copy_valid_in(l, t)
        H.set_time(0.0)
        H.advance(case["steps"], 0.5, s["flags"])
        return [H.copy_valid_out(l, t) for l, t in enumerate(s["out"])]
    if k == "react":
        L = s["reactor"].level
        L.copy_valid_in(s["flat"])
        s["reactor"].advance(1)
        L.copy_valid_out(s["out"])
        return s["out"]
    loss, gW, gb = s["net"].train_step(s["X"], s["T"], lr=1e-3, update=True, grads=True)
    return {"loss": loss, "gW": gW, "gb": gb}


# ------------------------------------------- the same results in plain torch
def _shift(a, d, o, n, g, w=0):
    """Cells o.. (w more than n along d) of `a` along direction d (0 = x), the valid range in the others;
    a is grown by g."""
    ax = a.dim() - 1 - d
    idx = [slice(None)] * (a.dim() - 3) + [slice(g, g + n[e]) for e in (2, 1, 0)]
    idx[ax] = slice(g + o, g + o + n[d] + w)
    return a[tuple(idx)]


def _weno5(v):
    """WENO-Z value at the face after v[2] of the stencil v[0..4] (ordered towards the face)."""
    a, b, c, d, e = v
    b1 = 13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2
    b2 = 13 / 12 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2
    b3 = 13 / 12 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2
    t = (b1 - b3).abs()
    w = [g * (1 + (t / (1e-6 + q)) ** 2) for g, q in ((1.0, b1), (6.0, b2), (3.0, b3))]
    p = [2 * a - 7 * b + 11 * c, -b + 5 * c + 2 * d, 2 * c + 5 * d - e]
    return (w[0] * p[0] + w[1] * p[1] + w[2] * p[2]) / (6 * (w[0] + w[1] + w[2]))


def _split(q, d, g):
    """Steger-Warming parts [f+, f-] of (rho, u, v, w, c) along d, and the species split factors."""
    rho, c = q["rho"], q["c"]
    un = q["v"][d]
    t1, t2, t3 = 1 / (2 * g), 2 * (g - 1), (3 - g) / (2 * (g - 1))
    lam = [un, un - c, un + c]
    kin = sum(v * v for v in q["v"])
    h = [0.5 * (kin - un * un + l * l) for l in lam[1:]]
    out, fac = [], []
    for sgn in (1, -1):
        e1, e2, e3 = [0.5 * (l + sgn * l.abs()) for l in lam]
        s = t2 * e1 + e2 + e3
        f = [rho * t1 * s]
        for m in range(3):
            f.append(rho * t1 * (t2 * e1 * un + e2 * lam[1] + e3 * lam[2]) if m == d else rho * t1 * s * q["v"][m])
        f.append(rho * t1 * (e1 * (g - 1) * kin + e2 * h[0] + e3 * h[1] + t3 * c * c * (e2 + e3)))
        out.append(torch.stack(f))
        fac.append(t1 * s)
    return out, fac


def _faces_weno(fp, fm, d, n):
    """WENO-Z face fluxes (n_d + 1 along d) of split fluxes over a grown array."""
    plus = _weno5([_shift(fp, d, o, n, NG, 1) for o in (-3, -2, -1, 0, 1)])
    minus = _weno5([_shift(fm, d, o, n, NG, 1) for o in (2, 1, 0, -1, -2)])
    return plus + minus


def _ideal_prims(U, P):
    rho = U[0].clamp_min(P.smallr)
    v = [U[m] / rho for m in (1, 2, 3)]
    p = ((P.eos_gamma - 1) * (U[4] - 0.5 * rho * sum(w * w for w in v))).clamp_min(P.smallp)
    T = p / (rho * P.Rg)
    return {"rho": rho, "v": v, "p": p, "T": T, "c": torch.sqrt(P.eos_gamma * P.Rg * T)}


def _at_face(a, d, n):
    """(low cell, high cell) of every d-face."""
    return _shift(a, d, -1, n, NG, 1), _shift(a, d, 0, n, NG, 1)


def _tau(q, d, n, dxinv, mu):
    """Viscous stresses tau[0..2] on the d-faces."""
    g = {}
    for m in range(3):
        l, h = _at_face(q["v"][m], d, n)
        g[m, d] = (h - l) * dxinv[d]
    for t in range(3):
        if t == d:
            continue
        for m in {d, t}:
            a = q["v"][m]
            hi, lo = torch.roll(a, -1, a.dim() - 1 - t), torch.roll(a, 1, a.dim() - 1 - t)
            (l1, h1), (l0, h0) = _at_face(hi, d, n), _at_face(lo, d, n)
            g[m, t] = (h1 + l1 - h0 - l0) * (0.25 * dxinv[t])
    div = g[0, 0] + g[1, 1] + g[2, 2]
    return [mu * (2 * g[d, d] - 2 / 3 * div) if m == d else mu * (g[m, d] + g[d, m]) for m in range(3)]


def _regular_rhs(S, n, dxinv, P, visc, gravity):
    """(dSdt, face fluxes) of one regular ideal-gas box, S grown by 4."""
    q = _ideal_prims(S, P)
    dS, fl = 0.0, []
    for d in range(3):
        (fp, fm), _ = _split(q, d, P.eos_gamma)
        f = _faces_weno(fp, fm, d, n)
        if visc:
            mu = P.C_s * q["T"] * torch.sqrt(q["T"]) / (q["T"] + P.T_s)
            ml, mh = _at_face(mu, d, n)
            tau = _tau(q, d, n, dxinv, 0.5 * (ml + mh))
            Tl, Th = _at_face(q["T"], d, n)
            w = 0.0
            for m in range(3):
                f[1 + m] -= tau[m]
                l, h = _at_face(q["v"][m], d, n)
                w = w + (l + h) * tau[m]
            f[4] -= 0.5 * (w + (ml + mh) * P.kOverMu * (Th - Tl) * dxinv[d])
        fl.append(f)
        ax = 3 - d
        dS = dS - dxinv[d] * torch.diff(f, dim=ax)
    if gravity:
        c = S[:, NG:-NG, NG:-NG, NG:-NG]
        dS[3] += -9.8 * c[0]
        dS[4] += -9.8 * c[3]
    return dS, fl


def _grow_periodic(U):
    for ax in (1, 2, 3):
        n = U.shape[ax]
        U = torch.index_select(U, ax, torch.arange(-NG, n + NG, device=U.device) % n)
    return U


def _grow_sod(U):
    """x: zeroth-order outflow; y, z: slip walls (mirror, normal momentum negated)."""
    n = U.shape[3]
    U = torch.index_select(U, 3, torch.arange(-NG, n + NG, device=U.device).clamp(0, n - 1))
    for ax, m in ((2, 2), (1, 3)):
        n = U.shape[ax]
        i = torch.arange(-NG, n + NG, device=U.device)
        j = torch.where(i < 0, -1 - i, torch.where(i >= n, 2 * n - 1 - i, i))
        out = (i < 0) | (i >= n)
        U = torch.index_select(U, ax, j)
        shape = [1, 1, 1]
        shape[ax - 1] = -1
        U[m] = torch.where(out.reshape(shape), -U[m], U[m])
    return U


def _level_exact(s):
    case, P, dx = s["case"], s["ctx"].parm, s["dx"]
    n = (case["nx"], case["ny"], case["nz"])
    grow = _grow_sod if case["flow"] == "sod" else _grow_periodic
    ab = {1: [(0, 1)], 2: [(0, 1), (0.5, 0.5)], 3: [(0, 1), (0.75, 0.25), (1 / 3, 2 / 3)]}[case["order"]]
    U, prev = s["U"], None
    for _ in range(case["steps"]):
        q = _ideal_prims(U, P)
        dt = 0.5 * min(float((dx / (v.abs() + q["c"])).min()) for v in q["v"])
        dt = dt if prev is None else min(dt, 1.1 * prev)
        prev = dt
        V = U
        for a, b in ab:
            V = a * U + b * (V + dt * _regular_rhs(grow(V), n, [1 / dx] * 3, P, case["visc"], False)[0])
        U = V
    return _pack(s["boxes"], U)


# ---- cut-cell box
def _conn(f, i, j, k):
    p = 4 + (i + 1) + 3 * (j + 1) + 9 * (k + 1)
    return ((f >> p) & 1).bool() if 0 <= p < 32 else torch.zeros_like(f, dtype=torch.bool)


def _minmod(a, b):
    return torch.where(a * b > 0, torch.where(a.abs() > b.abs(), b, a), torch.zeros_like(a))


def _van_leer(l, r, d, g, P):
    def side(q, sg):
        rho, p, c, v = q["rho"], q["p"].clamp_min(P.smallp), q["c"], q["v"]
        un = v[d]
        M = un / c
        kin = sum(w * w for w in v)
        full = [rho * un] + [rho * un * v[m] + (p if m == d else 0.0) for m in range(3)]
        full.append(un * (g / (g - 1) * p + 0.5 * rho * kin))
        m0 = sg * rho * c * 0.25 * (M + sg) ** 2
        sub = [m0] + [m0 * ((-un + sg * 2 * c) / g + v[m] if m == d else v[m]) for m in range(3)]
        sub.append(m0 * (((g - 1) * un + sg * 2 * c) ** 2 / (2 * (g * g - 1)) + 0.5 * (kin - un * un)))
        zero = torch.zeros_like(rho)
        return torch.stack([torch.where(sg * M >= 1, a, torch.where(M.abs() < 1, b, zero)) for a, b in zip(full, sub)])

    return side(l, 1) + side(r, -1)


def _eb_exact(s):
    case, P, G = s["case"], s["ctx"].parm, s["geom"]
    n = (case["nx"], case["ny"], case["nz"])
    q = _ideal_prims(s["S"], P)
    flag = G["flag"][0].long() & 0xffffffff
    fl = []
    for d in range(3):
        f = _shift(flag, d, 0, n, NG, 1)
        e = [int(d == m) for m in range(3)]
        lo, hi, lo2 = _conn(f, *[-x for x in e]), _conn(f, *e), _conn(f, *[-2 * x for x in e])

        def rec(a):
            m2, m1, c0, p1 = [_shift(a, d, o, n, NG, 1) for o in (-2, -1, 0, 1)]
            return (torch.where(lo & lo2, m1 + 0.5 * _minmod(c0 - m1, m1 - m2), m1),
                    torch.where(lo & hi, c0 - 0.5 * _minmod(p1 - c0, c0 - m1), c0))

        pair = {m: rec(q[m]) for m in ("rho", "p", "c")}
        vel = [rec(v) for v in q["v"]]
        l, r = [dict({m: pair[m][i] for m in pair}, v=[v[i] for v in vel]) for i in (0, 1)]
        fl.append(_van_leer(l, r, d, P.eos_gamma, P))
    inner = (slice(NG, -NG),) * 3
    fc, vf = flag[inner], G["vfrac"][0][inner]
    reg = sum(s["dxinv"][d] * torch.diff(fl[d], dim=3 - d) for d in range(3))
    tmp = s["dxinv"][0] / vf
    cut, wall = 0.0, []
    for d, a in enumerate(("apx", "apy", "apz")):
        cut = cut + torch.diff(G[a][0] * fl[d], dim=3 - d)
        wall.append(-torch.diff(G[a][0], dim=2 - d) * q["p"][inner])
    for d in range(3):
        cut[1 + d] += wall[d]
    out = -torch.where((fc & 3) == 3, torch.zeros_like(reg), torch.where((fc & 3) == 0, reg, tmp * cut))
    if case["redistribute"]:
        out = torch.where((vf < 0.5) & (vf > 0), vf * out, out)
    return [out] + (fl if case["flux"] else [])


# ---- Li-Dryer H2/O2
class _Mech:
    """The mechanism data of a Parm (NASA-7 fits, transport fits) as tensors."""
    SP = ("H2", "O2", "H2O", "H", "O", "OH", "HO2", "H2O2", "N2")

    def __init__(self, P):
        def arr(name, *shape):
            p = ctypes.cast(getattr(P, name), ctypes.POINTER(ctypes.c_double))
            return torch.tensor(np.ctypeslib.as_array(p, shape).copy(), dtype=F64, device=DEV)
        self.mw = arr("mw", 9)
        self.lo = torch.stack([arr(x + "_lo", 7) for x in self.SP])
        self.hi = torch.stack([arr(x + "_hi", 7) for x in self.SP])
        self.HP, self.A0 = arr("HP", 9), arr("A0", 9)
        self.visc, self.cond = arr("visccoeff", 9, 5), arr("conductcoeff", 9, 5)
        self.diff = arr("diffcoeff", 45, 5)
        self.Ru, self.Patm, self.P = P.Ru, P.Patm, P

    def coef(self, T):
        """NASA-7 rows a[k] (9, ...) at T, and h(0 K) / R of the high fit relative to the low one."""
        s = (9,) + (1,) * T.dim()
        low = (T < 1000)[None]
        a = [torch.where(low, self.lo[:, k].reshape(s), self.hi[:, k].reshape(s)) for k in range(7)]
        return a, a[5] - self.lo[:, 5].reshape(s)

    def h_poly(self, T):
        a, dh = self.coef(T)
        return a[0] * T + a[1] / 2 * T ** 2 + a[2] / 3 * T ** 3 + a[3] / 4 * T ** 4 + a[4] / 5 * T ** 5 + dh

    def u_rt(self, T):
        """e_n / (R T)."""
        return self.h_poly(T) / T - 1.0

    def energy(self, T, R):
        return (R / self.col(T) * self.u_rt(T)).sum(0) * self.Ru * T

    def cv(self, T, R):
        a, _ = self.coef(T)
        cp = a[0] + a[1] * T + a[2] * T ** 2 + a[3] * T ** 3 + a[4] * T ** 4
        return ((cp - 1.0) * R / self.col(T)).sum(0) * self.Ru

    def col(self, T):
        return self.mw.reshape((9,) + (1,) * T.dim())

    def temperature(self, e, R):
        """T of the internal energy e: Newton steps of at most 100 K from the linear estimate, ended where
        a step is below 1e-7 K; linear outside 250-3500 K."""
        lo, hi = torch.full_like(e, 250.0), torch.full_like(e, 3500.0)
        elo, ehi = self.energy(lo, R), self.energy(hi, R)
        T = e / (self.A0.reshape((9,) + (1,) * e.dim()) * self.Ru / self.col(e) * R).sum(0)
        T = torch.where((T < 250) | (T > 3500), 250 + 3250 / (ehi - elo) * (e - elo), T)
        done = torch.zeros_like(e, dtype=torch.bool)
        for _ in range(200):
            dt = ((e - self.energy(T, R)) / self.cv(T, R)).clamp(-100.0, 100.0)
            done = done | (dt.abs() < 1e-7) | (T + dt == T)
            if bool(done.all()):
                break
            T = torch.where(done, T, T + dt)
        T = torch.where(e < elo, 250 - (elo - e) / self.cv(lo, R), T)
        return torch.where(e > ehi, 3500 - (ehi - e) / self.cv(hi, R), T)


# A, b, Ta of the forward rate k = A T^b exp(-Ta / T) [cm3, mol, s], reactants, products, third body
_RXN = [
    ((3.55e15, -0.41, 8353.444256079512),), (3, 1), (4, 5), None,
    ((50800.0, 2.67, 3165.2508657072367),), (4, 0), (3, 5), None,
    ((2.16e8, 1.51, 1726.0429999007667),), (0, 5), (2, 3), None,
    ((2.97e6, 2.02, 6743.141748883461),), (4, 2), (5, 5), None,
    ((4.58e19, -1.4, 52526.05490660117),), (0,), (3, 3), "M",
    ((6.16e15, -0.5, 0.0),), (4, 4), (1,), "M",
    ((4.71e18, -1.0, 0.0),), (4, 3), (5,), "M",
    ((3.8e22, -2.0, 0.0),), (3, 5), (2,), "M",
    ((1.48e12, 0.6, 0.0),), (3, 1), (6,), (6.37e20, -1.72, 261.6741574193582, 0.8),
    ((1.66e13, 0.0, 412.64001746898793),), (6, 3), (0, 1), None,
    ((7.08e13, 0.0, 150.96586004962973),), (6, 3), (5, 5), None,
    ((3.25e13, 0.0, 0.0),), (6, 4), (1, 5), None,
    ((2.89e13, 0.0, -251.60976674938289),), (6, 5), (2, 1), None,
    ((4.2e14, 0.0, 6028.570011315214), (1.3e11, 0.0, -820.2478396029883)), (6, 6), (7, 1), None,
    ((2.95e14, 0.0, 24355.825421340265),), (7,), (5, 5), (1.20e17, 0.0, 22846.166820843966, 0.5),
    ((2.41e13, 0.0, 1997.7815479901),), (7, 3), (2, 5), None,
    ((4.82e13, 0.0, 4000.595291315188),), (7, 3), (6, 0), None,
    ((9.55e6, 2.0, 1997.7815479901),), (7, 4), (5, 6), None,
    ((1.0e12, 0.0, 0.0), (5.8e14, 0.0, 4810.778740248201)), (7, 5), (6, 2), None,
]


def _rates(m, c, T):
    """Production rates (9, ...) and their derivatives A[l][n] at concentrations c [mol/cm3]."""
    a, _ = m.coef(T)
    lnT = torch.log(T)
    g = a[0] * (1 - lnT) - a[1] / 2 * T - a[2] / 6 * T ** 2 - a[3] / 12 * T ** 3 - a[4] / 20 * T ** 4 + a[5] / T - a[6]
    RsT = m.Ru / m.Patm * 1e6 * T
    mix = c.sum(0)
    M = mix + 1.5 * c[0] + 11 * c[2]
    w = torch.zeros_like(c)
    A = torch.zeros((9,) + tuple(c.shape), dtype=F64, device=c.device)
    arr = lambda k: k[0] * torch.exp(k[1] * lnT - k[2] / T)  # noqa: E731
    for r in range(0, len(_RXN), 4):
        ks, re, pr, third = _RXN[r:r + 4]
        kf = sum(arr(k) for k in ks)
        if third == "M":
            kf = kf * M
        elif third is not None:
            al = mix + c[0] + 10 * c[2] - 0.22 * c[1] if third[3] == 0.8 else M
            red = al / kf * arr(third[:3])
            lf = math.log10(third[3])
            x = -0.4 - 0.67 * lf + torch.log10(red)
            x = x / (0.75 - 1.27 * lf - 0.14 * x)
            kf = kf * red / (1 + red) * 10.0 ** (lf / (1 + x * x))
        iK = torch.exp(sum(g[i] for i in pr) - sum(g[i] for i in re)) * RsT ** (len(pr) - len(re))
        wf, wr = kf, kf * iK
        for i in re:
            wf = wf * c[i]
        for i in pr:
            wr = wr * c[i]
        sp = sorted(set(re + pr))
        nu = {i: pr.count(i) - re.count(i) for i in sp}
        for i in sp:
            w[i] += (wf - wr) * nu[i]
            dn = (re.count(i) * wf - pr.count(i) * wr) / (c[i] + 1e-20)
            for l in sp:
                A[l, i] += dn * nu[l]
    return w, A


def _chem_step(m, U, R, dt):
    """One linearised backward-Euler substep; U (5, ...) and R (9, ...) are not changed."""
    rho = U[0].clamp_min(m.P.smallr)
    ei = U[4] - 0.5 * (U[1] ** 2 + U[2] ** 2 + U[3] ** 2) / rho
    T = m.temperature(ei, R)
    col = m.col(T)
    w, A = _rates(m, R / col * 1e-6, T)
    J = -A * dt * (col[:, None] / col[None, :])
    J = J.reshape(9, 9, -1).permute(2, 0, 1) + torch.eye(9, dtype=F64, device=J.device)
    b = (w * col * 1e6 * dt).reshape(9, -1).T
    d = torch.linalg.solve(J, b[:, :, None])[:, :, 0].T.reshape(R.shape)
    V = U.clone()
    V[4] += (-m.HP.reshape(col.shape) * m.Ru / col * d).sum(0)
    return V, (R + d).clamp_min(0.0)


def _mix_transport(m, T, p, R, rho):
    """(mu, lambda, D[9]): Wilke viscosity, averaged conductivity, mixture-averaged diffusivities."""
    col = m.col(T)
    X = R / rho / col
    X = X / X.sum(0)
    lnT = torch.log(T)
    poly = torch.stack([lnT ** k for k in range(5)])
    fit = lambda c: torch.tensordot(c, poly, 1)  # noqa: E731
    sm = T ** 0.25 * fit(m.visc)
    lam = torch.sqrt(T) * fit(m.cond)
    mui = sm * sm
    mu = 0.0
    for k in range(9):
        den = 0.0
        for j in range(9):
            r = float(m.mw[j] / m.mw[k])
            den = den + X[j] * (1 + sm[k] / sm[j] * r ** 0.25) ** 2 / math.sqrt(8 + 8 / r) if j != k else den + X[j]
        mu = mu + X[k] * mui[k] / den
    lm = 0.5 * ((X * lam).sum(0) + 1.0 / (X / lam).sum(0))
    bd = T * torch.sqrt(T) * fit(m.diff)
    W = (X * col).sum(0)
    D = []
    for k in range(9):
        s1, s2 = 0.0, 0.0
        for j in range(9):
            if j == k:
                continue
            lo, hi = min(j, k), max(j, k)
            x = X[j] / bd[lo * 9 - lo * (lo - 1) // 2 + hi - lo]
            s1, s2 = s1 + x, s2 + x * m.mw[j]
        D.append(1.0 / (s1 * p + s2 * p * X[k] / (W - m.mw[k] * X[k])))
    return mu, lm, torch.stack(D)


def _chem_rhs(m, S, R, n, dxinv, visc):
    """(dS, dR, flow fluxes, species fluxes) of one regular multispecies box grown by 4."""
    P = m.P
    rho = S[0].clamp_min(P.smallr)
    v = [S[k] / rho for k in (1, 2, 3)]
    ei = S[4] - 0.5 * rho * sum(w * w for w in v)
    T = m.temperature(ei, R)
    p = (R / m.col(T)).sum(0) * m.Ru * T
    g = p / ei + 1.0
    q = {"rho": rho, "v": v, "T": T, "p": p, "c": torch.sqrt(g * p / rho)}
    if visc:
        mu, lam, D = _mix_transport(m, T, p, R, rho)
    dS, dR, fl, fs = 0.0, 0.0, [], []
    for d in range(3):
        (fp, fm), (ap, am) = _split(q, d, g)
        f, h = _faces_weno(fp, fm, d, n), _faces_weno(R * ap, R * am, d, n)
        if visc:
            Yl, Yh = _at_face(R / rho, d, n)
            face = lambda a: 0.5 * sum(_at_face(a, d, n))  # noqa: E731
            fd = face(rho) * face(D) * (Yl - Yh) * dxinv[d]
            h = h + fd
            hflux = (fd * m.h_poly(face(T))).sum(0)
            tau = _tau(q, d, n, dxinv, face(mu))
            Tl, Th = _at_face(T, d, n)
            for k in range(3):
                f[1 + k] -= tau[k]
            f[4] -= sum(face(v[k]) * tau[k] for k in range(3)) + face(lam) * (Th - Tl) * dxinv[d] + hflux
        fl.append(f)
        fs.append(h)
        dS = dS - dxinv[d] * torch.diff(f, dim=3 - d)
        dR = dR - dxinv[d] * torch.diff(h, dim=3 - d)
    return dS, dR, fl, fs


def _react_exact(s):
    case, m = s["case"], _Mech(s["ctx"].parm)
    n = (case["n"],) * 3
    dt, sub = case["dt"], case["substeps"]
    U, R = s["U"][:5], s["U"][5:]
    for half in range(2):
        for _ in range(sub):
            U, R = _chem_step(m, U, R, 0.5 * dt / sub)
        if half == 0:
            V0 = torch.cat([U, R])
            V = V0
            for a, b in ((0.0, 1.0), (0.5, 0.5)):
                G = _grow_periodic(V)
                dS, dR, _, _ = _chem_rhs(m, G[:5], G[5:], n, [1 / s["dx"]] * 3, case["visc"])
                V = a * V0 + b * (V + dt * torch.cat([dS, dR]))
            U, R = V[:5], V[5:]
    R = R.clamp_min(0.0)
    return _pack(s["boxes"], torch.cat([U, R * (U[0] / R.sum(0))]))


def _mlp_exact(s):
    W, b = s["net"].get_params()
    W = torch.tensor(W, dtype=F64, device=DEV)
    b = torch.tensor(b, dtype=F64, device=DEV).requires_grad_()
    shapes = [(128, 16)] + [(128, 128)] * 3 + [(16, 128)]
    W.requires_grad_()
    h = torch.nn.functional.pad(s["X"].double(), (0, 4))
    o = ob = 0
    for l, (r, c) in enumerate(shapes):
        h = h @ W[o:o + r * c].reshape(r, c).T + b[ob:ob + r]
        o, ob = o + r * c, ob + r
        if l < 4:
            h = torch.nn.functional.gelu(h)
    loss = ((h[:, :10] - s["T"].double()) ** 2).mean()
    loss.backward()
    return {"loss": loss.detach(), "gW": W.grad, "gb": b.grad}


def exact(case, seed):
    k = case["kind"]
    if k == "jet":
        return None  # a subcycled, cut and refluxed hierarchy: minutes of plain torch, box by box
    s = prepare(case, seed)
    P = s["ctx"].parm
    if k == "rhs":
        dS, fl = _regular_rhs(s["S"], (case["nx"], case["ny"], case["nz"]), s["dxinv"], P, case["visc"],
                              case["gravity"])
        return [dS] + (fl if case["flux"] else [])
    if k == "eb":
        return _eb_exact(s)
    if k == "chem_rhs":
        dS, dR, fl, fs = _chem_rhs(_Mech(P), s["S"], s["R"], (case["nx"], case["ny"], case["nz"]), s["dxinv"],
                                   case["visc"])
        return [dS, dR] + (fl + fs if case["flux"] else [])
    if k == "chem":
        return list(_chem_step(_Mech(P), s["S0"], s["R0"], case["dt"]))
    if k == "level":
        return _level_exact(s)
    if k == "react":
        return _react_exact(s)
    return _mlp_exact(s)
