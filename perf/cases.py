"""Measured workloads of the solver: what a program that uses it runs, through
the package's public classes, over the range of grids it is used on.

A case is a dict of plain values.  `prepare` builds what such a program holds
before the call (solver handles, a flow state made from the seed, output
buffers), `run` is one pass, `exact` the same pass in 64 bits in plain torch.

The starting states are synthetic: a freestream with smooth disturbances and,
for supersonic flow, a normal-shock layer ahead of the obstacle, so that the
limiters, every branch of the wave fan, the wall faces and the boundary
conditions all take part.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "fvm-airidynamic-simulator_b200"))
import fvm_b200  # noqa: E402
from fvm_b200 import abi  # noqa: E402

DEV = "cuda"
FIELDS = (abi.FIELD_DENSITY, abi.FIELD_PRESSURE, abi.FIELD_TEMPERATURE, abi.FIELD_VELOCITY_MAG, abi.FIELD_MACH)
# obstacle classes used across the cases
SHAPES = {"circle": abi.SHAPE_CIRCLE, "star": abi.SHAPE_STAR, "diamond": abi.SHAPE_DIAMOND,
          "capsule": abi.SHAPE_CAPSULE, "triangle": abi.SHAPE_TRIANGLE, "starship": abi.SHAPE_STARSHIP,
          "cone": abi.SHAPE_CONE_CAPSULE}


# ----------------------------------------------------------------- the cases
def _steps(name, nx, ny, mach, viscous, flux, limiter, shape, steps, dt="cfl", isothermal=False):
    """`steps` time steps from a given state, then the five derived fields on the device."""
    return {"name": name, "kind": "steps", "nx": nx, "ny": ny, "mach": mach, "viscous": viscous, "flux": flux,
            "limiter": limiter, "shape": shape, "steps": steps, "dt": dt, "isothermal": isothermal}


def listed():
    return [
        # the interactive application at its default grid: per frame one step, the displayed field, the next time step
        {"name": "frames_512x256", "kind": "frames", "nx": 512, "ny": 256, "mach": 3.0, "viscous": False,
         "flux": "hllc", "limiter": "minmod", "shape": "circle", "frames": 4, "isothermal": False},
        # the smallest grid of the served mix: launches and latency
        _steps("steps_256x128_euler", 256, 128, 2.0, False, "hllc", "minmod", "diamond", 8),
        # Mach-3 circle, inviscid, AUSM+
        _steps("steps_512x256_euler_ausm", 512, 256, 3.0, False, "ausm+", "minmod", "circle", 8),
        # the reference's own KernelBenchmark case: viscous, time step given by the caller
        _steps("steps_1024x512_ns_fixed", 1024, 512, 3.0, True, "hllc", "minmod", "circle", 8, dt="fixed"),
        # Re-200 vortex street
        _steps("steps_2048x1024_ns_ausm", 2048, 1024, 0.3, True, "ausm+", "minmod", "circle", 4),
        # a grid that fits no tile: odd in both directions
        _steps("steps_1501x777_euler", 1501, 777, 2.5, False, "hllc", "vanleer", "star", 4),
        # Mach-8 blunted cone at full size, isothermal wall: the largest solve
        _steps("steps_8192x4096_ns_cone", 8192, 4096, 8.0, True, "hllc", "vanleer", "cone", 2, isothermal=True),
        # many small solves of uneven size advanced together, Euler and Navier-Stokes mixed
        {"name": "batch_16_uneven", "kind": "batch", "count": 16, "min_nx": 128, "max_nx": 1024, "mix": 3,
         "steps": 24},
        # an obstacle the user turns while the flow runs: geometry update, one step, displayed field
        {"name": "moving_1024x512", "kind": "moving", "nx": 1024, "ny": 512, "mach": 2.0, "viscous": True,
         "flux": "hllc", "limiter": "minmod", "shape": "starship", "isothermal": False},
        # one sample of a run's history: forces, totals, maxima, shock standoff
        {"name": "monitor_2048x1024", "kind": "monitor", "nx": 2048, "ny": 1024, "mach": 8.0, "viscous": True,
         "flux": "hllc", "limiter": "vanleer", "shape": "cone", "isothermal": True},
        # a picture of the flow at the largest size
        {"name": "image_8192x4096", "kind": "image", "nx": 8192, "ny": 4096, "mach": 3.0, "viscous": False,
         "flux": "hllc", "limiter": "minmod", "shape": "circle", "field": 4, "colormap": 4, "format": 1,
         "isothermal": False},
        # a state that lives on the host: uploaded, advanced, read back
        {"name": "roundtrip_640x320", "kind": "roundtrip", "nx": 640, "ny": 320, "mach": 3.0, "viscous": True,
         "flux": "hllc", "limiter": "minmod", "shape": "capsule", "steps": 16, "isothermal": False},
    ]


def _size(rng, lo, hi):
    nx = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return nx, max(48, int(round(nx * rng.choice((0.5, 0.5, rng.uniform(0.4, 0.7))))) + rng.choice((0, 0, 1, -1)))


def draw(rng):
    kind = rng.choice(("steps", "steps", "steps", "steps", "frames", "batch", "moving", "monitor", "image",
                       "roundtrip"))
    viscous = rng.random() < 0.5
    c = {"kind": kind, "mach": round(math.exp(rng.uniform(math.log(0.3), math.log(8.0))), 3), "viscous": viscous,
         "flux": rng.choice(("hllc", "hllc", "ausm+")), "limiter": rng.choice(("minmod", "vanleer")),
         "shape": rng.choice(sorted(SHAPES)), "isothermal": viscous and rng.random() < 0.5}
    if kind == "steps":
        c["nx"], c["ny"] = _size(rng, 96, 6000)
        c["steps"] = rng.choice((1, 2, 3, 4))
        c["dt"] = rng.choice(("cfl", "cfl", "fixed"))
    elif kind == "frames":
        c["nx"], c["ny"] = _size(rng, 128, 2048)
        c["frames"] = rng.choice((2, 3, 4))
    elif kind == "batch":
        c = {"kind": "batch", "count": rng.randint(4, 20), "min_nx": 128, "max_nx": rng.choice((256, 512, 1024)),
             "mix": rng.randrange(1000), "steps": rng.randint(8, 24)}
    elif kind == "moving":
        c["nx"], c["ny"] = _size(rng, 256, 2048)
        c["shape"] = rng.choice(("star", "diamond", "capsule", "triangle", "starship"))
    elif kind == "monitor":
        c["nx"], c["ny"] = _size(rng, 128, 6000)
    elif kind == "image":
        c["nx"], c["ny"] = _size(rng, 128, 6000)
        c["field"], c["colormap"], c["format"] = rng.randrange(5), rng.randrange(5), rng.randrange(2)
    else:
        c["nx"], c["ny"] = _size(rng, 128, 1600)
        c["steps"] = rng.choice((4, 8, 16))
    return c


# --------------------------------------------------------------- preparation
def _params(case, rnd):
    """SimParams and Ext of a case in SI units, mapped as the package's own
    workloads are: 300 K, 101325 Pa, a length scale of 1 m for inviscid flow
    and from the Reynolds number (1e5 on the obstacle diameter; 200 below
    Mach 1) for viscous flow.  The seed moves the obstacle."""
    p, e = abi.params_default(), abi.ext_default()
    p.nx, p.ny, p.mach = case["nx"], case["ny"], case["mach"]
    p.enable_viscosity = bool(case["viscous"])
    p.adiabatic_wall, p.T_wall = not case["isothermal"], 600.0
    p.obstacle_shape = SHAPES[case["shape"]]
    size = 0.08
    abi.compute_derived(p)
    L = 1.0
    if p.enable_viscosity:
        re = 200.0 if case["mach"] < 1.0 else 1e5
        L = re * abi.sutherland(300.0) / (p.rho_inf * p.u_inf * 2.0 * size)
    aspect = case["ny"] / case["nx"]
    p.domain_width, p.domain_height = 2.0 * L, 2.0 * L * aspect
    p.obstacle_x = (0.5 + 0.1 * rnd.random()) * L
    p.obstacle_r = size * (0.9 + 0.2 * rnd.random()) * L
    p.obstacle_rotation = rnd.uniform(0.0, 0.5) if case["shape"] in ("star", "diamond", "triangle") else 0.0
    p.cfl = 0.4
    e.cone_half_angle, e.cone_length = math.radians(15.0), 0.3 * L
    e.ref_length = 2.0 * p.obstacle_r
    e.flux_scheme = abi.FLUX_AUSM_PLUS if case["flux"] == "ausm+" else abi.FLUX_HLLC
    e.limiter = abi.LIMITER_VAN_LEER if case["limiter"] == "vanleer" else abi.LIMITER_MINMOD
    fixed = case["kind"] == "frames" or case.get("dt") == "fixed"
    e.dt_policy = abi.DT_FIXED if fixed else abi.DT_RECOMPUTE
    abi.compute_derived(p)
    # a caller's time step: well inside the limits of the state below
    h = min(p.dx, p.dy)
    p.dt = 0.15 * h / (1.2 * p.u_inf + 4.0 * p.c_inf)
    if p.enable_viscosity:
        p.dt = min(p.dt, 0.1 * h * h * p.rho_inf / abi.sutherland(300.0 * (1.0 + 0.2 * p.mach ** 2)))
    return p, e


def _flow(p, types, rnd):
    """A conserved state, float32 (5, ny, nx): see the module's docstring."""
    nx, ny = p.nx, p.ny
    f = dict(device=DEV, dtype=torch.float32)
    x = ((torch.arange(nx, **f) + 0.5) / nx)[None, :]
    y = ((torch.arange(ny, **f) + 0.5) / ny)[:, None]

    def waves(amp):
        s = torch.zeros((ny, nx), **f)
        for _ in range(3):
            kx, ky, ph = rnd.randint(1, 9), rnd.randint(1, 9), rnd.uniform(0, 2 * math.pi)
            s += torch.sin(2 * math.pi * (kx * x + ky * y) + ph) * (amp * rnd.uniform(0.3, 1.0) / 3)
        return s

    rho = p.rho_inf * (1 + waves(0.05))
    pr = p.p_inf * (1 + waves(0.05))
    u = p.u_inf * (1 + waves(0.05))
    v = p.u_inf * waves(0.05)
    # distance from the obstacle's centre in units of its radius
    X = (x * p.domain_width - p.obstacle_x) / p.obstacle_r
    Y = (y * p.domain_height - p.obstacle_y) / p.obstacle_r
    d = torch.sqrt(X * X + Y * Y)
    if p.mach > 1.1:
        m2, width = p.mach ** 2, 2.0 * max(p.dx, p.dy) / p.obstacle_r
        s = 0.5 * (1 - torch.tanh((d - rnd.uniform(1.7, 2.1)) / width)) * 0.5 * (1 - torch.tanh(2 * X + 0.5))
        jr = 2.4 * m2 / (2 + 0.4 * m2)
        jp = 1 + 2.8 / 2.4 * (m2 - 1)
        rho = rho * (1 + (jr - 1) * s)
        pr = pr * (1 + (jp - 1) * s)
        u = u / (1 + (jr - 1) * s)
    near = 1 - torch.exp(-((d / 1.2) ** 2))  # the flow slows towards the body
    u, v = u * near, v * near
    e = pr / 0.4
    U = torch.stack([rho, rho * u, rho * v, e + 0.5 * rho * (u * u + v * v), e])
    wall = torch.from_numpy(types).to(DEV)
    wall = (wall == abi.CELL_SOLID) | (wall == abi.CELL_GHOST)
    ei = p.p_inf / 0.4
    solid = torch.tensor([p.rho_inf, 0.0, 0.0, ei, ei], **f)[:, None, None]
    return torch.where(wall, solid, U).contiguous()


def _batch_instances(case, seed):
    """(SimParams, Ext) of each solve: sizes from the case, physics from the seed."""
    sizes = [s for s in (128, 256, 512, 1024) if case["min_nx"] <= s <= case["max_nx"]]
    shape, rng = random.Random(case["mix"]), abi.SeededStream(seed)
    got = []
    for _ in range(case["count"]):
        nx = shape.choice(sizes)
        got.append(abi.uneven_instance(rng, sizes=(nx,), p_viscous=float(shape.random() < 0.5)))
    return got


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        inst = _batch_instances(case, seed)
        b = fvm_b200.Batch(inst[0][1])
        return {"case": case, "batch": b, "ids": [b.add(p) for p, _ in inst]}
    rnd = random.Random(seed)
    p, e = _params(case, rnd)
    s = fvm_b200.Solver(p, e)
    U = _flow(p, s.cell_types(), rnd).cpu().numpy()
    s.write_fields(U)
    st = {"case": case, "solver": s}
    if kind == "steps":
        st["out"] = torch.zeros((5, p.ny, p.nx), device=DEV)
    elif kind in ("frames", "moving"):
        st["out"] = torch.zeros((p.ny, p.nx), device=DEV)
        torch.cuda.synchronize()
        s.set_display_field(abi.FIELD_MACH, st["out"].data_ptr())
        st["types"] = torch.zeros((p.ny, p.nx), device=DEV)
    elif kind == "image":
        st["out"] = (torch.zeros((p.ny, p.nx, 4), device=DEV, dtype=torch.uint8) if case["format"] == abi.RGBA_U8
                     else torch.zeros((p.ny, p.nx, 4), device=DEV))
    elif kind == "roundtrip":
        st["host"] = U
    torch.cuda.synchronize()
    return st


# ----------------------------------------------------------------- one pass
def run(st):
    case, kind = st["case"], st["case"]["kind"]
    if kind == "batch":
        b = st["batch"]
        b.step(case["steps"])
        return [b.fields(i) for i in st["ids"]]
    s = st["solver"]
    if kind == "steps":
        s.step(case["steps"])
        for k, f in enumerate(FIELDS):
            s.field_to_device(f, st["out"][k].data_ptr())
        return st["out"]
    if kind == "frames":
        for _ in range(case["frames"]):
            s.step(1)
            s.field_to_device(abi.FIELD_MACH, st["out"].data_ptr())
            s.params.dt = s.compute_dt()
        return {"mach": st["out"], "dt": s.params.dt}
    if kind == "moving":
        p = s.params
        p.obstacle_rotation += 0.01
        p.wing_rotation += 0.02
        s.update_obstacle(p)
        s.step(1)
        s.field_to_device(abi.FIELD_MACH, st["out"].data_ptr())
        s.cell_types_to_device(st["types"].data_ptr())
        return {"mach": st["out"], "types": st["types"]}
    if kind == "monitor":
        d = s.diagnostics()
        return {"wall": np.array([d.force_x, d.force_y, d.wall_heat, d.wall_heat_max]),
                "totals": np.array([d.mass, d.mom_x, d.mom_y, d.energy]),
                "max_T": s.max_temperature(), "max_mach": s.max_mach(), "standoff": s.shock_standoff()}
    if kind == "image":
        lo, hi = _image_range(case, s.params)
        s.colormap_to_device(case["field"], case["colormap"], lo, hi, st["out"].data_ptr(), case["format"])
        return st["out"]
    s.write_fields(st["host"])
    s.step(case["steps"])
    return s.fields()


def _image_range(case, p):
    top = {0: 300.0 * (1 + 0.2 * p.mach ** 2), 1: 3.0 * p.p_inf, 2: 3.0 * p.rho_inf, 3: 1.1 * p.u_inf, 4: p.mach}
    return 0.0, top[case["field"]]


# -------------------------------------------------------------- what it takes
def _cells(case):
    if case["kind"] == "batch":
        return sum(p.nx * p.ny for p, _ in _batch_instances(case, 1))
    return case["nx"] * case["ny"]


def work(case):
    """Bytes: the state (20 B a cell) read and written and the cell class read
    once per step, the inputs and outputs of the pass once.  Flops per cell:
    two RK stages of two faces (about 120 each), slopes, primitives and update
    (about 100 together), and two viscous half steps of about 110."""
    n, kind = float(_cells(case)), case["kind"]
    steps = {"steps": case.get("steps", 0), "frames": case.get("frames", 0), "batch": case.get("steps", 0),
             "roundtrip": case.get("steps", 0), "moving": 1}.get(kind, 0)
    if kind == "batch":
        visc = sum(p.nx * p.ny for p, _ in _batch_instances(case, 1) if p.enable_viscosity) / n
    else:
        visc = 1.0 if case["viscous"] else 0.0
    b, f = 41.0 * steps, (680.0 + 220.0 * visc) * steps
    if kind == "steps":
        b, f = b + 20, f + 40
    elif kind == "frames":
        b, f = b + 4 * steps, f + 12 * steps
    elif kind == "moving":
        b, f = b + 10, f + 120
    elif kind == "monitor":
        b, f = 25.0, 60.0
    elif kind == "image":
        b, f = 17.0 + (4 if case["format"] == abi.RGBA_U8 else 16), 40.0
    else:  # batch, roundtrip: the state to the host (and from it)
        b += 20.0 if kind == "batch" else 40.0
    return {"bytes": b * n, "flops": f * n}


# ------------------------------------------------------- the same in 64 bits
GA, RG, CP = 1.4, 287.05, 1.4 * 287.05 / 0.4
RMIN, PMIN, TMIN, TMAX = 1e-4, 1e-2, 50.0, 5000.0


class Exact:
    """The solver's method on a 64-bit state in plain torch: MUSCL + HLLC or
    AUSM+, the internal-energy equation, SSP-RK2, viscous half steps, boundary
    conditions.  `types` and `sdf` are the geometry the solve is given."""

    def __init__(self, p, e, types, sdf):
        self.p, self.e = p, e
        self.set_geometry(types, sdf)
        self.dx, self.dy = float(p.dx), float(p.dy)
        self.visc = bool(p.enable_viscosity)
        self.inf = (float(p.rho_inf), float(p.u_inf), float(p.v_inf), float(p.p_inf))

    def set_geometry(self, types, sdf):
        self.ct = torch.from_numpy(types.astype(np.int64)).to(DEV)
        self.wall = (self.ct == 1) | (self.ct == 2)
        self.fluid = self.ct == 0
        ny, nx = self.ct.shape
        gj, gi = torch.nonzero(self.ct == 2, as_tuple=True)
        self.g = (gj, gi)
        self.cand = []
        if gj.numel() == 0:
            return
        s = torch.from_numpy(sdf.astype(np.float64)).to(DEV)
        dx, dy = float(self.p.dx), float(self.p.dy)

        def at(j, i):
            return s[j.clamp(0, ny - 1), i.clamp(0, nx - 1)]

        gx, gy = (at(gj, gi + 1) - at(gj, gi - 1)) / (2 * dx), (at(gj + 1, gi) - at(gj - 1, gi)) / (2 * dy)
        ln = torch.sqrt(gx * gx + gy * gy) + 1e-10
        self.gx, self.gy = gx / ln, gy / ln
        near = ((-1, 0), (1, 0), (0, -1), (0, 1), (-1, -1), (1, -1), (-1, 1), (1, 1))
        dots, qj, qi = [], [], []
        for di, dj in near:
            i, j = gi + di, gj + dj
            ok = (i >= 0) & (i < nx) & (j >= 0) & (j < ny) & (at(j, i) > 0)
            dot = (di * self.gx + dj * self.gy) / math.sqrt(di * di + dj * dj)
            dots.append(torch.where(ok & (dot > -1), dot, torch.full_like(dot, -9.0)))
            qj.append(j.clamp(0, ny - 1))
            qi.append(i.clamp(0, nx - 1))
        dots = torch.stack(dots)
        val, order = torch.sort(dots, dim=0, descending=True, stable=True)
        qj, qi = torch.stack(qj).gather(0, order), torch.stack(qi).gather(0, order)
        self.cand = [(val[k] > -8, qj[k], qi[k]) for k in range(8)]

    # per-cell pieces
    def prims(self, U):
        r = U[0].clamp(min=RMIN)
        u, v = U[1] / r, U[2] / r
        e = U[3] - 0.5 * r * (u * u + v * v)
        e = torch.where((U[3] > 0) & (U[4] < 1e-3 * U[3]), U[4], e)
        p = (0.4 * e).clamp(min=PMIN)
        return u, v, p, (p / (r * RG)).clamp(TMIN, TMAX)

    def limited(self, a, b):
        if self.e.limiter == abi.LIMITER_MINMOD:
            one = torch.ones_like(a)
            return 0.5 * (torch.copysign(one, a) + torch.copysign(one, b)) * torch.minimum(a.abs(), b.abs())
        ab = a * b
        return torch.where(ab > 0, 2 * ab / torch.where(ab > 0, a + b, torch.ones_like(a)), torch.zeros_like(a))

    def riemann(self, rL, nL, tL, pL, rR, nR, tR, pR):
        EL, ER = pL / 0.4 + 0.5 * rL * (nL * nL + tL * tL), pR / 0.4 + 0.5 * rR * (nR * nR + tR * tR)
        HL, HR = (EL + pL) / rL, (ER + pR) / rR
        if self.e.flux_scheme == abi.FLUX_AUSM_PLUS:
            k = 2 * 0.4 / 2.4
            sL, sR = torch.sqrt(k * HL), torch.sqrt(k * HR)
            c = torch.minimum(sL * sL / torch.maximum(sL, nL), sR * sR / torch.maximum(sR, -nR))
            ML, MR = nL / c, nR / c

            def split(M, s):
                out, q = M.abs() >= 1, (M * M - 1)
                m = torch.where(out, 0.5 * (M + s * M.abs()), s * (0.25 * (M + s) ** 2 + 0.125 * q * q))
                w = torch.where(out, (s * M > 0).to(M.dtype), 0.25 * (M + s) ** 2 * (2 - s * M) + s * 0.1875 * M * q * q)
                return m, w

            mp, wp = split(ML, 1.0)
            mm, wm = split(MR, -1.0)
            m = mp + mm
            a, b = c * 0.5 * (m + m.abs()), c * 0.5 * (m - m.abs())
            return (a * rL + b * rR, a * rL * nL + b * rR * nR + wp * pL + wm * pR, a * rL * tL + b * rR * tR,
                    a * rL * HL + b * rR * HR)
        cL, cR = torch.sqrt(GA * pL / rL), torch.sqrt(GA * pR / rR)
        qL, qR = torch.sqrt(rL), torch.sqrt(rR)
        den = qL + qR + 1e-10
        n, t, H = (qL * nL + qR * nR) / den, (qL * tL + qR * tR) / den, (qL * HL + qR * HR) / den
        c2 = 0.4 * (H - 0.5 * (n * n + t * t))
        c = torch.where(c2 > 0, torch.sqrt(c2.clamp(min=0)), 0.5 * (cL + cR))
        SL, SR = torch.minimum(nL - cL, n - c), torch.maximum(nR + cR, n + c)
        dl = 0.1 * torch.maximum(cL, cR)
        SL, SR = torch.where(SL.abs() < dl, -dl, SL), torch.where(SR.abs() < dl, dl, SR)
        ds = rL * (SL - nL) - rR * (SR - nR)
        ds = torch.copysign(ds.abs().clamp(min=1e-10), ds)
        Ss = (pR - pL + rL * nL * (SL - nL) - rR * nR * (SR - nR)) / ds
        supL = SL >= 0
        supR = ~supL & (SR <= 0)
        left = supL | (~supR & (Ss >= 0))
        r, n, t, p, E, S = (torch.where(left, a, b) for a, b in ((rL, rR), (nL, nR), (tL, tR), (pL, pR), (EL, ER),
                                                                (SL, SR)))
        f = [r * n, r * n * n + p, r * n * t, (E + p) * n]
        cd = S - Ss
        cd = torch.where(cd.abs() < 1e-10, torch.where(cd >= 0, 1e-10, -1e-10).to(cd.dtype), cd)
        rs = (r * (S - n) / cd).clamp(min=RMIN)
        ps = (p + r * (S - n) * (Ss - n)).clamp(min=PMIN)
        Es = (E * (S - n) + ps * Ss - p * n) / cd
        S = torch.where(supL | supR, torch.zeros_like(S), S)
        return f[0] + S * (rs - r), f[1] + S * (rs * Ss - r * n), f[2] + S * (rs - r) * t, f[3] + S * (Es - E)

    def fluxes(self, W, ax):
        """Fluxes (mass, x-, y-momentum, energy, rho_e) and face velocities of
        the faces between neighbouring cells along axis ax (1: x, 0: y)."""
        n = W[0].shape[ax]

        def sh(q, k):  # q of the cell k further along, edge cells repeated
            return q.index_select(ax, (torch.arange(n, device=DEV) + k).clamp(0, n - 1))

        def lo(q):
            return q.narrow(ax, 0, n - 1)

        def hi(q):
            return q.narrow(ax, 1, n - 1)

        r, u, v, p = W
        wall = self.wall
        valid = lo(~wall) & hi(~wall)
        first = lo(sh(wall, -1)) | lo(sh(wall, 2)) | (lo(r) < 0.01) | (hi(r) < 0.01)
        om = torch.where(first, 0.0, 0.5).to(r.dtype)
        L, R = [], []
        for q in (r, u if ax else v, v if ax else u, p):
            s = self.limited(q - sh(q, -1), sh(q, 1) - q)
            L.append(lo(q) + om * lo(s))
            R.append(hi(q) - om * hi(s))
        L[0], R[0], L[3], R[3] = (L[0].clamp(min=RMIN), R[0].clamp(min=RMIN), L[3].clamp(min=PMIN),
                                  R[3].clamp(min=PMIN))
        m, fn, ft, fe = self.riemann(*L, *R)
        fre = torch.where(0.5 * (L[1] + R[1]) >= 0, L[3] / 0.4 * L[1], R[3] / 0.4 * R[1])
        z = torch.zeros_like(m)
        m, ft, fe, fre = (torch.where(valid, a, z) for a in (m, ft, fe, fre))
        fn = torch.where(valid, fn, lo(p))
        vel = m / (0.5 * (lo(r).clamp(min=RMIN) + hi(r).clamp(min=RMIN)))
        return ([m, fn, ft, fe, fre] if ax else [m, ft, fn, fe, fre]), vel

    def stage(self, U, dt):
        u, v, p, _ = self.prims(U)
        W = (U[0], u, v, p)
        N = [q.clone() for q in U]
        ny, nx = U[0].shape
        div = torch.zeros_like(p)
        for ax, h in ((1, self.dx), (0, self.dy)):
            F, vel = self.fluxes(W, ax)
            k = (nx if ax else ny) - 2
            if k < 1:
                continue

            def diff(q):
                return q.narrow(ax, 1, k) - q.narrow(ax, 0, k)

            for q in range(5):
                N[q].narrow(ax, 1, k).sub_(dt / h * diff(F[q]))
            div.narrow(ax, 1, k).add_(diff(vel) / h)
        N[4][1:-1, 1:-1] -= dt * (p * div)[1:-1, 1:-1]
        r = torch.where(torch.isfinite(N[0]) & (N[0] >= RMIN), N[0], U[0].clamp(min=RMIN))
        ru, rv, E = (torch.where(torch.isfinite(N[q]), N[q], U[q]) for q in (1, 2, 3))
        re = torch.where(torch.isfinite(N[4]) & (N[4] >= PMIN / 0.4), N[4], U[4])
        sp = torch.sqrt((ru / r) ** 2 + (rv / r) ** 2)
        sc = torch.where(sp > 5000.0, 5000.0 / sp.clamp(min=1.0), torch.ones_like(sp))
        ru, rv = ru * sc, rv * sc
        ke = 0.5 * (ru * ru + rv * rv) / r
        e = torch.where((E > 0) & (re < 1e-3 * E), re, E - ke)
        e = torch.minimum(torch.maximum(e, r * (RG * TMIN / 0.4)), r * (RG * TMAX / 0.4))
        return [torch.where(self.wall, a, b) for a, b in zip(U, (r, ru, rv, e + ke, e))]

    def viscous(self, U, dt):
        u, v, p, T = self.prims(U)
        mu = 1.716e-5 * (T / 273.15) ** 1.5 * (273.15 + 110.4) / (T + 110.4)
        k = mu * CP / float(self.e.prandtl)
        live = (self.ct != 1).to(p.dtype)

        def grad(q, ax, h):
            g = torch.zeros_like(q)
            n = q.shape[ax]
            g.narrow(ax, 1, n - 2).copy_((q.narrow(ax, 2, n - 2) - q.narrow(ax, 0, n - 2)) / (2 * h))
            g.narrow(ax, 0, 1).copy_((q.narrow(ax, 1, 1) - q.narrow(ax, 0, 1)) / h)
            g.narrow(ax, n - 1, 1).copy_((q.narrow(ax, n - 1, 1) - q.narrow(ax, n - 2, 1)) / h)
            return g

        ux, uy, vx, vy = grad(u, 1, self.dx), grad(u, 0, self.dy), grad(v, 1, self.dx), grad(v, 0, self.dy)
        dv = ux + vy
        txx, tyy, txy = (live * mu * a for a in (2 * ux - 2 / 3 * dv, 2 * vy - 2 / 3 * dv, uy + vx))
        qx, qy = -live * k * grad(T, 1, self.dx), -live * k * grad(T, 0, self.dy)
        dq = grad(qx, 1, self.dx) + grad(qy, 0, self.dy)
        dw = grad(u * txx + v * txy, 1, self.dx) + grad(u * txy + v * tyy, 0, self.dy)
        phi = txx * ux + tyy * vy + txy * (uy + vx)
        upd = self.fluid.clone()
        upd[0], upd[-1], upd[:, 0], upd[:, -1] = False, False, False, False
        rhs = (grad(txx, 1, self.dx) + grad(txy, 0, self.dy), grad(txy, 1, self.dx) + grad(tyy, 0, self.dy), dw - dq,
               phi - dq)
        return [U[0]] + [torch.where(upd, U[q + 1] + dt * rhs[q], U[q + 1]) for q in range(4)], mu

    # boundary conditions
    def nrbc(self, r, n, t, p, raw, sign):
        """Non-reflecting condition with outward direction `sign`: (rho, n, t, p)."""
        rI, uI, vI, pI = self.inf
        nI, tI = (uI, vI) if raw else (vI, uI)
        cl = torch.sqrt(GA * p / r.clamp(min=RMIN))
        c, cI = torch.sqrt(GA * p / r), math.sqrt(GA * pI / rI)
        o1, o3, o4 = sign * n > 0, sign * (n + cl) > 0, sign * (n - cl) > 0
        R1 = torch.where(o1, p * r ** -GA, pI * rI ** -GA)
        R2 = torch.where(o1, t, tI)
        R3 = torch.where(o3, n + 5 * c, nI + 5 * cI)
        R4 = torch.where(o4, n - 5 * c, nI - 5 * cI)
        c2 = (0.1 * (R3 - R4)) ** 2
        rn = (c2 / GA / R1) ** 2.5
        return rn, 0.5 * (R3 + R4), R2, rn * c2 / GA

    def put(self, U, at, r, u, v, p):
        for q, val in enumerate((r, r * u, r * v, p / 0.4 + 0.5 * r * (u * u + v * v), p / 0.4)):
            U[q][at] = val

    def bc(self, U):
        U = [q.clone() for q in U]
        rI, uI, vI, pI = self.inf
        ny, nx = U[0].shape
        ct, inner = self.ct, torch.ones_like(self.wall)
        first = ct == 3
        first[:, 0] = True
        out = (ct == 4) & ~first
        out[:, nx - 1] |= ~first[:, nx - 1]
        inner &= ~first & ~out
        one = torch.ones((), device=DEV, dtype=torch.float64)
        self.put(U, first, rI * one, uI * one, vI * one, pI * one)
        col = [q[out] for q in U]
        u, v, p, _ = self.prims(col)
        r, n, t, p = self.nrbc(col[0], u, v, p, True, 1.0)
        self.put(U, out, r, n, t, p)
        for j, sign in ((0, -1.0), (ny - 1, 1.0)):
            at = inner & (ct != 2)
            rows = torch.zeros_like(at)
            rows[j] = at[j]
            row = [q[rows] for q in U]
            r0 = row[0].clamp(min=RMIN)
            u, v, p, _ = self.prims([r0] + row[1:])
            r, n, t, p = self.nrbc(r0, v, u, p, False, sign)
            self.put(U, rows, r, t, n, p)
        self.put(U, inner & (ct == 1), rI * one, 0 * one, 0 * one, pI * one)
        return self.ghosts(U)

    def ghosts(self, A):
        gj, gi = self.g
        if gj.numel() == 0:
            return A
        rI, _, _, pI = self.inf
        found = torch.zeros_like(gj, dtype=torch.bool)
        qj, qi = gj.clone(), gi.clone()
        for ok, j, i in self.cand:
            use = ok & (A[0][j, i] >= RMIN) & ~found
            qj, qi = torch.where(use, j, qj), torch.where(use, i, qi)
            found |= use
        r, ru, rv, E = (A[q][qj, qi] for q in range(4))
        u, v = ru / r, rv / r
        p = 0.4 * (E - 0.5 * r * (u * u + v * v))
        r, p = r.clamp(min=RMIN), p.clamp(min=PMIN)
        gx, gy = self.gx, self.gy
        vn, vt = u * gx + v * gy, -v * gx + u * gy
        T = (p / (r * RG)).clamp(TMIN, TMAX)
        p = r * RG * T
        ug, vg = -u, -v
        if not self.visc:
            s = torch.where(vn > 0, (vn / (vn + 100.0)).clamp(max=0.8), torch.zeros_like(vn))
            ug, vg = (1 - s) * ug + s * (-vn * gx + vt * gy), (1 - s) * vg + s * (-vn * gy - vt * gx)
        sp = torch.sqrt(ug * ug + vg * vg)
        sc = torch.where(sp > 2500.0, 2500.0 / sp.clamp(min=1.0), torch.ones_like(sp))
        ug, vg = ug * sc, vg * sc
        Tg = T if self.p.adiabatic_wall else (2 * float(self.p.T_wall) - T).clamp(TMIN, TMAX)
        rg = (p / (RG * Tg)).clamp(min=RMIN)
        new = [rg, rg * ug, rg * vg, p / 0.4 + 0.5 * rg * (ug * ug + vg * vg), p / 0.4]
        none = (rI, 0.0, 0.0, pI / 0.4, pI / 0.4)
        for q in range(5):
            A[q] = A[q].index_put((gj, gi), torch.where(found, new[q], torch.full_like(rg, none[q])))
        return A

    # the time step
    def maxima(self, U, mu=None):
        u, v, p, T = self.prims(U)
        if mu is None:
            mu = 1.716e-5 * (T / 273.15) ** 1.5 * (273.15 + 110.4) / (T + 110.4)
        speed = torch.sqrt(u * u + v * v) + torch.sqrt(GA * p / (U[0] + 1e-10))
        nu = torch.where(self.ct == 1, torch.zeros_like(mu), mu / (U[0] + 1e-10))
        return float(speed.max()), float(nu.max())

    def dt_of(self, m):
        h = min(self.dx, self.dy)
        dt = float(self.p.cfl) * h / (m[0] + 1e-10)
        return min(dt, float(self.p.cfl_visc) * h * h / (m[1] + 1e-10)) if self.visc else dt

    def step(self, U, dt):
        """One step; (the new state, its CFL maxima)."""
        if self.visc:
            U, _ = self.viscous(U, 0.5 * dt)
        S = self.bc(self.stage(U, dt))
        S = self.stage(S, dt)
        N = [0.5 * a + 0.5 * b for a, b in zip(S, U)]
        mu = None
        if self.visc:
            N, mu = self.viscous(N, 0.5 * dt)
        N = self.bc(N)
        return N, self.maxima(N, mu)

    def steps(self, U, n):
        dt = float(self.p.dt) if self.e.dt_policy == abi.DT_FIXED else self.dt_of(self.maxima(U))
        for _ in range(n):
            U, m = self.step(U, dt)
            if self.e.dt_policy != abi.DT_FIXED:
                dt = self.dt_of(m)
        return U

    def freestream(self):
        rI, uI, vI, pI = self.inf
        E = pI / 0.4 + 0.5 * rI * (uI * uI + vI * vI)
        one = torch.ones(self.ct.shape, device=DEV, dtype=torch.float64)
        return self.bc([one * q for q in (rI, rI * uI, rI * vI, E, pI / 0.4)])

    # what is derived from a state
    def field(self, U, kind):
        r = U[0] + 1e-10
        T = 0.4 * (U[4] / r) / RG
        speed = torch.sqrt((U[1] / r) ** 2 + (U[2] / r) ** 2)
        if kind == abi.FIELD_MACH:
            return speed / (torch.sqrt(GA * RG * T) + 1e-10)
        return {abi.FIELD_TEMPERATURE: T, abi.FIELD_PRESSURE: 0.4 * U[4], abi.FIELD_DENSITY: U[0],
                abi.FIELD_VELOCITY_MAG: speed}[kind]

    def monitor(self, U, sdf):
        u, v, p, T = self.prims(U)
        dx, dy = self.dx, self.dy
        ny, nx = p.shape
        mu = 1.716e-5 * (T / 273.15) ** 1.5 * (273.15 + 110.4) / (T + 110.4)
        k = mu * CP / float(self.e.prandtl)

        def grad(q, ax, h):
            return torch.gradient(q, spacing=h, dim=ax, edge_order=1)[0]

        ux, uy, vx, vy = grad(u, 1, dx), grad(u, 0, dy), grad(v, 1, dx), grad(v, 0, dy)
        dv = ux + vy
        txx, tyy, txy = mu * (2 * ux - 2 / 3 * dv), mu * (2 * vy - 2 / 3 * dv), mu * (uy + vx)
        qx, qy = -k * grad(T, 1, dx), -k * grad(T, 0, dy)
        fx = fy = heat = peak = 0.0
        for ax, dA in ((1, dy), (0, dx)):
            n = nx if ax else ny
            wa, wb = self.wall.narrow(ax, 0, n - 1), self.wall.narrow(ax, 1, n - 1)
            face = wa != wb
            sg = torch.where(wa, 1.0, -1.0).to(p.dtype)[face]
            pa = p.narrow(ax, 0, n - 1)[face]

            def fl(q):  # of the fluid cell beside the face
                return torch.where(wa, q.narrow(ax, 1, n - 1), q.narrow(ax, 0, n - 1))[face]

            f = [-pa * sg * dA, torch.zeros_like(pa)]
            if self.visc:
                f[0] = f[0] + fl(txx if ax else tyy) * sg * dA
                f[1] = f[1] + fl(txy) * sg * dA
                qw = -fl(qx if ax else qy) * sg
                heat += float((qw * dA).sum())
                peak = max(peak, float(qw.max()) if qw.numel() else 0.0)
            fx += float((f[0] if ax else f[1]).sum())
            fy += float((f[1] if ax else f[0]).sum())
        live = (~self.wall).to(p.dtype) * dx * dy
        j = ny // 2
        row, pj = sdf[j].astype(np.float64), p[j].cpu().numpy()
        standoff = math.nan
        m2 = float(self.p.u_inf) ** 2 / (GA * self.inf[3] / self.inf[0])
        if m2 > 1:
            mid = self.inf[3] * (1 + 0.5 * (2.8 / 2.4 * (m2 - 1)))
            hit = np.nonzero((row[:-1] > 0) & (row[1:] <= 0))[0]
            if hit.size:
                b = int(hit[0])
                xb = (b + 0.5) * dx + dx * row[b] / (row[b] - row[b + 1])
                up = np.nonzero((pj[:b] < mid) & (pj[1:b + 1] >= mid))[0]
                if up.size:
                    i = int(up[0])
                    standoff = xb - ((i + 0.5) * dx + dx * (mid - pj[i]) / (pj[i + 1] - pj[i]))
        mach = torch.sqrt(u * u + v * v) / (torch.sqrt(GA * p / (U[0] + 1e-10)) + 1e-10)
        return {"wall": np.array([fx, fy, heat, peak]),
                "totals": np.array([float((q * live).sum()) for q in U[:4]]),
                "max_T": float(T.max()), "max_mach": float(mach.max()), "standoff": standoff}


def exact(case, seed):
    """The geometry (cell classes and distance field) is an input, read from a
    handle: which class a cell at the edge of a band falls into is a matter of
    32-bit rounding and not of the flow's accuracy."""
    kind = case["kind"]
    if kind == "batch":
        got = []
        for p, e in _batch_instances(case, seed):
            with fvm_b200.Solver(p, e) as s:
                x = Exact(p, e, s.cell_types(), s.sdf())
            got.append(torch.stack(x.steps(x.freestream(), case["steps"])))
        return got
    rnd = random.Random(seed)
    p, e = _params(case, rnd)
    with fvm_b200.Solver(p, e) as s:
        types, sdf = s.cell_types(), s.sdf()
        U = list(_flow(p, types, rnd).double())
        x = Exact(p, e, types, sdf)
        if kind == "moving":
            p.obstacle_rotation += 0.01
            p.wing_rotation += 0.02
            s.update_obstacle(p)
            new, sdf = s.cell_types(), s.sdf()
            bare = x.wall & torch.from_numpy(new == 0).to(DEV)  # cells that the obstacle left
            x.set_geometry(new, sdf)
            U = x.bc([torch.where(bare, torch.zeros_like(q), q) for q in U])
            return {"mach": x.field(x.steps(U, 1), abi.FIELD_MACH), "types": x.ct.double()}
    if kind == "steps":
        U = x.steps(U, case["steps"])
        return torch.stack([x.field(U, f) for f in FIELDS])
    if kind == "frames":
        dt = float(p.dt)
        for _ in range(case["frames"]):
            U, m = x.step(U, dt)
            dt = x.dt_of(m)
        return {"mach": x.field(U, abi.FIELD_MACH), "dt": dt}
    if kind == "monitor":
        return x.monitor(U, sdf)
    if kind == "image":
        if case["format"] == abi.RGBA_U8:
            return None
        lo, hi = _image_range(case, p)
        s = ((x.field(U, case["field"]) - lo) / (hi - lo + 1e-4)).clamp(0, 1) * 256 - 0.5
        fl = torch.floor(s)
        lut = torch.from_numpy(fvm_b200.colormap_table(case["colormap"]).astype(np.float64)).to(DEV)
        i0, i1 = fl.long().clamp(0, 255), (fl.long() + 1).clamp(0, 255)
        rgb = (1 - (s - fl))[..., None] * lut[i0] + (s - fl)[..., None] * lut[i1]
        rgb = torch.where(x.wall[..., None], torch.full_like(rgb, 0.3), rgb)
        return torch.cat([rgb, torch.ones_like(rgb[..., :1])], dim=2)
    return torch.stack(x.steps(U, case["steps"]))
