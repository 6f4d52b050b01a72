"""Workloads that a user of this framework runs, each through the public Python
entry points: periodic Taylor-Green vortices from a test box to a large one,
ducts with walls, an inlet and an outlet in the storages used in earnest, a
monitored run that changes its inlet every step, an obstacle flow with the LES
collision, a coupled scalar with field output, an ensemble of small lattices
and a gradient through time.  Sizes follow the repository's benchmark, tests
and examples, with odd and ragged ones beside them.

A case runs `steps` time steps per pass on a lattice prepared as the README
does it (create, map, inlet, initial state, autotune); the populations it
returns are those of the lattice's own device buffer.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch
import torch.utils.checkpoint

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tnl-lbm_b200"))
import pytnl_lbm as pl  # noqa: E402

DEV = "cuda"
STORAGE = {"f64": pl.STORE_F64, "f32": pl.STORE_F32, "f16s": pl.STORE_F16S, "bf16s": pl.STORE_BF16S}
ELEM = {"f64": 8, "f32": 4, "f16s": 2, "bf16s": 2}
COLL = {"cum": pl.COLL_CUM, "srt": pl.COLL_SRT, "bgk": pl.COLL_BGK, "mrt": pl.COLL_MRT}
FLUID, WALL, INFLOW, INFLOW_LEFT, OUTFLOW_EQ, OUTFLOW_RIGHT, NOTHING = 0, 1, 2, 3, 6, 7, 10
U0 = 0.05      # vortex amplitude
U_MAX = 0.04   # inlet peak


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------

def _vortex(name, x, y, z, storage="f32", steps=10, energy=False):
    return dict(name=name, kind="vortex", x=x, y=y, z=z, storage=storage, coll="cum", steps=steps, energy=energy)


def _duct(name, x, y, z, storage="f32", coll="cum", steps=20, use="run", spheres=0):
    return dict(name=name, kind="duct", x=x, y=y, z=z, storage=storage, coll=coll, steps=steps, use=use, spheres=spheres)


def listed():
    return [
        # the smallest box that a test or a first try runs: ten launches of a few microseconds each
        _vortex("vortex_32", 32, 32, 32),
        # the 64^3 vortex of the reference's own example, kinetic energy read every ten steps
        _vortex("vortex_64_energy", 64, 64, 64, energy=True),
        # a box whose edges are no powers of two, and odd
        _vortex("vortex_odd", 125, 97, 61),
        # a resolved vortex, far larger than the caches
        _vortex("vortex_256", 256, 256, 256),
        # the headline workload: the duct with walls, inlet and outlet
        _duct("duct_f32", 512, 128, 128),
        # the same lattice in 16-bit shifted storage
        _duct("duct_f16", 512, 128, 128, storage="f16s"),
        # double precision with A-B streaming and the pulling outlet: the reference's default configuration
        _duct("duct_f64_ab", 256, 96, 96, storage="f64", steps=10, use="ab"),
        # a controlled run: new inlet profile, one step, its sums read back
        _duct("duct_monitor", 300, 100, 100, steps=1, use="monitor"),
        # flow around obstacles with the LES collision, a ragged box
        _duct("spheres_les", 333, 85, 59, coll="mrt", spheres=12),
        # a scalar carried by the duct, with the flow and scalar fields written out at the end
        _duct("duct_scalar", 192, 64, 64, steps=100, use="scalar"),
        # a parameter study: many small boxes advanced together, every member's sums read
        dict(name="ensemble", kind="ensemble", members=128, shapes=5, steps=50),
        # gradient of a flow mismatch with respect to a body force, through the whole run
        dict(name="gradient", kind="gradient", x=160, y=48, z=48, storage="f32", steps=64),
    ]


def _logint(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    pick = rng.choice(["vortex", "vortex", "vortex", "duct", "duct", "duct", "ab", "monitor", "les", "scalar", "ensemble",
                       "gradient"])
    if pick == "vortex":
        c = _vortex("", *(_logint(rng, 16, 256) for _ in range(3)), storage=rng.choice(["f32", "f32", "f64", "f16s"]),
                    steps=10, energy=rng.random() < 0.3)
    elif pick == "duct":
        c = _duct("", _logint(rng, 48, 512), _logint(rng, 16, 128), _logint(rng, 16, 128),
                  storage=rng.choice(["f32", "f32", "f16s", "bf16s", "f64"]), coll=rng.choice(["cum", "cum", "srt", "bgk", "mrt"]),
                  steps=rng.choice([10, 20]))
    elif pick == "ab":
        c = _duct("", _logint(rng, 48, 256), _logint(rng, 16, 96), _logint(rng, 16, 96), storage=rng.choice(["f64", "f32"]),
                  steps=10, use="ab")
    elif pick == "monitor":
        c = _duct("", _logint(rng, 64, 400), _logint(rng, 24, 128), _logint(rng, 24, 128), steps=1, use="monitor")
    elif pick == "les":
        c = _duct("", _logint(rng, 64, 400), _logint(rng, 32, 128), _logint(rng, 32, 128), coll="mrt",
                  spheres=rng.randint(3, 20))
    elif pick == "scalar":
        c = _duct("", _logint(rng, 64, 256), _logint(rng, 24, 80), _logint(rng, 24, 80), steps=100, use="scalar")
    elif pick == "ensemble":
        c = dict(kind="ensemble", members=_logint(rng, 16, 256), shapes=rng.randint(1, 1000), steps=50)
    else:
        c = dict(kind="gradient", x=_logint(rng, 64, 192), y=_logint(rng, 24, 56), z=_logint(rng, 24, 56),
                 storage=rng.choice(["f32", "f64"]), steps=rng.choice([16, 36, 64]))
    c.pop("name", None)
    return c


def work(case):
    """Populations in and out once per step (all 27 of every site, the scalar's
    7 with them) and the fields that go to or come from the caller once.  The
    collision takes about 500 operations per site."""
    if case["kind"] == "ensemble":
        sites = sum(a * b * c for a, b, c in _shapes(case))
        return {"bytes": 2.0 * 27 * 4 * sites * case["steps"], "flops": 500.0 * sites * case["steps"]}
    sites = case["x"] * case["y"] * case["z"]
    elem = ELEM[case["storage"]]
    per_step = 2 * 27 * elem
    flops = 500.0
    once = 0
    if case["kind"] == "gradient":
        # forward step with its force; backward step: primal in, FP64 adjoint in and out, force and gradient
        per_step += 24 + 27 * elem + 2 * 27 * 8 + 24 + 48
        flops = 1500.0
    elif case.get("use") == "scalar":
        per_step += 2 * 7 * elem
        flops = 600.0
        once = 5 * 8
    return {"bytes": float(sites) * (per_step * case["steps"] + once), "flops": flops * sites * case["steps"]}


def tolerance(case):
    """Two correct 32-bit evaluations differ by some 1e-8 per step of the
    populations' size, and as slowly growing rounding noise after that; the
    sums and fields follow.  In 16-bit storage a different last bit of the sum
    moves a stored value by one unit of its 11 (8) bits."""
    if case["kind"] == "ensemble":
        return {"rel": 1e-5, "max": 1e-3}
    if case["kind"] == "gradient":
        # the 32-bit primal's velocities carry rounding of 1e-7 / u ~ 1e-5 into the mismatch
        return {"rel": 1e-3, "max": 0.05} if case["storage"] == "f32" else {"rel": 1e-9, "max": 1e-6}
    return {"f64": {"rel": 1e-12, "max": 1e-9}, "f32": {"rel": 1e-5, "max": 1e-3}, "f16s": {"rel": 5e-3, "max": 0.5},
            "bf16s": {"rel": 0.02, "max": 0.9}}[case["storage"]]


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------

def _rand(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _axes(x, y, z):
    return (torch.arange(z, device=DEV, dtype=torch.float64)[:, None, None],
            torch.arange(y, device=DEV, dtype=torch.float64)[None, :, None],
            torch.arange(x, device=DEV, dtype=torch.float64)[None, None, :])


def _vortex_fields(case, seed):
    """Taylor-Green vortex of a seeded phase with 0.1 % noise: rho, vx, vy, vz [Z][Y][X]."""
    x, y, z = case["x"], case["y"], case["z"]
    g = _rand(seed)
    a, b, c = (torch.rand(3, generator=g, device=DEV, dtype=torch.float64) * 2 * math.pi).tolist()
    zz, yy, xx = _axes(x, y, z)
    kx, ky, kz = 2 * math.pi / x, 2 * math.pi / y, 2 * math.pi / z
    px, py, pz = kx * xx + a, ky * yy + b, kz * zz + c
    noise = 1e-3 * U0 * (2 * torch.rand((3, z, y, x), generator=g, device=DEV, dtype=torch.float32).double() - 1)
    # the transverse amplitude kx / ky keeps the field free of divergence; flat boxes keep it below U0
    u0 = U0 * min(1.0, ky / kx)
    vx = u0 * torch.sin(px) * torch.cos(py) * torch.cos(pz) + noise[0]
    vy = -u0 * (kx / ky) * torch.cos(px) * torch.sin(py) * torch.cos(pz) + noise[1]
    rho = 1 + 3 * (u0 * u0 / 16) * (torch.cos(2 * px) + torch.cos(2 * py)) * (torch.cos(2 * pz) + 2)
    return rho.expand(z, y, x).contiguous(), vx, vy, noise[2]


def _vortex_nu(case):
    return U0 * (case["x"] / (2 * math.pi)) / 400.0


def _duct_map(case, seed):
    x, y, z = case["x"], case["y"], case["z"]
    m = np.zeros((z, y, x), np.uint8)
    if case.get("spheres"):
        rng = np.random.default_rng(seed)
        zz, yy, xx = np.ogrid[0:z, 0:y, 0:x]
        for _ in range(case["spheres"]):
            r = rng.uniform(0.06, 0.14) * min(y, z)
            cx, cy, cz = rng.uniform(0.15 * x, 0.8 * x), rng.uniform(0.2 * y, 0.8 * y), rng.uniform(0.2 * z, 0.8 * z)
            m[(xx - cx) ** 2 + (yy - cy) ** 2 + (zz - cz) ** 2 < r * r] = WALL
    m[:, :, 0] = INFLOW if case["kind"] == "gradient" else INFLOW_LEFT
    m[:, :, -1] = OUTFLOW_RIGHT if case.get("use") == "ab" else OUTFLOW_EQ
    m[:, 1, :] = m[:, -2, :] = WALL
    m[1, :, :] = m[-2, :, :] = WALL
    m[:, 0, :] = m[:, -1, :] = NOTHING
    m[0, :, :] = m[-1, :, :] = NOTHING
    return m


def _profile(case):
    """Parabolic inlet velocity between the walls, [Z][Y]."""
    yy = (np.arange(case["y"]) - 1.0) / (case["y"] - 3.0)
    zz = (np.arange(case["z"]) - 1.0) / (case["z"] - 3.0)
    return U_MAX * np.outer(np.clip(4 * zz * (1 - zz), 0, None), np.clip(4 * yy * (1 - yy), 0, None))


def _duct_nu(case):
    # Reynolds number of 400 on the duct's width; the LES collision is run at a higher one
    return U_MAX * (case["y"] - 2) / (2000.0 if case["coll"] == "mrt" else 400.0)


def _duct_fields(case, seed, geo):
    """The inlet profile along the whole duct with 1 % noise, at rest off the fluid."""
    x, y, z = case["x"], case["y"], case["z"]
    fluid = torch.from_numpy(geo).to(DEV) == FLUID
    noise = 0.01 * U_MAX * (2 * torch.rand((3, z, y, x), generator=_rand(seed), device=DEV, dtype=torch.float32).double() - 1)
    prof = torch.from_numpy(_profile(case)).to(DEV)[:, :, None]
    zero = torch.zeros((), device=DEV, dtype=torch.float64)
    return (torch.ones((z, y, x), device=DEV, dtype=torch.float64), torch.where(fluid, prof + noise[0], zero),
            torch.where(fluid, noise[1], zero), torch.where(fluid, noise[2], zero))


def _pulses(case):
    """Eight inlet profiles of one pulse."""
    return [_profile(case) * (1 + 0.1 * math.sin(2 * math.pi * k / 8 + 0.3)) for k in range(8)]


def _scalar_map(geo):
    a = np.zeros_like(geo)
    a[geo == WALL] = 1
    a[geo == INFLOW_LEFT] = 7
    a[geo == OUTFLOW_EQ] = 15
    a[geo == NOTHING] = 10
    return a


def _shapes(case):
    rng = np.random.default_rng(case["shapes"])
    return [tuple(int(v) for v in rng.choice([16, 20, 24, 27, 32], 3)) for _ in range(case["members"])]


def _ensemble_inputs(case, seed):
    rng = np.random.default_rng(seed)
    shapes = _shapes(case)
    nus = [float(U0 * (s[0] / (2 * math.pi)) / r) for s, r in zip(shapes, np.exp(rng.uniform(math.log(50), math.log(800), len(shapes))))]
    return shapes, nus, float(rng.uniform(0.03, 0.05))


def _bumps(case, seed):
    """Body force [3][Z][Y][X] along x: Gaussian bumps of amplitude 1e-4."""
    rng = np.random.default_rng(seed)
    zz, yy, xx = _axes(case["x"], case["y"], case["z"])
    f = torch.zeros((3, case["z"], case["y"], case["x"]), device=DEV, dtype=torch.float64)
    w = case["y"] / 10.0
    for _ in range(8):
        cx, cy, cz = rng.uniform(0.1, 0.9) * case["x"], rng.uniform(0.2, 0.8) * case["y"], rng.uniform(0.2, 0.8) * case["z"]
        f[0] += float(rng.choice([-1.0, 1.0])) * torch.exp(-((xx - cx) ** 2 + (yy - cy) ** 2 + (zz - cz) ** 2) / (2 * w * w))
    return f * (1e-4 / f.abs().max())


def _samples(case, geo):
    """Fluid sites of four cross-sections, and the velocity wanted there."""
    z, y, x = np.nonzero(geo == FLUID)
    keep = np.isin(x, [int(case["x"] * k / 5) for k in (1, 2, 3, 4)])
    idx = ((z * case["y"] + y) * case["x"] + x)[keep].astype(np.int64)
    target = np.zeros((len(idx), 4))
    target[:, 0] = 1.0
    target[:, 1] = 0.5 * U_MAX
    return idx, target


# --------------------------------------------------------------------------
# prepare and run
# --------------------------------------------------------------------------

def _host(fields):
    return [f.cpu().numpy() for f in fields]


def _populations(lat, case):
    """The lattice's populations in place: [27][Z][Y][X], without the ghost layer."""
    t = lat.populations_tensor()
    x0 = lat.device_view().x0
    t = t[:, 1:1 + case["z"], 1:1 + case["y"], x0:x0 + case["x"]]
    t.lattice = lat  # the memory is the lattice's own: it lives as long as the view
    return t


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        shapes, nus, u0 = _ensemble_inputs(case, seed)
        ens = pl.Ensemble(shapes, nus, cum_flags=3)
        ens.init_taylor_green(u0)
        ens.autotune()
        return {"case": case, "ens": ens}
    x, y, z = case["x"], case["y"], case["z"]
    st = STORAGE[case["storage"]]
    if kind == "vortex":
        lat = pl.LBM(x, y, z, viscosity=_vortex_nu(case), cum_flags=3, storage=st, periodic=True)
        lat.init_equilibrium(*_host(_vortex_fields(case, seed)))
        lat.autotune()
        return {"case": case, "lat": lat, "pop": _populations(lat, case)}
    geo = _duct_map(case, seed)
    if kind == "gradient":
        lat = pl.LBM(x, y, z, viscosity=0.02, collision=pl.COLL_SRT, equilibrium=pl.EQ_SECOND_ORDER, storage=st)
        lat.set_map(geo)
        lat.set_inflow(_profile(case))
        idx, target = _samples(case, geo)
        force = _bumps(case, seed)
        return {"case": case, "lat": lat, "force": force, "grad": torch.empty_like(force), "samples": idx, "target": target}
    lat = pl.LBM(x, y, z, viscosity=_duct_nu(case), collision=COLL[case["coll"]],
                 equilibrium=pl.EQ_INV_CUM if case["coll"] == "cum" else pl.EQ_SECOND_ORDER, storage=st)
    if case["use"] == "ab":
        lat.set_streaming(pl.STREAMING_AB)
    lat.set_map(geo)
    lat.set_inflow(_profile(case))
    lat.init_equilibrium(*_host(_duct_fields(case, seed, geo)))
    if case["use"] == "scalar":
        lat.ade_enable(_duct_nu(case), collision=pl.ADE_CLBM, inflow_phi=1.0)
        lat.ade_set_map(_scalar_map(geo))
        lat.ade_init_equilibrium(uniform_phi=0.0)
        lat.set_kernel(pl.KERNEL_PAIR)
    else:
        lat.autotune()
    return {"case": case, "lat": lat, "pop": _populations(lat, case), "pulses": _pulses(case), "pass": 0}


def run(state):
    case = state["case"]
    kind, steps = case["kind"], case["steps"]
    if kind == "ensemble":
        ens = state["ens"]
        ens.step(steps, sums=True)
        return {"sums": ens.sums(), "last": ens.get_populations(len(ens) - 1, layout=pl.LAYOUT_INTERIOR, dtype=np.float32)}
    lat = state["lat"]
    if kind == "gradient":
        lat.init_equilibrium()
        loss = lat.adjoint_forward(state["force"], steps, state["samples"], state["target"])
        return {"loss": loss, "grad": lat.adjoint_backward(out=state["grad"])}
    if kind == "vortex" and case["energy"]:
        lat.step(steps, sums=True)
        return {"energy": pl.kinetic_energy(lat), "pop": state["pop"]}
    if case.get("use") == "monitor":
        lat.set_inflow(state["pulses"][state["pass"] % 8])
        state["pass"] += 1
        lat.step(1, sums=True)
        return {"sums": lat.sums()[:5], "pop": state["pop"]}
    if case.get("use") == "scalar":
        lat.step(steps, macro=True)
        return {"phi": lat.ade_phi(), "macro": lat.macro(), "pop": state["pop"]}
    lat.step(steps)
    return {"pop": state["pop"]}


# --------------------------------------------------------------------------
# the same passes in 64 bits, as plain tensor code
# --------------------------------------------------------------------------

C = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0), (1, -1, 0),
     (-1, 1, 0), (1, 0, 1), (-1, 0, -1), (1, 0, -1), (-1, 0, 1), (0, 1, 1), (0, -1, -1), (0, 1, -1), (0, -1, 1), (1, 1, 1),
     (-1, -1, -1), (1, 1, -1), (-1, -1, 1), (1, -1, 1), (-1, 1, -1), (1, -1, -1), (-1, 1, 1)]
OPP = [C.index((-a, -b, -c)) for a, b, c in C]
W = [(8 / 27, 2 / 27, 1 / 54, 1 / 216)[abs(a) + abs(b) + abs(c)] for a, b, c in C]


def _moments(f):
    rho = sum(f)
    mom = [sum(f[q] * C[q][k] for q in range(27) if C[q][k]) for k in range(3)]
    return rho, mom


def _equilibrium(kind, rho, u):
    if kind == "second":
        usq = u[0] * u[0] + u[1] * u[1] + u[2] * u[2]
        out = []
        for q in range(27):
            cu = sum(C[q][k] * u[k] for k in range(3))
            out.append(W[q] * rho * (1 - 1.5 * usq + 3 * cu + 4.5 * cu * cu))
        return out
    axis = [{0: 2 / 3 - v * v, 1: (1 / 3 + v + v * v) / 2, -1: (1 / 3 - v + v * v) / 2} for v in u]
    return [rho * axis[0][c[0]] * axis[1][c[1]] * axis[2][c[2]] for c in C]


def _central(m, u, back):
    """Central moments of a 3 x 3 x 3 cube of populations, axis by axis, or back."""
    m = dict(m)
    for axis in ((0, 1, 2) if back else (2, 1, 0)):
        v = u[axis]
        for i in range(3):
            for j in range(3):
                key = [(i, j)[:axis] + (k,) + (i, j)[axis:] for k in range(3)]
                a, b, c = (m[k] for k in key)
                if back:
                    m[key[0]] = (a * (v * v - v) + b * (2 * v - 1) + c) / 2
                    m[key[1]] = a * (1 - v * v) - 2 * v * b - c
                    m[key[2]] = (a * (v * v + v) + b * (2 * v + 1) + c) / 2
                else:
                    m[key[0]] = a + b + c
                    m[key[1]] = a * (-1 - v) - b * v + c * (1 - v)
                    m[key[2]] = a * (1 + v) ** 2 + b * v * v + c * (1 - v) ** 2
    return m


def _cumulant(f, rho, u, nu, full):
    """The cumulant collision (Geier 2015) with omega2 = 1; `full`: with the
    limited third-order rates and the fourth-order terms of Geier 2017, whose
    trace is that of the density deviation."""
    m = _central({(C[q][0] + 1, C[q][1] + 1, C[q][2] + 1): f[q] for q in range(27)}, u, False)
    w = 1 / (0.5 + 3 * nu)
    ir = 1 / rho
    x2, y2, z2 = u[0] ** 2, u[1] ** 2, u[2] ** 2
    c110, c101, c011 = m[1, 1, 0], m[1, 0, 1], m[0, 1, 1]
    c200, c020, c002 = m[2, 0, 0], m[0, 2, 0], m[0, 0, 2]
    zero = torch.zeros_like(rho)
    dx = dy = dz = zero
    k120 = k102 = k210 = k012 = k201 = k021 = k111 = zero
    f220 = f202 = f022 = f211 = f121 = f112 = zero
    if full:
        dx = -w / 2 * ir * (2 * c200 - c020 - c002) - 0.5 * ir * (c200 + c020 + c002 - (rho - 1))
        dy = dx + 1.5 * w * ir * (c200 - c020)
        dz = dx + 1.5 * w * ir * (c200 - c002)
    a, b, c = (1 - w) * c110, (1 - w) * c101, (1 - w) * c011
    e1 = (1 - w) * (c200 - c020) - 3 * (1 - w / 2) * rho * (x2 * dx - y2 * dy)
    e2 = (1 - w) * (c200 - c002) - 3 * (1 - w / 2) * rho * (x2 * dx - z2 * dz)
    e3 = m[0, 0, 0] - 1.5 * rho * (x2 * dx + y2 * dy + z2 * dz)
    p, q, r = (e1 + e2 + e3) / 3, (e2 + e3 - 2 * e1) / 3, (e1 + e3 - 2 * e2) / 3
    if full:
        w3 = 8 * (w - 2) * (3 * w - 1 - 5 * w) / (8 * (5 - 2 * w) * w + 8 + w * (9 * w - 26))
        w4 = 8 * (w - 2) * (4 * w - 7) / (56 - 50 * w + 9 * w * w)
        w5 = (24 * (w - 2) * (4 * w * w + w * (18 - 13 * w) + 2 + w * (6 * w - 11))
              / (16 * w * w * (w - 6) - 2 * w * (216 + 5 * w * (9 * w - 46)) + w * (3 * w - 10) * (15 * w - 28) - 48))
        den = (w - 1) * (2 + 3 * w - 8 * w)
        ca = (4 * w * w + 2 * w * (w - 6) + w * (10 - 3 * w) - 4) / den
        cb = (4 * w * (9 * w - 16) - 4 * w * w - 2 * (2 + 9 * w * (w - 2))) / (3 * den)
        g = 1 / w - 0.5

        def limited(rate, v):
            return (1 - (rate + (1 - rate) * v.abs() / (0.01 * rho + v.abs()))) * v

        def pair(v, t):
            s, d = limited(w3, v + t), limited(w4, v - t)
            return (s + d) / 2, (s - d) / 2

        k120, k102 = pair(m[1, 2, 0], m[1, 0, 2])
        k210, k012 = pair(m[2, 1, 0], m[0, 1, 2])
        k201, k021 = pair(m[2, 0, 1], m[0, 2, 1])
        k111 = limited(w5, m[1, 1, 1])
        e4 = 2 / 3 * g * ca * rho * (dx - 2 * dy + dz)
        e5 = 2 / 3 * g * ca * rho * (dx + dy - 2 * dz)
        e6 = -4 / 3 * g * ca * rho * (dx + dy + dz)
        f220, f202, f022 = (e4 + e5 + e6) / 3, (e6 - e4) / 3, (e6 - e5) / 3
        # the mixed derivatives are -3 w k / rho
        f211, f121, f112 = (g * cb * w * v for v in (c011, c101, c110))
    n = dict.fromkeys(m, zero)
    n[0, 0, 0] = m[0, 0, 0]
    n[1, 0, 0], n[0, 1, 0], n[0, 0, 1] = -m[1, 0, 0], -m[0, 1, 0], -m[0, 0, 1]
    n[1, 1, 0], n[1, 0, 1], n[0, 1, 1], n[2, 0, 0], n[0, 2, 0], n[0, 0, 2] = a, b, c, p, q, r
    n[1, 2, 0], n[1, 0, 2], n[2, 1, 0], n[0, 1, 2], n[2, 0, 1], n[0, 2, 1], n[1, 1, 1] = k120, k102, k210, k012, k201, k021, k111
    n[2, 1, 1] = f211 + (p * c + 2 * b * a) * ir
    n[1, 2, 1] = f121 + (q * b + 2 * a * c) * ir
    n[1, 1, 2] = f112 + (r * a + 2 * c * b) * ir
    n[2, 2, 0] = f220 + (q * p + 2 * a * a) * ir
    n[0, 2, 2] = f022 + (r * q + 2 * c * c) * ir
    n[2, 0, 2] = f202 + (p * r + 2 * b * b) * ir
    n[1, 2, 2] = (q * k102 + r * k120 + 4 * c * k111 + 2 * (a * k012 + b * k021)) * ir
    n[2, 1, 2] = (r * k210 + p * k012 + 4 * b * k111 + 2 * (c * k201 + a * k102)) * ir
    n[2, 2, 1] = (p * k021 + q * k201 + 4 * a * k111 + 2 * (b * k120 + c * k210)) * ir
    n[2, 2, 2] = ((4 * k111 * k111 + p * n[0, 2, 2] + q * n[2, 0, 2] + r * n[2, 2, 0]
                   + 4 * (c * n[2, 1, 1] + b * n[1, 2, 1] + a * n[1, 1, 2]) + 2 * (k120 * k102 + k210 * k012 + k201 * k021)) * ir
                  - (16 * a * b * c + 4 * (b * b * q + c * c * p + a * a * r) + 2 * p * q * r) * ir * ir)
    n = _central(n, u, True)
    return [n[C[i][0] + 1, C[i][1] + 1, C[i][2] + 1] for i in range(27)]


def _srt(f, rho, u, nu, force=None):
    tau = 3 * nu + 0.5
    eq = _equilibrium("second", rho, u)
    out = []
    for q in range(27):
        v = f[q] + (eq[q] - f[q]) / tau
        if force is not None:
            v = v + (1 - 0.5 / tau) * 3 * sum((C[q][k] - u[k]) * force[k] for k in range(3)) / rho * eq[q]
        out.append(v)
    return out


def _bgk(f, rho, u, nu):
    w = 1 / (0.5 + 3 * nu)
    eq = _equilibrium("product", rho, u)
    return [f[q] + (eq[q] - f[q]) * w for q in range(27)]


def _mrt(f, rho, u, nu):
    """LES: the second moments relaxed with a Smagorinsky rate, the rest at equilibrium."""
    tau = 3 * nu + 0.5
    pi = {(i, j): sum(f[q] * (C[q][i] * C[q][j]) for q in range(27) if C[q][i] * C[q][j]) for i in range(3) for j in range(i, 3)}
    neq = {k: v - rho * ((1 / 3 if k[0] == k[1] else 0) + u[k[0]] * u[k[1]]) for k, v in pi.items()}
    size = 2 * sum((1 if i == j else 2) * neq[i, j] ** 2 for i, j in neq)
    rate = 2 / (torch.sqrt(tau * tau + 2 * 0.0342 * 9 * torch.sqrt(size) / rho) + tau)
    pi = {k: pi[k] - rate * neq[k] for k in pi}
    trace = pi[0, 0] + pi[1, 1] + pi[2, 2]
    out = []
    for q in range(27):
        cu = sum(C[q][k] * u[k] for k in range(3))
        cc = sum((1 if i == j else 2) * C[q][i] * C[q][j] * pi[i, j] for i, j in pi)
        out.append(W[q] * (rho * (2.5 - 1.5 * sum(v * v for v in C[q]) + 3 * cu) + 4.5 * cc - 1.5 * trace))
    return out


def _collide(case, f, rho, u):
    if case["kind"] == "vortex":
        return _cumulant(f, rho, u, _vortex_nu(case), True)
    nu = _duct_nu(case)
    if case["coll"] == "cum":
        return _cumulant(f, rho, u, nu, False)
    return {"srt": _srt, "bgk": _bgk, "mrt": _mrt}[case["coll"]](f, rho, u, nu)


def _inlet(f, u):
    """Moment inlet (Eichler et al.) on the left: density and the nine directions that enter."""
    def s(x, y=None, z=None):
        return sum(f[q] for q in range(27) if C[q][0] == x and (y is None or C[q][1] == y) and (z is None or C[q][2] == z))
    rho = (s(0) + 2 * s(-1)) / (1 - u[0])
    f = list(f)
    m = {(b, c): rho * ((1, u[1], 1 / 3 + u[1] ** 2)[b] * (1, u[2], 1 / 3 + u[2] ** 2)[c]) for b in range(3) for c in range(3)}
    m10 = rho * u[0]
    new = {}
    for b in (1, -1):
        new[b, 0] = 0.5 * (m[2, 0] - m[2, 2] + b * (m[1, 0] - m[1, 2]))
        new[0, b] = 0.5 * (m[0, 2] - m[2, 2] + b * (m[0, 1] - m[2, 1]))
        for c in (1, -1):
            new[b, c] = 0.25 * (m[2, 2] + b * c * m[1, 1] + c * m[2, 1] + b * m[1, 2])
    for (b, c), v in new.items():
        f[C.index((1, b, c))] = v - (f[C.index((-1, b, c))] + f[C.index((0, b, c))])
    rest = sum(f[C.index((0, b, c))] for b in (-1, 0, 1) for c in (-1, 0, 1) if b or c)
    left = sum(f[C.index((-1, b, c))] for b in (-1, 0, 1) for c in (-1, 0, 1) if b or c)
    f[1] = m10 + (m[2, 2] - (m[2, 0] + m[0, 2])) + f[2] + rest + 2 * left
    return rho, f


def _site(case, geo, f, inlet, force=None):
    """Boundary treatment and collision of all sites: populations out, density and velocity."""
    rho, mom = _moments(f)
    if force is not None:
        mom = [mom[k] + 0.5 * force[k] for k in range(3)]
    u = [v / rho for v in mom]
    gradient = case["kind"] == "gradient"
    if geo is None:
        return _collide(case, f, rho, u), rho, u
    zero, one = torch.zeros_like(rho), torch.ones_like(rho)
    uin = [inlet.expand_as(rho), zero, zero]
    is_in = geo == (INFLOW if gradient else INFLOW_LEFT)
    if not gradient:
        r_in, f_in = _inlet(f, uin)
        f = [torch.where(is_in, a, b) for a, b in zip(f_in, f)]
        rho = torch.where(is_in, r_in, rho)
        u = [torch.where(is_in, a, b) for a, b in zip(uin, u)]
    eq = "product" if not gradient and case["coll"] == "cum" else "second"
    out = geo == OUTFLOW_RIGHT
    rho = torch.where(out, one, rho)
    new = _srt(f, rho, u, 0.02, force) if gradient else _collide(case, f, rho, u)
    wall, out = geo == WALL, geo == OUTFLOW_EQ
    f_out = _equilibrium(eq, one, u)
    new = [torch.where(wall, f[OPP[q]], torch.where(out, f_out[q], new[q])) for q in range(27)]
    if gradient:
        f_in = _equilibrium(eq, one, uin)
        new = [torch.where(is_in, a, b) for a, b in zip(f_in, new)]
        u = [torch.where(is_in, a, b) for a, b in zip(uin, u)]
    still = wall | (geo == NOTHING)
    rho = torch.where(still | out | (is_in if gradient else still), one, rho)
    u = [torch.where(still, zero, v) for v in u]
    return new, rho, u


def _scalar_site(case, kind, g, u):
    """The D3Q7 scalar with central-moment collision: populations out and phi."""
    w = 1 / (0.5 + 4 * _duct_nu(case))
    phi = sum(g)
    one = [(phi * u[k] + g[2 * k + 2] - g[2 * k + 1]) * w for k in range(3)]
    two = [phi * (0.25 - u[k] ** 2) + 2 * u[k] * (g[2 * k + 1] - g[2 * k + 2]) - g[2 * k + 2] - g[2 * k + 1] for k in range(3)]
    new = [g[0] - 2 * sum(one[k] * u[k] for k in range(3)) - sum(two)]
    for k in range(3):
        new += [g[2 * k + 1] + one[k] * u[k] + 0.5 * (two[k] + one[k]), g[2 * k + 2] + one[k] * u[k] + 0.5 * (two[k] - one[k])]
    wall, inlet, mirror = kind == 1, kind == 7, kind == 15
    usq = sum(v * v for v in u)
    held = list(g)
    held[2] = g[1]
    for q in range(7):
        cu = sum(C[q][k] * u[k] for k in range(3))
        at = (0.25 if q == 0 else 0.125) * (1 - 2 * usq + 4 * cu + 8 * cu * cu)
        new[q] = torch.where(wall, g[OPP[q]], torch.where(inlet, at, torch.where(mirror, held[q], new[q])))
    phi = torch.where(inlet, torch.ones_like(phi), torch.where(mirror, sum(held), phi))
    return new, torch.where(kind == 10, torch.zeros_like(phi), phi)


def _shift(t, c):
    """Values of t moved by c (x, y, z), wrapping."""
    return torch.roll(t, (c[2], c[1], c[0]), (0, 1, 2)) if any(c) else t


def _gather(slots, odd):
    """Directions at each site from the A-A slots."""
    n = len(slots)
    return [_shift(slots[OPP[q]], C[q]) for q in range(n)] if odd else list(slots)


def _scatter(slots, new, odd, active):
    """A-A slots after the sites' new directions; sites that are not active keep theirs."""
    n = len(slots)
    if odd:
        moved = [_shift(new[q], C[q]) for q in range(n)]
        return moved if active is None else [torch.where(_shift(active, C[q]), moved[q], slots[q]) for q in range(n)]
    return [new[OPP[q]] if active is None else torch.where(active, new[OPP[q]], slots[q]) for q in range(n)]


def _padded(t, value):
    return torch.nn.functional.pad(t, (1,) * 6, value=value)


def _inner(t):
    return t[1:-1, 1:-1, 1:-1]


def _start(case, fields, pad):
    kind = "product" if case["kind"] == "vortex" or case.get("coll") == "cum" else "second"
    if pad:
        fields = [_padded(v, 1.0 if k == 0 else 0.0) for k, v in enumerate(fields)]
    return _equilibrium(kind, fields[0], fields[1:])


def _stored(case, slots):
    """The populations as the storage keeps them, without its rounding."""
    t = torch.stack(slots)
    w = torch.tensor(W, device=t.device, dtype=t.dtype)[:, None, None, None]
    if case["storage"] == "f16s":
        scale = torch.tensor([(4.0, 16.0, 64.0, 256.0)[sum(abs(v) for v in c)] for c in C], device=t.device, dtype=t.dtype)
        return (t - w) * scale[:, None, None, None]
    return t - w if case["storage"] == "bf16s" else t


def _sums(rho, u):
    return [float(v.sum()) for v in (rho, rho * u[0], rho * u[1], rho * u[2], rho * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2))]


def _vortex_run(case, slots, steps, nu=None):
    rho = u = None
    for t in range(steps):
        f = _gather(slots, t % 2 == 1)
        if nu is None:
            new, rho, u = _site(case, None, f, None)
        else:
            rho, mom = _moments(f)
            u = [v / rho for v in mom]
            new = _cumulant(f, rho, u, nu, True)
        slots = _scatter(slots, new, t % 2 == 1, None)
    return slots, rho, u


def _exact_ensemble(case, seed):
    shapes, nus, u0 = _ensemble_inputs(case, seed)
    rows = []
    for (x, y, z), nu in zip(shapes, nus):
        zz, yy, xx = _axes(x, y, z)
        kx, ky, kz = 2 * math.pi / x, 2 * math.pi / y, 2 * math.pi / z
        px, py, pz = kx * (xx + 0.5 - 0.5 * x), ky * (yy + 0.5 - 0.5 * y), kz * (zz + 0.5 - 0.5 * z)
        vx = u0 * torch.sin(px) * torch.cos(py) * torch.cos(pz)
        vy = -u0 * (kx / ky) * torch.cos(px) * torch.sin(py) * torch.cos(pz)
        rho = 1 + 3 * (u0 * u0 / 16) * (torch.cos(2 * px) + torch.cos(2 * py)) * (torch.cos(2 * pz) + 2)
        slots = _equilibrium("product", rho, [vx, vy, torch.zeros_like(vx)])
        slots, rho, u = _vortex_run(case, slots, case["steps"], nu)
        rows.append(_sums(rho, u) + [0.0])
    return {"sums": np.array(rows), "last": torch.stack(slots)}


def _exact_gradient(case, seed):
    geo = _duct_map(case, seed)
    idx, target = _samples(case, geo)
    force = _bumps(case, seed).requires_grad_(True)
    g = _padded(torch.from_numpy(geo).to(DEV), NOTHING)
    active = g != NOTHING
    inlet = torch.nn.functional.pad(torch.from_numpy(_profile(case)).to(DEV), (1, 1, 1, 1))[:, :, None]
    one = torch.ones(tuple(n + 2 for n in geo.shape), device=DEV, dtype=torch.float64)
    slots = torch.stack(_equilibrium("second", one, [0 * one] * 3))

    def step(s, f, odd):
        pad = [_padded(f[k], 0.0) for k in range(3)]
        new, _, _ = _site(case, g, _gather(list(s), odd), inlet, pad)
        return torch.stack(_scatter(list(s), new, odd, active))

    for t in range(case["steps"]):
        slots = torch.utils.checkpoint.checkpoint(step, slots, force, t % 2 == 1, use_reentrant=False)
    f = [_inner(v).reshape(-1)[torch.from_numpy(idx).to(DEV)] for v in _gather(list(slots), case["steps"] % 2 == 1)]
    rho, mom = _moments(f)
    at = force.reshape(3, -1)[:, torch.from_numpy(idx).to(DEV)]
    want = torch.from_numpy(target).to(DEV)
    loss = 0.5 * sum((((mom[k] + 0.5 * at[k]) / rho - want[:, k + 1]) ** 2).sum() for k in range(3))
    (grad,) = torch.autograd.grad(loss, force)
    return {"loss": float(loss.detach()), "grad": grad}


def _exact_pull(case, seed):
    """A-B: every site pulls from its clamped neighbours; the outlet pulls from x - 1 in every direction."""
    host = _duct_map(case, seed)
    geo = torch.from_numpy(host).to(DEV)
    slots = _start(case, _duct_fields(case, seed, host), False)
    inlet = torch.from_numpy(_profile(case)).to(DEV)[:, :, None]
    last = torch.arange(case["x"], device=DEV) == case["x"] - 1
    at = [torch.arange(n, device=DEV) for n in geo.shape]
    for _ in range(case["steps"]):
        f = []
        for q, c in enumerate(C):
            iz, iy = ((at[k] - c[2 - k]).clamp(0, geo.shape[k] - 1) for k in (0, 1))
            ix = torch.where(last & (case["x"] > 1), at[2] - 1, (at[2] - c[0]).clamp(0, case["x"] - 1))
            out = slots[q].index_select(0, iz).index_select(1, iy)
            edge = geo[:, :, -1:] == OUTFLOW_RIGHT
            v = out.index_select(2, ix)
            v = torch.cat([v[:, :, :-1], torch.where(edge, v[:, :, -1:], slots[q].index_select(0, iz).index_select(1, iy)
                           .index_select(2, (at[2][-1:] - c[0]).clamp(0, case["x"] - 1)))], 2)
            f.append(v)
        new, _, _ = _site(case, geo, f, inlet)
        slots = [torch.where(geo != NOTHING, new[q], slots[q]) for q in range(27)]
    return {"pop": _stored(case, slots)}


def exact(case, seed):
    kind, steps = case["kind"], case["steps"]
    if kind == "gradient":
        return _exact_gradient(case, seed)
    with torch.no_grad():
        if kind == "ensemble":
            return _exact_ensemble(case, seed)
        if case.get("use") == "ab":
            return _exact_pull(case, seed)
        if kind == "vortex":
            slots, rho, u = _vortex_run(case, _start(case, _vortex_fields(case, seed), False), steps)
            out = {"pop": _stored(case, slots)}
            if case["energy"]:
                out["energy"] = _sums(rho, u)[4] / 2 / (case["x"] * case["y"] * case["z"])
            return out
        host = _duct_map(case, seed)
        geo = _padded(torch.from_numpy(host).to(DEV), NOTHING)
        active = geo != NOTHING
        slots = _start(case, _duct_fields(case, seed, host), True)
        prof = _pulses(case)[0] if case["use"] == "monitor" else _profile(case)
        inlet = torch.nn.functional.pad(torch.from_numpy(prof).to(DEV), (1, 1, 1, 1))[:, :, None]
        scalar = case["use"] == "scalar"
        if scalar:
            kinds = _padded(torch.from_numpy(_scalar_map(host)).to(DEV), 10)
            moves = kinds != 10
            g = [torch.zeros_like(slots[0]) for _ in range(7)]
        for t in range(steps):
            new, rho, u = _site(case, geo, _gather(slots, t % 2 == 1), inlet)
            if scalar:
                grown, phi = _scalar_site(case, kinds, _gather(g, t % 2 == 1), u)
                g = _scatter(g, grown, t % 2 == 1, moves)
            slots = _scatter(slots, new, t % 2 == 1, active)
        out = {"pop": _stored(case, [_inner(v) for v in slots])}
        if case["use"] == "monitor":
            out["sums"] = np.array(_sums(_inner(rho), [_inner(v) for v in u]))
        if scalar:
            out["phi"] = _inner(phi)
            out["macro"] = torch.stack([_inner(rho)] + [_inner(v) for v in u])
        return out
