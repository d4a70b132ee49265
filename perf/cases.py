"""Workloads of the unsplit hydro solver for performance measurement.

Every case is a stretch of a simulation as a driver program runs it through
`HydroDevice`: the state goes to the device, some steps run, the state comes
back.  Uniform grids take their state from the host UNK (`put_interior`,
`get_interior`: what a program does around a checkpoint, a plot file or a host
physics unit); AMR meshes take it from leaf messages on the device
(`unpack_leaves`, `pack_leaves`).  In between, `how` says who drives:

  advance   the on-device driver loop (`advance`)
  driver    the host driver loop, `Hydro` and `Hydro_computeDt` every step
  host      as `driver`, with the state going to the host and back every step

The library holds one grid, so the states of one case share its device, the
way a program keeps it over a run.

`exact` restates the step in plain torch in 64 bits.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (ROOT, os.path.join(ROOT, "flash-x_b200")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

from flashx_b200 import amr as A  # noqa: E402
from flashx_b200.hydro import LEAF_MSG_VARS, HydroDevice, driver_dt  # noqa: E402
from flashx_b200.params import (BC_OUTFLOW, BC_PERIODIC, BC_REFLECTING, Geometry, HydroParams,  # noqa: E402
                                NUNK, UNK_VARS)

G = 4                                   # guard layers
BCS = {"p": BC_PERIODIC, "o": BC_OUTFLOW, "r": BC_REFLECTING}
SLOT = {v: UNK_VARS.index(v) for v in LEAF_MSG_VARS}


def _ug(name, problem, n, blocks, prec, steps, how="advance", order=3, riemann="HLLC", limiter="mc", bc="ppp",
        gravity=False):
    """A uniform grid of blocks of n cells a side."""
    return {"name": name, "grid": "ug", "ndim": len(blocks), "problem": problem, "n": n, "bx": blocks[0],
            "by": blocks[1], "bz": blocks[2] if len(blocks) == 3 else 1, "prec": prec, "steps": steps, "how": how,
            "order": order, "riemann": riemann, "limiter": limiter, "bc": bc, "gravity": gravity, "maxlev": 1}


def _amr(name, n, roots, maxlev, prec, steps, how="advance", order=3, riemann="HLLC", limiter="mc"):
    """A mesh refined around the seeded level-set interface, periodic."""
    return {"name": name, "grid": "amr", "ndim": 3, "problem": "levelset", "n": n, "bx": roots[0], "by": roots[1],
            "bz": roots[2], "prec": prec, "steps": steps, "how": how, "order": order, "riemann": riemann,
            "limiter": limiter, "bc": "ppp", "gravity": False, "maxlev": maxlev}


def listed():
    return [
        # the smallest call: a shock tube of four blocks stepped by the host's
        # driver loop, all launches and synchronisations
        _ug("sod2d_32_driver", "sod", 16, (2, 2), "fp64", 20, how="driver", bc="ooo"),
        # the shock tube benchmark at its size, many small steps on the device
        _ug("sod2d_256", "sod", 16, (16, 16), "fp64", 100, bc="ooo"),
        # a host physics unit touches UNK after every step
        _ug("kh2d_512_host", "kh", 16, (32, 32), "fp64", 4, how="host"),
        # the Kelvin-Helmholtz benchmark in both precisions
        _ug("kh2d_2048", "kh", 16, (128, 128), "fp64", 100),
        _ug("kh2d_2048_mixed", "kh", 16, (128, 128), "mixed", 100),
        # WENO5 on a ragged 2-D grid, reflecting walls in y
        _ug("gas2d_weno_816x624", "gas", 16, (51, 39), "fp64", 40, order=5, bc="prp"),
        # a small 3-D box
        _ug("gas3d_32", "gas", 16, (2, 2, 2), "fp64", 40),
        # the Rayleigh-Taylor benchmark's setup (WENO5, gravity, full CTU)
        _ug("rt3d_128", "rt", 16, (8, 8, 8), "fp64", 20, order=5, bc="ppr", gravity=True),
        _ug("rt3d_192_mixed", "rt", 32, (6, 6, 6), "mixed", 20, order=5, bc="ppr", gravity=True),
        # PPM in 3-D on unequal, odd extents
        _ug("gas3d_ppm_136x88x120", "gas", 8, (17, 11, 15), "fp64", 20, limiter="vanLeer", bc="por"),
        # a small AMR mesh driven from the host, and the AMR benchmark's mesh
        _amr("amr_small_driver", 16, (2, 2, 2), 2, "fp64", 10, how="driver"),
        _amr("amr_5230_mixed", 16, (4, 4, 4), 4, "mixed", 6),
    ]


def draw(rng):
    """One more case of the same ranges."""
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    prec = rng.choice(("fp64", "fp64", "mixed"))
    order = rng.choice((3, 3, 5))
    riemann = rng.choice(("HLLC", "HLLC", "HLL"))
    limiter = rng.choice(("mc", "mc", "vanLeer", "minmod"))
    how = rng.choice(("advance", "advance", "advance", "driver"))
    kind = rng.choice(("2d", "2d", "3d", "3d", "amr"))
    if kind == "2d":
        blocks = (logint(2, 128), logint(2, 128))
        zones = 256 * blocks[0] * blocks[1]
        steps = max(4, min(100, int(4e8 * (0.5 if order == 5 else 1.0) / zones)))
        bc = rng.choice(("ppp", "ooo", "prp", "rop"))
        problem = "kh" if bc == "ppp" and rng.random() < 0.5 else ("sod" if bc == "ooo" else "gas")
        if problem == "gas":            # HLL is not stable on grid-scale noise at this CFL number
            riemann = "HLLC"
        return {k: v for k, v in _ug("", problem, 16, blocks, prec, steps, how, order, riemann, limiter, bc).items()
                if k != "name"}
    if kind == "3d":
        n = rng.choice((8, 16, 16, 32))
        most = (96 if n == 8 else 160) // n
        blocks = tuple(logint(max(1, 16 // n), most) for _ in range(3))
        zones = n ** 3 * blocks[0] * blocks[1] * blocks[2]
        steps = max(2, min(40, int(6e7 / zones)))
        gravity = rng.random() < 0.4
        bc = "ppr" if gravity else rng.choice(("ppp", "por", "ooo"))
        return {k: v for k, v in _ug("", "rt" if gravity else "gas", n, blocks, prec, steps, how, order, "HLLC",
                                     limiter, bc, gravity).items() if k != "name"}
    n = rng.choice((8, 16, 16))
    roots = (rng.randint(2, 3), rng.randint(2, 4), rng.randint(2, 3))
    return {k: v for k, v in _amr("", n, roots, rng.randint(2, 3), prec, rng.randint(2, 6), how, order, "HLLC",
                                  limiter).items() if k != "name"}


# ------------------------------------------------------------------- set-up
def _geometry(c):
    bc = tuple(BCS[c["bc"][a]] for a in (0, 0, 1, 1, 2, 2))
    # cubic cells, except where the problem's length scale is the box
    box = c["problem"] in ("rt", "sod", "kh")
    ext = [1.0 if box else c[k] / c["bx"] for k in ("bx", "by", "bz")]
    return Geometry(c["ndim"], c["n"], c["n"], c["n"] if c["ndim"] == 3 else 1, c["bx"], c["by"], c["bz"],
                    bbox=tuple((0.0, e) for e in ext), bc=bc, nguard=G)


def _params(c):
    return HydroParams(order=c["order"], RiemannSolver=c["riemann"], slopeLimiter=c["limiter"],
                       gamma=5.0 / 3.0 if c["problem"] == "gas" else 1.4, useGravity=bool(c["gravity"]),
                       gravity=(0.0, 0.0, -0.1) if c["gravity"] else (0.0, 0.0, 0.0))


_meshes = {}


def _mesh(c):
    key = (c["n"], c["bx"], c["by"], c["bz"], c["maxlev"])
    if key not in _meshes:
        geom = _geometry(c)
        rho = A.levelset_density(geom, c["maxlev"])
        _meshes[key] = A.build_mesh(geom, c["maxlev"], A.gradient_refine(geom, rho))
    return _meshes[key]


def _primitives(c, seed, X, Y, Z, dfine):
    """Seeded density, velocities and pressure at the coordinates X, Y, Z
    (broadcastable torch tensors)."""
    rng = np.random.default_rng(seed)
    dev = X.device
    shape = torch.broadcast_shapes(X.shape, Y.shape, Z.shape)
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(rng.integers(1 << 40)))

    def noise():
        return torch.randn(shape, generator=gen, device=dev, dtype=torch.float64)

    one = torch.ones(shape, dtype=torch.float64, device=dev)
    zero = torch.zeros_like(one)
    if c["problem"] == "sod":           # a shock tube at 45 degrees, slightly perturbed states
        a = rng.uniform(-0.05, 0.05, 4)
        left = (X + Y + zero) < 1.0 + a[0]
        rho = torch.where(left, one * (1.0 + a[1]), one * 0.125)
        p = torch.where(left, one * (1.0 + a[2]), one * (0.1 + 0.1 * a[3]))
        return rho, zero, zero, zero, p
    if c["problem"] == "kh":            # a periodic shear layer with noisy vy
        inner = (Y - 0.5 + zero).abs() < 0.25
        rho = torch.where(inner, 2.0 * one, one)
        vx = torch.where(inner, 0.5 * one, -0.5 * one)
        vy = 0.01 * noise().clamp(-2, 2) * torch.sin(4.0 * math.pi * X)
        return rho, vx, vy, zero, 2.5 * one
    if c["problem"] == "rt":            # heavy over light gas, random modes at the interface
        heavy = (Z + zero) > 0.5
        rho = torch.where(heavy, 2.0 * one, one)
        p = 2.5 - 0.1 * rho * (Z - 0.5)
        s = zero
        for _ in range(16):
            kx, ky, ph = int(rng.integers(1, 5)), int(rng.integers(1, 5)), rng.uniform(0, 2 * math.pi)
            s = s + torch.sin(2.0 * math.pi * (kx * X + ky * Y) + ph)
        return rho, zero, zero, 0.01 * s * torch.exp(-((Z - 0.5) / 0.1) ** 2), p
    if c["problem"] == "gas":           # uniform gas, 5 % noise in every field
        v = [0.1 * noise() for _ in range(c["ndim"])] + [zero] * (3 - c["ndim"])
        return 1.0 + 0.05 * noise().clamp(-4, 4), v[0], v[1], v[2], 1.0 + 0.05 * noise().clamp(-4, 4)
    # the AMR benchmark's interface (rho 1 and 10, smoothed over two finest cells), seeded flow
    phi = zero + Z - 0.5
    m, am = 8, 0.08
    from flashx_b200 import simulations as S
    u, w = S.uniform01(np.arange(m, dtype=np.uint64), stream=20)
    q, r = S.uniform01(np.arange(m, dtype=np.uint64), stream=21)
    for i in range(m):
        arg = (1.0 + math.floor(3.0 * u[i])) * X + (1.0 + math.floor(3.0 * w[i])) * Y
        phi = phi - am * (0.5 + r[i]) / m * 2.0 * torch.sin(2.0 * math.pi * (arg + q[i]))
    rho = 1.0 + 4.5 * (1.0 + torch.tanh(phi / (2.0 * dfine)))
    s = 0.02 * torch.sin(2.0 * math.pi * X + rng.uniform(0, 6)) * torch.sin(2.0 * math.pi * Y + rng.uniform(0, 6))
    a = rng.uniform(0.9, 1.1, 4)
    s = s + zero
    return rho, 0.25 * a[0] + s, 0.125 * a[1] - s, 0.0625 * a[2] * one, 2.5 * a[3] * one


def _eos(hp, u, where=None):
    """Eos_wrapped(MODE_DENS_EI) on a dict of tensors (optionally only where a mask is set)."""
    ek = 0.5 * (u["velx"] * u["velx"] + u["vely"] * u["vely"] + u["velz"] * u["velz"])
    cand = u["ener"] - ek
    eint = torch.where(cand > torch.clamp(hp.eintSwitch * ek, min=hp.smalle), cand, u["eint"])
    gm1 = hp.gamma - 1.0
    pres = u["dens"] * eint * gm1
    new = {"pres": pres, "temp": eint * (gm1 / hp.gasConstant) * hp.eos_singleSpeciesA, "eint": eint, "ener": eint + ek,
           "gamc": torch.full_like(eint, hp.gamma), "game": pres / (eint * u["dens"]) + 1.0}
    for k, v in new.items():
        u[k] = v if where is None else torch.where(where, v, u[k])
    return u


def _initial(c, seed, device):
    """Interior state as a dict of ten tensors: (1, nz, ny, nx) of a uniform
    grid, (leaf, n, n, n) of an AMR mesh."""
    geom, hp = _geometry(c), _params(c)
    t = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device=device)  # noqa: E731
    if c["grid"] == "ug":
        nx, ny, nz = c["n"] * c["bx"], c["n"] * c["by"], c["n"] * c["bz"] if c["ndim"] == 3 else 1
        d = geom.deltas()
        ax = [(torch.arange(m, device=device, dtype=torch.float64) + 0.5) * d[a] for a, m in enumerate((nx, ny, nz))]
        X, Y, Z = ax[0].view(1, 1, 1, -1), ax[1].view(1, 1, -1, 1), ax[2].view(1, -1, 1, 1)
        dfine = d[0]
    else:
        mesh = _mesh(c)
        n = c["n"]
        d0 = geom.deltas()
        w = t(0.5 ** (mesh.levels.astype(np.float64) - 1))
        co = t(mesh.bcoords)
        cell = torch.arange(n, device=device, dtype=torch.float64) + 0.5
        ax = [(co[:, a, None] * n + cell) * (d0[a] * w[:, None]) for a in range(3)]
        X, Y, Z = ax[0][:, None, None, :], ax[1][:, None, :, None], ax[2][:, :, None, None]
        dfine = min(d0) / 2.0 ** (c["maxlev"] - 1)
    rho, vx, vy, vz, p = _primitives(c, seed, X, Y, Z, dfine)
    eint = p / ((hp.gamma - 1.0) * rho)
    u = {"dens": rho, "velx": vx, "vely": vy, "velz": vz, "eint": eint, "ener": eint + 0.5 * (vx * vx + vy * vy + vz * vz)}
    return {k: v.contiguous() for k, v in _eos(hp, u).items()}


def _deltas(c, device):
    """Cell sizes per axis: numbers, or per-leaf tensors shaped (leaf, 1, 1, 1)."""
    d = _geometry(c).deltas()
    if c["grid"] == "ug":
        return list(d)
    w = torch.as_tensor(0.5 ** (_mesh(c).levels.astype(np.float64) - 1), device=device).view(-1, 1, 1, 1)
    return [w * x for x in d]


def _rate(c, hp, u, d):
    cs = torch.sqrt(u["gamc"] * u["pres"] / u["dens"])
    r = ((u["velx"].abs() + cs) / d[0]).max()
    r = torch.maximum(r, ((u["vely"].abs() + cs) / d[1]).max())
    return float(torch.maximum(r, ((u["velz"].abs() + cs) / d[2]).max()) if c["ndim"] == 3 else r)


def _to_unk(c, u, device):
    """The block array (block, k, j, i, variable) of a uniform grid's state,
    zeros in guard cells and in slots the solver does not own."""
    n, nd = c["n"], c["ndim"]
    nk, gk = (n, G) if nd == 3 else (1, 0)
    unk = torch.zeros((c["bx"] * c["by"] * c["bz"], nk + 2 * gk, n + 2 * G, n + 2 * G, NUNK), dtype=torch.float64,
                      device=device)
    for v, s in SLOT.items():
        f = u[v].view(c["bz"], nk, c["by"], n, c["bx"], n).permute(0, 2, 4, 1, 3, 5).reshape(-1, nk, n, n)
        unk[:, gk:gk + nk, G:G + n, G:G + n, s] = f
    return unk


def _to_message(u):
    """The leaf message (leaf, variable, k, j, i) of an AMR state."""
    return torch.stack([u[v] for v in LEAF_MSG_VARS], dim=1).reshape(-1)


_held = {"key": None}


def _device(c):
    """The solver for this case, made at its first state and kept."""
    key = tuple(sorted((k, v) for k, v in c.items() if k != "name"))
    if _held["key"] != key:
        if _held.get("dev") is not None:
            _held["dev"].close()
        _held.clear()
        _held["key"] = None
        geom, hp = _geometry(c), _params(c)
        u = _initial(c, 1, "cuda")
        if c["grid"] == "ug":
            dev = HydroDevice(geom, hp, c["prec"])
            _held["out"] = torch.zeros(dev.unk_shape, dtype=torch.float64, pin_memory=True).numpy()
            dev.attach_unk(_to_unk(c, u, "cuda").cpu().numpy())
        else:
            mesh = _mesh(c)
            dev = HydroDevice(geom, hp, c["prec"], mesh=mesh)
            n = c["n"]
            unk = np.zeros(dev.unk_shape)
            inner = unk[:, G:G + n, G:G + n, G:G + n]
            for v, s in SLOT.items():
                inner[..., s] = u[v].cpu().numpy()
            dev.attach_unk(unk)
            _held["out"] = torch.zeros(mesh.nleaf * len(LEAF_MSG_VARS) * n ** 3, dtype=torch.float64, device="cuda")
            _held["leaves"] = np.arange(mesh.nleaf, dtype=np.int32)
            dev.unk = None
        _held["dev"] = dev
        _held["key"] = key
    return _held


def prepare(case, seed):
    h = _device(case)
    hp = _params(case)
    u = _initial(case, seed, "cuda")
    dt = 0.5 * hp.cfl / _rate(case, hp, u, _deltas(case, "cuda"))
    if case["grid"] == "ug":
        unk = torch.empty(h["dev"].unk_shape, dtype=torch.float64, pin_memory=True)
        unk.copy_(_to_unk(case, u, "cuda"))
        data = unk.numpy()
    else:
        data = _to_message(u)
    torch.cuda.synchronize()
    return {"h": h, "hp": hp, "data": data, "dt": dt, "steps": case["steps"], "how": case["how"], "grid": case["grid"]}


def run(state):
    h, hp, how = state["h"], state["hp"], state["how"]
    dev, out = h["dev"], h["out"]
    dt = dt_old = state["dt"]
    ug = state["grid"] == "ug"
    if ug:
        dev.put_interior(state["data"])
    else:
        dev.unpack_leaves(h["leaves"], state["data"])
    if how == "advance":
        dt, dt_old = dev.advance(state["steps"], dt, dt_old)
    else:
        for s in range(state["steps"]):
            if how == "host" and s:
                dev.get_interior(out)
                dev.put_interior(out)
            dev.Hydro(0.0, dt, dt_old)
            dt_old, dt = dt, driver_dt(dev.Hydro_computeDt(), dt, hp)
    if ug:
        dev.get_interior(out)
    else:
        dev.pack_leaves(h["leaves"], out)
    return {"state": out, "dt": dt, "dt_old": dt_old}


# -------------------------------------------------------------- work and limits
def _zones(c):
    if c["grid"] == "amr":
        return _mesh(c).ncells()
    return c["n"] ** c["ndim"] * c["bx"] * c["by"] * c["bz"]


# floating-point operations of one zone-update, counted from the formulas:
# eigensystem, slopes or WENO weights, tracing, transverse and CTU terms,
# Riemann solve per direction, update and Eos
FLOPS = {(2, 3): 2000, (2, 5): 4300, (3, 3): 4300, (3, 5): 7900}


def work(case):
    z, s = _zones(case), case["steps"]
    moves = s if case["how"] == "host" else 1
    # a step reads nine and writes ten values of a zone; the state comes and goes with ten
    return {"bytes": 152.0 * z * s + 160.0 * z * moves, "flops": float(FLOPS[case["ndim"], case["order"]]) * z * s}


def tolerance(case):
    # about four times the distance from `exact` measured over these ranges:
    # 4.7e-14 in FP64, 3.3e-7 with FP32 reconstruction and Riemann solve
    if case["prec"] == "fp64":
        return {"rel": 2e-13, "max": 1e-10}
    return {"rel": 1.5e-6, "max": 1e-3}


# ------------------------------------------------------------ the step in 64 bits
PRIM = ("dens", "velx", "vely", "velz", "pres", "eint")


def _sh(x, d, o):
    """The value o cells further along axis d, at every cell."""
    return torch.roll(x, -o, dims=-1 - d)


def _sweep_order(d):
    """Positions in PRIM of density, normal and the two transverse velocities, pressure and eint."""
    return (0, 1 + d, 1 + (d + 1) % 3, 1 + (d + 2) % 3, 4, 5)


def _upwind(lam, m, c, p):
    return torch.where(lam > 0, c - m, p - c)


def _transverse(E, un, m, c, p):
    """hy_upwindTransverseFlux: sum over the waves of lambda r (l . upwind difference)."""
    l0, l4 = un - E["c"], un + E["c"]
    t = [_upwind(l0, m[k], c[k], p[k]) for k in range(5)]
    d0 = E["lp"] * t[4] - E["ah"] * t[1]
    t = [_upwind(l4, m[k], c[k], p[k]) for k in range(5)]
    d4 = E["ah"] * t[1] + E["lp"] * t[4]
    t = [_upwind(un, m[k], c[k], p[k]) for k in range(6)]
    sD = l0 * E["rho"] * d0 + un * (t[0] - E["a2i"] * t[4]) + l4 * E["rho"] * d4
    s1 = -l0 * E["c"] * d0 + l4 * E["c"] * d4
    return [sD, s1, un * t[2], un * t[3], l0 * E["rp"] * d0 + l4 * E["rp"] * d4, un * t[5]]


def _ldot(E, x):
    return [E["lp"] * x[4] - E["ah"] * x[1], x[2], x[0] - E["a2i"] * x[4], x[3], E["ah"] * x[1] + E["lp"] * x[4]]


def _rsum(E, w):
    return [E["rho"] * w[0] + w[2] + E["rho"] * w[4], E["c"] * (w[4] - w[0]), w[1], w[3], E["rp"] * (w[0] + w[4])]


def _limit(name, a, b):
    s = torch.copysign(torch.ones_like(a), a) + torch.copysign(torch.ones_like(b), b)
    if name == "mc":
        return s * torch.minimum(torch.minimum(a.abs(), 0.25 * (a + b).abs()), b.abs())
    if name == "minmod":
        return 0.5 * s * torch.minimum(a.abs(), b.abs())
    ab = a * b
    return torch.where(ab <= 0, torch.zeros_like(a), 2.0 * ab / torch.where(ab <= 0, torch.ones_like(a), a + b))


def _weno(I):
    """WENO5 values at i + 1/2 and i - 1/2 from five cells."""
    a, b, c, d, e = I
    p = [(2 * a - 7 * b + 11 * c) / 6, (-b + 5 * c + 2 * d) / 6, (2 * c + 5 * d - e) / 6]
    m = [(-a + 5 * b + 2 * c) / 6, (2 * b + 5 * c - d) / 6, (11 * c - 7 * d + 2 * e) / 6]
    s = [13. / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2,
         13. / 12 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2,
         13. / 12 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2]
    out = []
    for g, v in (((0.1, 0.6, 0.3), p), ((0.3, 0.6, 0.1), m)):
        w = [g[q] / (1e-36 + s[q]) for q in range(3)]
        t = w[0] + w[1] + w[2]
        out.append(w[0] / t * v[0] + w[1] / t * v[1] + w[2] / t * v[2])
    return out


def _fluxes(c, hp, V, gam, dt, dl):
    """Face fluxes on the left faces of every cell and the face-state
    pressures, per direction, from guard-filled primitives V (six tensors in
    PRIM order) and gam = (gamc, game)."""
    nd = c["ndim"]
    gc, ge = gam
    rho, p = V[0], V[4]
    cs = torch.sqrt(gc * p / rho)
    E = {"rho": rho, "c": cs, "a2i": 1.0 / (cs * cs), "ah": 0.5 / cs, "rp": rho * cs * cs}
    E["lp"] = 0.5 * E["a2i"] / rho
    sig = []
    for d in range(nd):
        o = _sweep_order(d)
        x = [V[q] for q in o]
        t = _transverse(E, x[1], [_sh(q, d, -1) for q in x], x, [_sh(q, d, 1) for q in x])
        s = [None] * 6
        for q in range(6):
            s[o[q]] = t[q]
        sig.append(s)
    grav = [hp.gravity[a] if hp.useGravity else 0.0 for a in range(3)]
    res = []
    for d in range(nd):
        o = _sweep_order(d)
        C = [V[q] for q in o]
        dtn = dt / dl[d]
        un = C[1]
        if hp.order == 3:
            dm = [q - _sh(q, d, -1) for q in C]
            dp = [_sh(q, d, 1) - q for q in C]
            wm, wp = _ldot(E, dm), _ldot(E, dp)
            db = _rsum(E, [_limit(hp.slopeLimiter.lower(), a, b) for a, b in zip(wm, wp)])
            db.append(_limit(hp.slopeLimiter.lower(), dm[5], dp[5]))
            L = [0.5 * (C[q] + _sh(C[q], d, -1)) - (db[q] - _sh(db[q], d, -1)) / 6 for q in range(6)]
            R = [0.5 * (C[q] + _sh(C[q], d, 1)) - (_sh(db[q], d, 1) - db[q]) / 6 for q in range(6)]
        else:
            S = [[_sh(q, d, k) for q in C] for k in range(-2, 3)]
            W = [_ldot(E, s) for s in S]
            r, l = zip(*[_weno([W[k][w] for k in range(5)]) for w in range(5)])
            r5, l5 = _weno([S[k][5] for k in range(5)])
            L, R = _rsum(E, l) + [l5], _rsum(E, r) + [r5]
        dW, W6 = [], []
        for q in range(6):
            a, b, x = L[q], R[q], C[q]
            flat = (b - x) * (x - a) <= 0
            a, b = torch.where(flat, x, a), torch.where(flat, x, b)
            a = torch.where(6 * (b - a) * (x - 0.5 * (a + b)) > (b - a) ** 2, 3 * x - 2 * b, a)
            b = torch.where(6 * (b - a) * (x - 0.5 * (a + b)) < -(b - a) ** 2, 3 * x - 2 * a, b)
            L[q], R[q] = a, b
            dW.append(b - a)
            W6.append(6 * (x - 0.5 * (a + b)))
        hd = 0.5 * dtn
        up, dn = torch.clamp(un, min=0.0) * hd, -torch.clamp(un, max=0.0) * hd
        Wp5 = R[5] - up * (dW[5] - (1 - up * 4 / 3) * W6[5])
        Wm5 = L[5] + dn * (dW[5] + (1 - dn * 4 / 3) * W6[5])
        cA, cB = _ldot(E, dW), _ldot(E, [-w for w in W6])
        lam = (un - cs, un, un, un, un + cs)
        lw = [0.5 * (-1 - dtn * v) * a + 0.25 * (1 + 2 * dtn * v + 4. / 3 * (dtn * v) ** 2) * b
              for v, a, b in zip(lam, cA, cB)]
        rw = [0.5 * (1 - dtn * v) * a + 0.25 * (1 - 2 * dtn * v + 4. / 3 * (dtn * v) ** 2) * b
              for v, a, b in zip(lam, cA, cB)]
        Wm = [C[q] + W6[q] / 12 + s for q, s in enumerate(_rsum(E, lw))] + [Wm5]
        Wp = [C[q] + W6[q] / 12 + s for q, s in enumerate(_rsum(E, rw))] + [Wp5]
        Wm = [Wm[o.index(q)] for q in range(6)]
        Wp = [Wp[o.index(q)] for q in range(6)]
        for e in range(nd):
            if e != d:
                h = 0.5 * dt / dl[e]
                Wm = [a - h * s for a, s in zip(Wm, sig[e])]
                Wp = [a - h * s for a, s in zip(Wp, sig[e])]
        bad = (Wm[0] < 0) | (Wp[0] < 0) | (Wm[4] < 0) | (Wp[4] < 0)
        Wm = [torch.where(bad, V[q], Wm[q]) for q in range(6)]
        Wp = [torch.where(bad, V[q], Wp[q]) for q in range(6)]
        if hp.useGravity:
            for a in range(3):
                Wm[1 + a], Wp[1 + a] = Wm[1 + a] + 0.5 * dt * grav[a], Wp[1 + a] + 0.5 * dt * grav[a]
        if nd == 3:                     # full CTU: sigma of one transverse axis upwinded along the other
            e1, e2 = (d + 1) % 3, (d + 2) % 3
            T = None
            for e, s in ((e1, e2), (e2, e1)):
                oe = _sweep_order(e)
                x = [sig[s][q] for q in oe]
                t = _transverse(E, V[1 + e], [_sh(q, e, -1) for q in x], x, [_sh(q, e, 1) for q in x])
                t = [t[oe.index(q)] for q in range(6)]
                T = t if T is None else [a + b for a, b in zip(T, t)]
            f = dt * dt / (6.0 * dl[e1] * dl[e2])
            Wm = [a + t * f for a, t in zip(Wm, T)]
            Wp = [a + t * f for a, t in zip(Wp, T)]
            bad = (Wm[0] <= 0) | (Wp[0] <= 0) | (Wm[4] <= 0) | (Wp[4] <= 0)
            Wm = [torch.where(bad, V[q], Wm[q]) for q in range(6)]
            Wp = [torch.where(bad, V[q], Wp[q]) for q in range(6)]
        F = _riemann(hp, d, [_sh(q, d, -1) for q in Wp], _sh(gc, d, -1), _sh(ge, d, -1), Wm, gc, ge)
        res.append((F, Wm[4] + Wp[4]))
    return res


def _riemann(hp, d, l, gcl, gel, r, gcr, ger):
    """HLL or HLLC fluxes of density, momenta and energy, then the eint and volume fluxes."""
    def side(v, ge):
        E = 0.5 * v[0] * (v[1] * v[1] + v[2] * v[2] + v[3] * v[3]) + v[4] / (ge - 1)
        U = [v[0], v[0] * v[1], v[0] * v[2], v[0] * v[3], E]
        F = [u * v[1 + d] for u in U]
        F[1 + d] = F[1 + d] + v[4]
        F[4] = F[4] + v[4] * v[1 + d]
        return U, F
    (UL, FL), (UR, FR) = side(l, gel), side(r, ger)
    ul, ur = l[1 + d], r[1 + d]
    cl, cr = torch.sqrt(gcl * l[4] / l[0]), torch.sqrt(gcr * r[4] / r[0])
    SL, SR = torch.minimum(ul - cl, ur - cr), torch.maximum(ul + cl, ur + cr)
    if hp.RiemannSolver == "HLL":
        F = [torch.where(SL > 0, a, torch.where(SR < 0, b, (SR * a - SL * b + SR * SL * (v - u)) / (SR - SL)))
             for a, b, u, v in zip(FL, FR, UL, UR)]
    else:
        q = (r[0] * ur * (SR - ur) - l[0] * ul * (SL - ul) + l[4] - r[4]) / (r[0] * (SR - ur) - l[0] * (SL - ul))
        ps = l[0] * (SL - ul) * (q - ul) + l[4]

        def star(v, U, F, S, un):
            k = (S - un) / (S - q)
            C = [u * k for u in U]
            C[1 + d] = U[0] * k * q
            C[4] = U[4] * k + (ps * q - v[4] * un) / (S - q)
            return [f + S * (x - u) for f, x, u in zip(F, C, U)]
        A_, B_ = star(l, UL, FL, SL, ul), star(r, UR, FR, SR, ur)
        F = [torch.where(SL >= 0, a, torch.where(q >= 0, x, torch.where(SR >= 0, y, b)))
             for a, x, y, b in zip(FL, A_, B_, FR)]
    pos = F[0] > 0
    return F + [F[0] * torch.where(pos, l[5], r[5]), F[0] / torch.where(pos, l[0], r[0])]


def _update(c, hp, u, faces, dt, dl):
    """The conserved update of the interior state u; faces: per direction the
    lower and upper face fluxes of every cell and the sum of its face pressures."""
    nd = c["ndim"]
    rho0 = u["dens"]
    U = [rho0, rho0 * u["velx"], rho0 * u["vely"], rho0 * u["velz"], rho0 * u["ener"]]
    mom0 = U[1:4]
    pav = None
    for d, (lo, hi, ps) in enumerate(faces):
        U = [x - dt / dl[d] * (b - a) for x, a, b in zip(U, lo, hi)]
        pav = ps if pav is None else pav + ps
    pav = pav / (2.0 * nd)
    inten = rho0 * u["eint"]
    for d, (lo, hi, ps) in enumerate(faces):
        inten = inten + dt / dl[d] * (lo[5] - hi[5] + pav * (lo[6] - hi[6]))
    if hp.useGravity:
        g = hp.gravity
        U[4] = U[4] + 0.5 * dt * sum(m * a for m, a in zip(mom0, g))
        for a in range(3):
            U[1 + a] = U[1 + a] + 0.5 * dt * rho0 * g[a]
    rho = torch.clamp(U[0], min=hp.smlrho)
    v = [U[1 + a] / rho for a in range(3)]
    ener, eint = U[4] / rho, inten / rho
    if hp.useGravity:
        v = [x + 0.5 * dt * g[a] for a, x in enumerate(v)]
        ener = ener + 0.5 * dt * sum(x * a for x, a in zip(v, g))
    ek = 0.5 * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2])
    ee = ener - ek
    eint = torch.clamp(torch.where(ee > hp.eintSwitch * ek, ee, eint), min=hp.smalle)
    return _eos(hp, {"dens": rho, "velx": v[0], "vely": v[1], "velz": v[2], "eint": eint, "ener": eint + ek})


def _pad_map(n, lo, hi, device):
    """Interior index and velocity sign of cells -G .. n + G - 1 under the boundary conditions."""
    idx, sgn = [], []
    for i in range(-G, n + G):
        j, s, bc = i, 1.0, lo if i < 0 else hi
        if i < 0 or i >= n:
            if bc == BC_PERIODIC:
                j = i % n
            elif bc == BC_OUTFLOW:
                j = 0 if i < 0 else n - 1
            else:
                j, s = (-1 - i if i < 0 else 2 * n - 1 - i), -1.0
        idx.append(j)
        sgn.append(s)
    return torch.tensor(idx, device=device), torch.tensor(sgn, dtype=torch.float64, device=device)


def _padded_ug(c, geom, u):
    out = {}
    dims = [(-1, 0), (-2, 1)] + ([(-3, 2)] if c["ndim"] == 3 else [])
    maps = [_pad_map(u["dens"].shape[ax], geom.bc[2 * a], geom.bc[2 * a + 1], u["dens"].device) for ax, a in dims]
    for k in PRIM + ("gamc", "game"):
        x = u[k]
        for (ax, a), (idx, sgn) in zip(dims, maps):
            x = x.index_select(ax, idx)
            if k == ("velx", "vely", "velz")[a]:
                x = x * sgn.view([-1] + [1] * (-ax - 1))
        out[k] = x
    return out


PER_MASS = ("velx", "vely", "velz", "ener", "eint")


class _Tree:
    """Dense per-level copies of an AMR state (periodic boxes), for the guard fill."""

    def __init__(self, c, device):
        mesh = _mesh(c)
        self.n, self.dev = c["n"], device
        self.lev = torch.as_tensor(mesh.levels.astype(np.int64), device=device)
        self.co = torch.as_tensor(mesh.bcoords.astype(np.int64), device=device)
        self.maxlev = mesh.maxlev
        self.nb = {l: [c[k] << (l - 1) for k in ("bx", "by", "bz")] for l in range(1, mesh.maxlev + 1)}
        self.leaf = {}                  # leaf slot, -1 elsewhere, per level [z][y][x]
        for l in self.nb:
            t = torch.full(self.nb[l][::-1], -1, dtype=torch.int64, device=device)
            s = (self.lev == l).nonzero().view(-1)
            q = self.co[s]
            t[q[:, 2], q[:, 1], q[:, 0]] = s
            self.leaf[l] = t
        self.parent = {self.maxlev: torch.zeros_like(self.leaf[self.maxlev], dtype=torch.bool)}
        for l in range(self.maxlev - 1, 0, -1):
            f = (self.leaf[l + 1] >= 0) | self.parent[l + 1]
            z, y, x = self.leaf[l].shape
            self.parent[l] = f.view(z, 2, y, 2, x, 2).any(5).any(3).any(1)

    def cells(self, mask):
        for ax in range(3):
            mask = mask.repeat_interleave(self.n, ax)
        return mask

    def window(self, l, s):
        """Wrapped cell indices of the guard-filled blocks s of level l, one tensor per axis."""
        r = torch.arange(-G, self.n + G, device=self.dev)
        return [((self.co[s, a, None] * self.n + r) % (self.nb[l][a] * self.n)) for a in range(3)]

    def fill(self, hp, u):
        """Guard-filled blocks (leaf, n + 2G, ...) of every leaf."""
        n = self.n
        names = tuple(u)
        dense = {}
        for l in range(self.maxlev, 0, -1):
            z, y, x = self.leaf[l].shape
            s = (self.lev == l).nonzero().view(-1)
            q = self.co[s]
            D = {}
            for k in names:
                t = torch.zeros((z, n, y, n, x, n), dtype=torch.float64, device=self.dev)
                t[q[:, 2], :, q[:, 1], :, q[:, 0], :] = u[k][s]
                D[k] = t.view(z * n, y * n, x * n)
            if l < self.maxlev:         # parents: averages of the children in conserved form
                P = self.cells(self.parent[l])
                F = dense[l + 1]
                rd = None
                for k in ("dens",) + tuple(k for k in names if k != "dens"):
                    f = F[k] * F["dens"] if k in PER_MASS else F[k]
                    f = f.view(z * n, 2, y * n, 2, x * n, 2).sum((1, 3, 5)) * 0.125
                    if k == "dens":
                        rd = f
                    elif k in PER_MASS:
                        f = f / torch.where(P, rd, torch.ones_like(rd))
                    D[k] = torch.where(P, f, D[k])
            dense[l] = D
        for l in range(2, self.maxlev + 1):
            have = self.cells((self.leaf[l] >= 0) | self.parent[l])
            C, D, fd = dense[l - 1], dense[l], None
            for k in ("dens",) + tuple(k for k in names if k != "dens"):
                f = C[k] * C["dens"] if k in PER_MASS else C[k]
                for ax in range(3):     # linear in each axis, weights 1/4 and 3/4
                    lo = 0.25 * torch.roll(f, 1, ax) + 0.75 * f
                    hi = 0.75 * f + 0.25 * torch.roll(f, -1, ax)
                    f = torch.stack((lo, hi), ax + 1).flatten(ax, ax + 1)
                if k == "dens":
                    fd = f
                elif k in PER_MASS:
                    f = f / torch.where(have, torch.ones_like(fd), fd)
                D[k] = torch.where(have, D[k], f)
        e = n + 2 * G
        out = {k: torch.empty((len(self.lev), e, e, e), dtype=torch.float64, device=self.dev) for k in names}
        region = torch.tensor([0] * G + [1] * n + [2] * G, device=self.dev)
        for l in range(1, self.maxlev + 1):
            s = (self.lev == l).nonzero().view(-1)
            for s in s.split(512):
                wx, wy, wz = self.window(l, s)
                B = {k: dense[l][k][wz[:, :, None, None], wy[:, None, :, None], wx[:, None, None, :]] for k in names}
                # Eos on the guard regions next to another level
                off = torch.arange(-1, 2, device=self.dev)
                q = [(self.co[s, a, None] + off) % self.nb[l][a] for a in range(3)]
                other = self.leaf[l][q[2][:, :, None, None], q[1][:, None, :, None], q[0][:, None, None, :]] < 0
                other = other[:, region][:, :, region][:, :, :, region]
                B = _eos(hp, B, other)
                for k in names:
                    out[k][s] = B[k]
        return out

    def finer(self):
        """(leaf, face, its four fine leaves) for every leaf face next to finer leaves."""
        todo = []
        for l in range(1, self.maxlev):
            s = (self.lev == l).nonzero().view(-1)
            for f in range(6):
                d, side = f >> 1, f & 1
                q = self.co[s].clone()
                q[:, d] = (q[:, d] + (1 if side else -1)) % self.nb[l][d]
                at = self.parent[l][q[:, 2], q[:, 1], q[:, 0]]
                a1, a2 = [a for a in range(3) if a != d]
                kids = []
                for o in range(4):
                    k = 2 * q[at]
                    k[:, d] += 0 if side else 1
                    k[:, a1] += o & 1
                    k[:, a2] += o >> 1
                    kids.append(self.leaf[l + 1][k[:, 2], k[:, 1], k[:, 0]])
                if bool(at.any()):
                    todo.append((s[at], f, torch.stack(kids, 1)))
        return todo


def _step(c, hp, geom, tree, u, dt, dl):
    n, nd = c["n"], c["ndim"]
    pad = tree.fill(hp, u) if tree else _padded_ug(c, geom, u)
    inner = (slice(None),) + tuple(slice(G, -G) if nd == 3 or a else slice(None) for a in range(3))
    count = pad["dens"].shape[0]
    per = max(1, (1 << 23) // (n + 2 * G) ** 3) if tree else count
    faces = [None] * nd
    for b0 in range(0, count, per):
        P = {k: v[b0:b0 + per] for k, v in pad.items()}
        sub = [x[b0:b0 + per] for x in dl] if tree else dl
        res = _fluxes(c, hp, [P[k] for k in PRIM], (P["gamc"], P["game"]), dt, sub)
        for d in range(nd):
            F, ps = res[d]
            got = ([f[inner] for f in F], [_sh(f, d, 1)[inner] for f in F], ps[inner])
            if faces[d] is None:
                faces[d] = ([], [], [])
            for store, part in zip(faces[d], got):
                store.append(part)
    cat = lambda parts: [torch.cat([p[k] for p in parts]) for k in range(7)]  # noqa: E731
    faces = [(cat(lo), cat(hi), torch.cat(ps)) for lo, hi, ps in faces]
    if tree:                            # coarse faces next to finer leaves take their mean fluxes
        h = n // 2
        new = []
        for s, f, kids in tree.finer():
            d, side = f >> 1, f & 1
            src, at = faces[d][1 - side], [slice(None)] * 4
            at[3 - d] = 0 if side else n - 1
            for k in range(7):
                plane = src[k][tuple([kids.view(-1)] + at[1:])].view(len(s), 2, 2, n, n)
                m = plane.view(len(s), 2, 2, h, 2, h, 2).mean((4, 6))          # (leaf, o2, o1, t2, t1)
                new.append((s, f, k, m.permute(0, 1, 3, 2, 4).reshape(len(s), n, n)))
        for s, f, k, m in new:
            d, side = f >> 1, f & 1
            at = [s, slice(None), slice(None), slice(None)]
            at[3 - d] = n - 1 if side else 0
            faces[d][side][k][tuple(at)] = m
    return _update(c, hp, u, faces, dt, dl)


def exact(case, seed):
    if case["grid"] == "amr" and _zones(case) * case["steps"] > 2e8:
        return None                     # over twenty seconds
    device = "cuda" if torch.cuda.is_available() else "cpu"
    c, hp, geom = case, _params(case), _geometry(case)
    u = _initial(c, seed, device)
    dl = _deltas(c, device)
    dt = dt_old = 0.5 * hp.cfl / _rate(c, hp, u, dl)
    tree = _Tree(c, device) if c["grid"] == "amr" else None
    for _ in range(c["steps"]):
        u = _step(c, hp, geom, tree, u, dt, dl)
        dt_old, dt = dt, driver_dt(hp.cfl / _rate(c, hp, u, dl), dt, hp)
    out = _to_message(u) if tree else _to_unk(c, u, device)
    return {"state": out, "dt": dt, "dt_old": dt_old}
