"""Timed workloads of the MHD step, through the package's public entry points.

A case is one call pattern of a user's program on one kind of grid:

  run    n steps of a fixed dt on a resident state, then the state read back
         (``mhd_steps``, ``mhd_download_state``)
  cfl    the same with the CFL dt of every step (``mhd_steps_cfl``)
  host   n steps of a host-resident driver, whose state goes in and out of
         host memory at every step (``mhd_steps_host``)
  batch  n steps of a ragged batch of independent instances, then every state
         read back (``mhd_batch_steps``)
  rhs    the right-hand sides on the caller's own device arrays
         (``mhd_fluxes_noalloc``)

Read-backs go into a pinned buffer that the program keeps.  The state of an
FP32-storage instance is handed on in the type it is stored in.
"""
import ctypes as C
import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "rast-3dmhd-cpp_gb300" / "python"))

from mhd_gb300 import abi  # noqa: E402
from mhd_gb300.case import Case, STATE_FIELDS, metrics  # noqa: E402
from mhd_gb300.sim import Batch, Simulation  # noqa: E402

DT = 1e-4
# wall conditions: izCon, iTCon, TP
WALLS = {"fixed": (0, 0, 0.0), "flux": (1, 1, 0.0), "spot": (1, 4, float(np.float32(0.1)))}


def _case(kind, nx, ny, nz, steps, mag=True, rot=False, shr=False, walls="fixed", precision="fp64", count=1, mix=0,
          name=None):
    c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "steps": steps, "mag": mag, "rot": rot, "shr": shr,
         "walls": walls, "precision": precision, "count": count, "mix": mix}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest grid that the server admits, read back after a few steps: launches and latency
        _case("run", 32, 32, 32, 20, name="run_fp64_32x32x32"),
        # the small plain-method configuration: 100 steps, then a dump
        _case("run", 64, 64, 32, 100, name="run_fp64_64x64x32"),
        # the reference's default physics (no field, spot on the upper wall) with rotation, odd sizes
        _case("run", 97, 45, 61, 50, mag=False, rot=True, walls="spot", name="run_fp64_hydro_97x45x61"),
        # the headline configuration: field, rotation and shear on the largest grid
        _case("run", 512, 512, 256, 3, rot=True, shr=True, name="run_fp64_512x512x256"),
        # a driver that keeps its arrays on the host, as the reference's own does
        _case("host", 256, 256, 128, 4, name="host_fp64_256x256x128"),
        # the reference's run mode: the CFL dt of every step, flux walls
        _case("cfl", 128, 128, 64, 20, rot=True, walls="flux", name="cfl_fp64_128x128x64"),
        # FP32 storage on a small grid
        _case("run", 64, 64, 32, 100, precision="fp32", name="run_fp32_64x64x32"),
        # the FP32-storage precision configuration
        _case("run", 256, 256, 128, 100, precision="fp32", name="run_fp32_256x256x128"),
        # FP32 storage with the CFL dt and rotation, sizes that fill no tile
        _case("cfl", 200, 150, 100, 30, rot=True, precision="fp32", name="cfl_fp32_200x150x100"),
        # a served mix of instances of uneven sizes, one batch of each precision
        _case("batch", 32, 128, 64, 10, count=24, mix=2, name="batch_fp64_24"),
        _case("batch", 32, 128, 64, 40, count=24, mix=3, precision="fp32", name="batch_fp32_24"),
        # right-hand sides for a caller with arrays of its own
        _case("rhs", 64, 64, 32, 1, name="rhs_64x64x32"),
    ]


def draw(rng: random.Random):
    """One more case: any kind, sizes spread over the logarithm of the listed range, odd ones among them."""
    size = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    kind = rng.choice(["run", "run", "run", "cfl", "cfl", "host", "batch", "batch", "rhs"])
    precision = "fp64" if kind in ("host", "rhs") else rng.choice(["fp64", "fp32"])
    phys = dict(mag=rng.random() < 0.75, rot=rng.random() < 0.4, walls=rng.choice(["fixed", "flux", "spot"]))
    if kind == "rhs":
        return _case(kind, size(24, 80), size(24, 70), size(20, 60), 1, **phys)
    if kind == "batch":
        return _case(kind, 32, size(40, 144), size(24, 80), 20 if precision == "fp32" else 8, precision=precision,
                     count=rng.randint(4, 24), mix=rng.randrange(1 << 20), **phys)
    nx, ny, nz = size(32, 320), size(24, 320), size(20, 160)
    if kind == "cfl":  # the CFL dt of a coarse grid takes repeated passes out of the range where the flow is resolved
        nx, ny, nz = size(128, 320), size(128, 320), size(96, 160)
    most = (4e8 if precision == "fp32" else 1e8) / (nx * ny * nz)
    steps = max(2, min(4 if kind == "host" else 60, int(most)))
    # the shear switch sums the temperature's right-hand side over all steps, so such runs are short ones
    phys["shr"] = kind == "run" and nx * ny * nz > 4_000_000 and rng.random() < 0.5
    return _case(kind, nx, ny, nz, steps, precision=precision, **phys)


# ---- what a user's program has in hand -------------------------------------

def _grids(case):
    """(nx, ny, nz) of every instance; a batch has square grids of uneven sizes, fixed by its `mix`."""
    if case["kind"] != "batch":
        return [(case["nx"], case["ny"], case["nz"])]
    r = random.Random(case["mix"])
    lo, hi, nz = case["nx"], case["ny"], case["nz"]
    steps = [lo, (lo + hi) // 4, (lo + hi) // 3, (lo + hi) // 2, (lo + 3 * hi) // 4, hi]
    got = []
    for _ in range(case["count"]):
        n = r.choice(steps)
        got.append((n, n, r.choice([max(16, nz // 2), nz])))
    return got


def _physics(case, seed, k):
    """RE and the mean vertical field of instance k: log-uniform in a batch, as a served mix has them."""
    if case["kind"] != "batch":
        return 100.0, 1e-3
    r = random.Random(1000003 * seed + k)
    return 1.0 / math.exp(r.uniform(math.log(3e-3), math.log(3e-2))), math.exp(r.uniform(math.log(1e-4), math.log(1e-2)))


# RM: a magnetic Prandtl number of 10; the one-sided wall stencils of B amplify it slowly, at a rate that falls with RM
THETA, GRAV, ZMAX, STRETCH, RM = 4.5, 9.0, 2.0, 1.5, 1000.0


def _depth(nz):
    xi = np.arange(nz) / (nz - 1)
    z = 0.5 * ZMAX * (1.0 + np.tanh(STRETCH * (2.0 * xi - 1.0)) / np.tanh(STRETCH))
    return np.concatenate([z[:1], z, z[-1:]])


def _fields(case, seed, k):
    """An evolved-looking state on the GPU: a polytrope with noise, a smooth flow with noise, a vertical field with
    a smooth horizontal part; walls as the wall conditions leave them, periodic ghosts."""
    nx, ny, nz = _grids(case)[k]
    _, bz0 = _physics(case, seed, k)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1000 * int(seed) + k)
    f64 = dict(dtype=torch.float64, device="cuda")
    shape = (nz + 2, ny + 2, nx + 2)
    noise = lambda: torch.randn(shape, generator=gen, dtype=torch.float32, device="cuda").to(torch.float64)  # noqa: E731
    z = torch.tensor(_depth(nz), **f64)[:, None, None]
    y = torch.arange(ny + 2, **f64)[None, :, None] * (2 * math.pi / ny)
    x = torch.arange(nx + 2, **f64)[None, None, :] * (2 * math.pi / nx)
    ph = torch.rand(9, generator=gen, **f64) * 2 * math.pi
    up = torch.sin(math.pi * z / ZMAX)
    t1 = 1.0 + THETA * z
    r1 = t1 ** (GRAV / THETA - 1.0)
    st = torch.zeros((8 if case["mag"] else 5,) + shape, **f64)
    st[4] = r1 * (1.0 + 1e-3 * noise())
    st[3] = t1 * (1.0 + 1e-3 * noise())
    st[0] = st[4] * (0.03 * up * torch.sin(2 * y + ph[0]) * torch.cos(x + ph[1]) + 1e-3 * noise())
    st[1] = st[4] * (0.03 * up * torch.sin(x + ph[2]) * torch.cos(y + ph[3]) + 1e-3 * noise())
    st[2] = st[4] * up * (0.03 * torch.sin(x + ph[4]) * torch.sin(2 * y + ph[5]) + 1e-3 * noise())
    if case["mag"]:
        st[5] = bz0 * (torch.sin(y + ph[6]) * up + 0.1 * noise())
        st[6] = bz0 * (torch.sin(x + ph[7]) * up + 0.1 * noise())
        st[7] = bz0 * (1.0 + 0.1 * up * noise())
    for w, wall in ((0, 1), (0, 0), (-1, -2), (-1, -1)):
        st[3, wall] = t1[w]
        st[2, wall] = 0.0
        if case["shr"]:
            st[0, wall] = 0.0
            st[1, wall] = st[4, wall] if w == 0 else -st[4, wall]
        if case["mag"]:
            st[7, wall] = 0.0
    st[:, :, 0], st[:, :, -1] = st[:, :, -2].clone(), st[:, :, 1].clone()
    st[:, :, :, 0], st[:, :, :, -1] = st[:, :, :, -2].clone(), st[:, :, :, 1].clone()
    return st


def _description(case, seed, k):
    nx, ny, nz = _grids(case)[k]
    re, bz0 = _physics(case, seed, k)
    iz, it, tp = WALLS[case["walls"]]
    return Case(nPx=nx, nPy=ny, nPz=nz, lMag=case["mag"], lRot=case["rot"], lShr=case["shr"], izCon=iz, iTCon=it, TP=tp,
                RE=re, RM=RM, bz0=bz0, dt=DT, THETA=THETA, GRAV=GRAV, zMax=ZMAX, z_stretch=STRETCH)


def _pointer(t):
    return C.cast(t.data_ptr(), C.POINTER(C.c_double))


def prepare(case, seed):
    if case["kind"] == "rhs":
        return _prepare_rhs(case, seed)
    sims, outs = [], []
    for k in range(len(_grids(case))):
        st = _fields(case, seed, k)
        host = torch.empty(st.shape, dtype=torch.float64, pin_memory=True)
        host.copy_(st)
        del st
        sim = Simulation(_description(case, seed, k), precision=case["precision"])
        for f, name in enumerate(STATE_FIELDS[:host.shape[0]]):
            sim.upload(name, host[f].numpy())
        sims.append(sim)
        outs.append(host)
    state = {"case": case, "sims": sims, "outs": outs}
    if case["kind"] == "host":
        state["ins"] = outs[0].numpy()
        state["outs"] = [torch.empty(outs[0].shape, dtype=torch.float64, pin_memory=True)]
    if case["kind"] == "batch":
        state["batch"] = Batch(sims)
        state["batch"].autotune(report=False)
    return state


def _prepare_rhs(case, seed):
    d = _description(case, seed, 0)
    m = metrics(d)
    st = _fields(case, seed, 0)
    flux = torch.zeros_like(st)
    iz, it, tp = WALLS[case["walls"]]
    a = abi.MhdFluxesNoallocArgs()
    a.nPx, a.nPy, a.nPz = d.nPx, d.nPy, d.nPz
    a.switches = (abi.SW_LROT if d.lRot else 0) | (abi.SW_LMAG if d.lMag else 0) | (abi.SW_LSHR if d.lShr else 0)
    a.izCon, a.iTCon, a.iBCon = iz, it, 0
    for k in ("RE", "PR", "THETA", "GRAV", "RY", "ANG", "RM", "BETA", "TP", "GAMMA", "SFF"):
        setattr(a, k, float(getattr(d, k)))
    a.TB = d.tb
    keep = [torch.tensor(v, dtype=torch.float64, device="cuda") for v in m.arrays()]
    for n, t in zip(("dxxdx", "d2xxdx2", "DDX", "dyydy", "d2yydy2", "DDY", "dzzdz", "d2zzdz2", "DDZ", "RKAPA", "DKAPA"), keep):
        setattr(a, n, t.data_ptr())
    for f in range(st.shape[0]):
        a.state[f] = st[f].data_ptr()
        a.flux[f] = flux[f].data_ptr()
    return {"case": case, "lib": abi.load(), "args": a, "state": st, "flux": flux, "keep": keep}


def run(state):
    case = state["case"]
    if case["kind"] == "rhs":
        abi.check(state["lib"].mhd_fluxes_noalloc(C.byref(state["args"]), torch.cuda.current_stream().cuda_stream))
        return list(state["flux"])
    sims, outs = state["sims"], state["outs"]
    if case["kind"] == "host":
        sims[0].steps_host(case["steps"], state["ins"], outs[0].numpy())
        return list(outs[0])
    if case["kind"] == "batch":
        state["batch"].steps(case["steps"])
    elif case["kind"] == "cfl":
        sims[0].steps_cfl(case["steps"])
    else:
        sims[0].steps(case["steps"])
    for sim, out in zip(sims, outs):
        abi.check(sim.L.mhd_download_state(sim.ctx, _pointer(out)), sim.ctx)
    if case["precision"] == "fp32":
        outs = [out.to(torch.float32) for out in outs]
    return outs if case["kind"] == "batch" else list(outs[0])


def work(case):
    """A step is three substages, each reading and writing the state and the RK register (the first needs no register
    in FP64, the last writes none); the read-back adds the state once."""
    nf = 8 if case["mag"] else 5
    cells = sum(nx * ny * nz for nx, ny, nz in _grids(case))
    ops = 200 if case["mag"] else 120
    if case["kind"] == "rhs":
        return {"bytes": cells * nf * 16, "flops": cells * 2 * ops}
    per_step = nf * (72 if case["precision"] == "fp32" else 80) + (48 if case["shr"] else 0)
    per_step += nf * 16 if case["kind"] == "host" else 0
    return {"bytes": cells * (case["steps"] * per_step + nf * 8), "flops": cells * case["steps"] * 3 * 2 * ops}


# ---- the same in plain torch, 64 bits --------------------------------------

def _metric(n, umax, stretch):
    """du/dxi-type factors (duudu, d2uudu2, spacing) with the ghosts repeating the walls."""
    if not stretch:
        d1, d2 = np.full(n + 2, 1.0 / umax), np.zeros(n + 2)
        return d1, d2, np.full(n + 2, float(np.float32(1.0) / np.float32(n - 1)) / d1[0])
    a = stretch * (2.0 * np.arange(n) / (n - 1) - 1.0)
    th, ts = np.tanh(a), np.tanh(stretch)
    du, d2u = umax * stretch * (1 - th * th) / ts, -4.0 * umax * stretch * stretch * th * (1 - th * th) / ts
    pad = lambda v: np.concatenate([v[:1], v, v[-1:]])  # noqa: E731
    return pad(1.0 / du), pad(-d2u / du**3), pad(du / (n - 1))


class _Plain:
    def __init__(self, case, seed, k):
        self.case = case
        self.n = nx, ny, nz = _grids(case)[k]
        self.re, _ = _physics(case, seed, k)
        t = lambda v: torch.tensor(v, dtype=torch.float64, device="cuda")  # noqa: E731
        half = lambda n: 0.5 * (n - 1)  # noqa: E731
        (self.x1, _, self.ddx), (self.y1, _, self.ddy) = _metric(nx, 6.0, 0), _metric(ny, 6.0, 0)
        z1, z2, self.ddz = _metric(nz, ZMAX, STRETCH)
        self.cx, self.cx2 = self.x1[1] * half(nx), self.x1[1] ** 2 * (nx - 1.0) ** 2
        self.cy, self.cy2 = self.y1[1] * half(ny), self.y1[1] ** 2 * (ny - 1.0) ** 2
        col = lambda v: t(v[1:-1])[:, None, None]  # noqa: E731
        self.cz, self.cza, self.czb = col(z1 * half(nz)), col(z2 * half(nz)), col(z1 * z1 * (nz - 1.0) ** 2)
        self.z1 = z1
        f = lambda v: float(np.float32(v))  # noqa: E731
        self.c13 = f(np.float32(1) / np.float32(3))
        self.gam = [f(np.float32(a) / np.float32(b)) for a, b in ((8, 15), (5, 12), (3, 4))]
        self.zet = [f(np.float32(-17) / np.float32(60)), f(np.float32(-5) / np.float32(12)), 0.0]
        self.gamma = f(np.float32(5) / np.float32(3))
        self.cv = 1.0 / (self.gamma - 1.0)
        self.ft = 0.0

    def dx(self, a):
        return (a[1:-1, 1:-1, 2:] - a[1:-1, 1:-1, :-2]) * self.cx

    def dy(self, a):
        return (a[1:-1, 2:, 1:-1] - a[1:-1, :-2, 1:-1]) * self.cy

    def dz(self, a):
        return (a[2:, 1:-1, 1:-1] - a[:-2, 1:-1, 1:-1]) * self.cz

    def d2(self, a, axis):
        c = a[1:-1, 1:-1, 1:-1]
        if axis == 0:
            return (a[1:-1, 1:-1, 2:] - 2 * c + a[1:-1, 1:-1, :-2]) * self.cx2
        if axis == 1:
            return (a[1:-1, 2:, 1:-1] - 2 * c + a[1:-1, :-2, 1:-1]) * self.cy2
        p, m = a[2:, 1:-1, 1:-1], a[:-2, 1:-1, 1:-1]
        return (p - m) * self.cza + (p - 2 * c + m) * self.czb

    def dxdy(self, a):
        d = a[1:-1, :, 2:] - a[1:-1, :, :-2]
        return (d[:, 2:] - d[:, :-2]) * (self.cx * self.cy)

    def dxdz(self, a):
        d = a[:, 1:-1, 2:] - a[:, 1:-1, :-2]
        return (d[2:] - d[:-2]) * (self.cx * self.cz)

    def dydz(self, a):
        d = a[:, 2:, 1:-1] - a[:, :-2, 1:-1]
        return (d[2:] - d[:-2]) * (self.cy * self.cz)

    def rhs(self, st):
        case, ore, orm, obeta = self.case, 1.0 / self.re, 1.0 / RM, 1.0
        c = lambda a: a[1:-1, 1:-1, 1:-1]  # noqa: E731
        one = lambda a, s: (4 * a[1 + s] - a[1 + 2 * s] if s > 0 else a[-4] - 4 * a[-3]) * self.cz[0 if s > 0 else -1]  # noqa: E731
        ru, rv, rw, tt, ro = st[:5]
        ri = 1.0 / ro
        u, v, w, p = ru * ri, rv * ri, rw * ri, ro * tt
        rwz = self.dz(rw)
        for s in (1, -1):
            rwz[0 if s > 0 else -1] = one(rw, s)[1:-1, 1:-1]
        fr = -self.dx(ru) - self.dy(rv) - rwz
        fu = -self.dx(p) - self.dx(ru * u) - self.dy(ru * v) - self.dz(ru * w)
        fv = -self.dy(p) - self.dx(rv * u) - self.dy(rv * v) - self.dz(rv * w)
        fw = GRAV * c(ro) - self.dz(p) - self.dx(rw * u) - self.dy(rw * v) - self.dz(rw * w)
        k13 = self.c13 * ore
        for f, a, ax, cross in ((fu, u, 0, ((v, self.dxdy), (w, self.dxdz))), (fv, v, 1, ((u, self.dxdy), (w, self.dydz))),
                                (fw, w, 2, ((u, self.dxdz), (v, self.dydz)))):
            for axis in range(3):
                f += self.d2(a, axis) * (ore * (4 * self.c13 if axis == ax else 1.0))
            for b, d in cross:
                f += k13 * d(b)
        ft = (self.d2(tt, 0) + self.d2(tt, 1) + self.d2(tt, 2)) * c(ri) / (self.cv * self.re)
        ux, uy, uz, vx, vy, vz, wx, wy, wz = (d(a) for a in (u, v, w) for d in (self.dx, self.dy, self.dz))
        if case["shr"]:
            ft = ft + self.ft
        else:
            ft -= c(u) * self.dx(tt) + c(v) * self.dy(tt) + c(w) * self.dz(tt) + c(tt) * (ux + vy + wz) / self.cv
            ft += (ore / self.cv) * c(ri) * (4 * self.c13 * (ux * ux + vy * vy + wz * wz - ux * vy - ux * wz - vy * wz)
                                             + (uy + vx) ** 2 + (uz + wx) ** 2 + (vz + wy) ** 2)
        if case["rot"]:
            om = 1.0 / 10.0
            fu += om * c(rv)
            fv -= om * c(ru)
        out = [fu, fv, fw, ft, fr]
        if case["mag"]:
            bx, by, bz = st[5:8]
            for s in (1, -1):
                wz[0 if s > 0 else -1] = one(w, s)[1:-1, 1:-1]
            X, Y, Z = c(bx), c(by), c(bz)
            bxx, bxy, bxz, byx, byy, byz, bzx, bzy, bzz = (d(a) for a in (bx, by, bz) for d in (self.dx, self.dy, self.dz))
            lap = [self.d2(a, 0) + self.d2(a, 1) for a in (bx, by, bz)]
            for a, lp in zip((bx, by, bz), lap):
                q = self.d2(a, 2)
                if a is not bz:
                    for s, e in ((1, 0), (-1, -1)):
                        b = [a[(1 if s > 0 else -2) + s * j][1:-1, 1:-1] for j in range(4)]
                        q[e] = s * (-3 * b[0] + 4 * b[1] - b[2]) * self.cza[e] + (2 * b[0] - 5 * b[1] + 4 * b[2] - b[3]) * self.czb[e]
                lp += q
            cu, cv, cw = c(u), c(v), c(w)
            out += [Y * uy + Z * uz - X * (vy + wz) - cu * bxx - cv * bxy - cw * bxz + orm * lap[0],
                    X * vx + Z * vz - Y * (ux + wz) - cu * byx - cv * byy - cw * byz + orm * lap[1],
                    X * wx + Y * wy - Z * (ux + vy) - cu * bzx - cv * bzy - cw * bzz + orm * lap[2]]
            jx, jy, jz = bzy - byz, bxz - bzx, byx - bxy
            fu += obeta * (Z * jy - Y * jz)
            fv += obeta * (X * jz - Z * jx)
            fw += obeta * (Y * jx - X * jy)
            ft += obeta * orm / self.cv * c(ri) * (jx * jx + jy * jy + jz * jz)
        if case["shr"]:
            self.ft = ft
        return out

    def walls(self, st):
        case = self.case
        iz, it, tp = WALLS[case["walls"]]
        c13, c43, c23 = self.c13, 4 * self.c13, 2 * self.c13
        for w, a, b in ((1, 2, 3), (-2, -3, -4)):
            if case["shr"]:
                st[0, w] = 0.0
                st[1, w] = st[4, w] if w == 1 else -st[4, w]
            else:
                for k in (0, 1):
                    st[k, w] = st[4, w] * (c43 * st[k, a] / st[4, a] - c13 * st[k, b] / st[4, b])
            st[2, w] = 0.0
            step = c23 * float(np.float32(1) / np.float32(self.n[2] - 1)) / self.z1[w] * THETA
            if w == 1 and it != 1:
                st[3, w] = 1.0
                if it == 4:
                    st[3, w, :, : (self.n[0] + 2) // 2] = float(np.float32(1.0)) - tp
            elif w == -2 and iz == 0:
                st[3, w] = 1.0 + THETA * ZMAX
            else:
                st[3, w] = c43 * st[3, a] - c13 * st[3, b] - step
            if case["mag"]:
                st[7, w] = 0.0
        st[:, 1:-1, 0], st[:, 1:-1, -1] = st[:, 1:-1, -2].clone(), st[:, 1:-1, 1].clone()
        st[:, 1:-1, :, 0], st[:, 1:-1, :, -1] = st[:, 1:-1, :, -2].clone(), st[:, 1:-1, :, 1].clone()

    def cfl(self, st):
        c = lambda a: a[1:-1, 1:-1, 1:-1]  # noqa: E731
        s = torch.tensor(np.minimum(np.minimum(self.ddx[1], self.ddy[1]), self.ddz[1:-1]), device="cuda")[:, None, None]
        ro, tt = c(st[4]), c(st[3])
        uu = (c(st[0]) ** 2 + c(st[1]) ** 2 + c(st[2]) ** 2) / (ro * ro)
        g = self.gamma * tt
        if self.case["mag"]:
            g = g + (c(st[5]) ** 2 + c(st[6]) ** 2 + c(st[7]) ** 2) / ro
        fast = uu + g + 2 * torch.sqrt(uu * g)
        got = [(s / torch.sqrt(fast)).min(), (0.5 * s * s * self.re * self.cv * ro).min(), (0.375 * s * s * self.re * ro).min()]
        if self.case["mag"]:
            got.append((0.5 * s * s * RM).min())
        return float(np.float32(0.8)) * float(min(v.item() for v in got))

    def step(self, st):
        dt = self.cfl(st) if self.case["kind"] == "cfl" else DT
        reg = st[:, 1:-1, 1:-1, 1:-1].clone()
        for g, z in zip(self.gam, self.zet):
            for k, f in enumerate(self.rhs(st)):
                new = reg[k] + g * dt * f
                st[k, 1:-1, 1:-1, 1:-1] = new
                reg[k] = new + z * dt * f
            self.walls(st)


def exact(case, seed):
    outs = []
    for k in range(len(_grids(case))):
        plain, st = _Plain(case, seed, k), _fields(case, seed, k)
        if case["kind"] == "rhs":
            flux = torch.zeros_like(st)
            for dst, f in zip((0, 1, 2, 4, 3, 5, 6, 7), plain.rhs(st)):
                flux[dst, 1:-1, 1:-1, 1:-1] = f
            return list(flux)
        for _ in range(case["steps"]):
            plain.step(st)
        outs.append(st.cpu())
    return outs if case["kind"] == "batch" else list(outs[0])
