"""The work that a user of the package has it do, as measurable cases.

A topology-optimisation run is a few dozen SIMP iterations (``SimpRunner.step``: filter and
projection, stiffness, multigrid-preconditioned CG, sensitivity, OC update, history values), then
one as-built check (an FP64 solve to 1e-9 and the von Mises stress) and one surface export; a mesh
part is voxelised before. The iterations take nearly all of the time, so most cases are SIMP
iterations, from the small grids that are tuned interactively to the 12.8M-DOF bracket; the others
are the parts of an iteration through their own entry points (K u, the filter, the update after
the solve) and the calls around the loop.

Every kind of case has one function each for its inputs, its pass and its FP64 values; ``draw``
gives sizes and options of the same ranges. Grids are x-fastest, h = 1.
"""
import functools
import math

import numpy as np
import torch

from anneal_gb300 import export, geometry, optimize, problems
from anneal_gb300.context import Context
from anneal_gb300.fem import FEM, Grid

NU, E0, EMIN, ETA, MOVE, P = 0.3, 1.0, 1e-6, 0.5, 0.2, 3.0
F32, F64, U8 = torch.float32, torch.float64, torch.uint8


def listed():
    return [
        # the 48x24x24 cantilever of the reference's own runs, late in its schedule (projection
        # on): a small interactive part
        {"name": "simp_cantilever_48", "kind": "simp", "part": "cantilever", "nx": 48, "ny": 24, "nz": 24,
         "vf": 0.3, "r": 1.5, "beta": 2.0},
        # an odd-sized part of the many-part set, no projection, a two-element filter halo
        {"name": "simp_cantilever_97x53x34", "kind": "simp", "part": "cantilever", "nx": 97, "ny": 53, "nz": 34,
         "vf": 0.25, "r": 2.4, "beta": 0.0},
        # the L-bracket at half scale (96x48x48): an ordinary part, voids and frozen shells
        {"name": "simp_lbracket_96", "kind": "simp", "part": "lbracket", "scale": 0.5, "vf": 0.25, "r": 2.0,
         "beta": 1.0},
        # six load cases on the bracket (three distinct solves in one batch), 80x40x40
        {"name": "simp_sixcase_80", "kind": "simp", "part": "sixcase", "scale": 5.0 / 12.0, "vf": 0.25, "r": 2.0,
         "beta": 0.0},
        # the 12.8M-DOF bracket of the benchmark (256x128x128)
        {"name": "simp_lbracket_256", "kind": "simp", "part": "lbracket", "scale": 4.0 / 3.0, "vf": 0.25, "r": 2.0,
         "beta": 0.0},
        # the as-built check after a run: an FP64 solve to 1e-9 with host vectors, then the stress
        {"name": "asbuilt_64x32x32", "kind": "asbuilt", "nx": 64, "ny": 32, "nz": 32},
        # one K u: the smallest grid (the validation cantilever's), where the call counts, and the
        # 192x96x96 grid
        {"name": "ku_32x8x12", "kind": "ku", "nx": 32, "ny": 8, "nz": 12},
        {"name": "ku_192x96x96", "kind": "ku", "nx": 192, "ny": 96, "nz": 96},
        # the density filter forward (with projection) and backward
        {"name": "filter_128x64x64", "kind": "filter", "nx": 128, "ny": 64, "nz": 64, "r": 2.6, "beta": 2.0},
        # the rest of an iteration after its solve: sensitivity of two cases, two filter backward
        # passes, the projected OC update, the new physical density and the history values
        {"name": "update_160x80x80", "kind": "update", "nx": 160, "ny": 80, "nz": 80, "r": 1.5, "beta": 4.0,
         "cases": 2},
        # the surface of a finished design, upsampled, smoothed, split into components
        {"name": "surface_96x48x48", "kind": "surface", "nx": 96, "ny": 48, "nz": 48},
        # a mesh part voxelised (27 samples an element)
        {"name": "voxel_128x64x64", "kind": "voxel", "nx": 128, "ny": 64, "nz": 64, "subdivisions": 5},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, lo, hi):
    """A grid longer along x than across, as the parts are; odd sizes among them."""
    nx = _log_int(rng, lo, hi)
    return {"nx": nx, "ny": max(6, int(nx * rng.uniform(0.3, 0.6))), "nz": max(6, int(nx * rng.uniform(0.3, 0.6)))}


def draw(rng):
    kind = rng.choice(["simp"] * 5 + ["asbuilt", "ku", "ku", "filter", "update", "surface", "voxel"])
    r = round(rng.uniform(1.5, 3.2), 2)
    beta = rng.choice([0.0, 0.0, 1.0, 2.0, 4.0])
    if kind == "simp":
        part = rng.choice(["cantilever", "cantilever", "lbracket", "sixcase"])
        c = {"kind": kind, "part": part, "vf": round(rng.uniform(0.2, 0.4), 3), "r": r, "beta": beta}
        if part == "cantilever":
            return {**c, **_dims(rng, 24, 160)}
        lo, hi = (0.3, 1.0) if part == "lbracket" else (0.25, 0.6)
        return {**c, "scale": round(math.exp(rng.uniform(math.log(lo), math.log(hi))), 4)}
    if kind == "asbuilt":
        return {"kind": kind, **_dims(rng, 24, 64)}
    if kind == "ku":
        return {"kind": kind, **_dims(rng, 16, 256)}
    if kind == "filter":
        return {"kind": kind, **_dims(rng, 32, 192), "r": r, "beta": beta}
    if kind == "update":
        return {"kind": kind, **_dims(rng, 32, 192), "r": r, "beta": beta, "cases": rng.randint(1, 3)}
    if kind == "surface":
        return {"kind": kind, **_dims(rng, 32, 128)}
    return {"kind": kind, **_dims(rng, 32, 192), "subdivisions": rng.randint(3, 5)}


# ------------------------------------------------------------------ inputs

def _key(case):
    return tuple(sorted((k, v) for k, v in case.items() if k != "name"))


@functools.lru_cache(maxsize=4)
def _workload(key):
    c = dict(key)
    if c["part"] == "cantilever":
        return problems.cantilever(c["nx"], c["ny"], c["nz"], vf=c["vf"], r_vox=c["r"], emin=EMIN)
    make = problems.six_case_bracket if c["part"] == "sixcase" else problems.lbracket
    return make(scale=c["scale"], vf=c["vf"], r_vox=c["r"], emin=EMIN)


def _shape(case):
    return (case["nx"], case["ny"], case["nz"]) if "nx" in case else _workload(_key(case)).shape


def _noise(shape, seed, cell):
    """Smooth seeded noise of unit scale on an x-fastest (nz, ny, nx) grid, features of about
    `cell` values: what a design's members or a displacement's bends look like."""
    g = torch.Generator().manual_seed(int(seed) * 7919 + 17)
    nx, ny, nz = shape
    z = torch.randn((1, 1, nz // cell + 3, ny // cell + 3, nx // cell + 3), generator=g).cuda()
    return torch.nn.functional.interpolate(z, size=(nz, ny, nx), mode="trilinear", align_corners=True)[0, 0]


def _design(shape, seed, sharp=4.0, least=0.1):
    """Element densities of a developing design in (least, 1), flat, x fastest (float32)."""
    return (least + (1 - least) * torch.sigmoid(sharp * (_noise(shape, seed, 6) - 0.3))).reshape(-1)


def _displacements(shape, seed, cases):
    """(cases, 3 N_n) float64: a cantilever's bend with smooth local variation, zero at x = 0."""
    nx, ny, nz = shape
    n = (nx + 1, ny + 1, nz + 1)
    t = torch.linspace(0, 1, nx + 1, device="cuda", dtype=F64)
    out = torch.empty((cases, nz + 1, ny + 1, nx + 1, 3), device="cuda", dtype=F64)
    for c in range(cases):
        for d in range(3):
            amp = 1.0 if d == 2 - c % 3 else 0.3
            out[c, ..., d] = nx * t * t * amp + t * _noise(n, seed + 31 * c + 7 * d + 1, 8).double()
    return out.reshape(cases, -1)


def _clamped(shape):
    """uint8 per DOF: the x = 0 face clamped."""
    nx, ny, nz = shape
    f = torch.zeros((nz + 1, ny + 1, nx + 1, 3), dtype=U8, device="cuda")
    f[:, :, 0] = 1
    return f.reshape(-1)


def _context(shape, r=None):
    ctx = Context(shape, 1.0, NU)
    ctx.set_domain(torch.ones(ctx.ne, dtype=U8, device="cuda"), _clamped(shape))
    if r is not None:
        ctx.filter_init(r)
    return ctx


def _stiffness(shape, seed):
    return (E0 * (EMIN + _design(shape, seed) ** 3 * (1 - EMIN))).float()


class State:
    def __init__(self, case, **kw):
        self.case = case
        self.__dict__.update(kw)


def _quiet(*a):
    return None


def _prepare_simp(case, seed):
    w = _workload(_key(case))
    x0 = _design(w.shape, seed).double().cpu().numpy()
    run = optimize.SimpRunner(Grid(w.shape, 1.0, (0, 0, 0)), w.fill, w.active, w.frozen, w.fixed, w.loads, w.weights,
                              E0, NU, case["vf"], iters=80, r_mm=case["r"], p_final=P, move=MOVE, x0=x0,
                              beta_max=2 * case["beta"], log=_quiet)
    return State(case, run=run, x=run.x_t.clone())


def _run_simp(s):
    r = s.run
    r.x_t.copy_(s.x)   # the design of this iteration, from a zero displacement
    r.U_t.zero_()
    rec = r.step()
    return {"x": r.x_t, "xphys": r.xphys_t, "dcx": r.dcx_t, "u": r.U_t.float(),
            "compliance": rec["compliance"], "volume": rec["volumeFraction"]}


def _asbuilt_parts(case, seed):
    w = _workload(_key({"part": "cantilever", "vf": 0.3, "r": 1.5, **{k: case[k] for k in ("nx", "ny", "nz")}}))
    return w, (E0 * (EMIN + _design(w.shape, seed, 6.0, 0.05).double() ** 3 * (1 - EMIN)))


def _prepare_asbuilt(case, seed):
    w, Ee = _asbuilt_parts(case, seed)
    fem = FEM(Grid(w.shape, 1.0, (0, 0, 0)), w.active, w.fixed, NU)
    return State(case, fem=fem, Ee=Ee.cpu().numpy(), F=fem.reduce_load(w.loads["c"]))


def _run_asbuilt(s):
    u = s.fem.solve(s.fem.assemble(s.Ee), [s.F], rtol=1e-9)[0]
    return {"u": u, "vm": s.fem.von_mises(s.fem.expand(u), s.Ee)}


def _prepare_ku(case, seed):
    shape = _shape(case)
    ctx = _context(shape)
    u = (_displacements(shape, seed, 1)[0] * (_clamped(shape) == 0)).float()
    return State(case, ctx=ctx, E=_stiffness(shape, seed), u=u, y=torch.empty_like(u))


def _run_ku(s):
    s.ctx.apply_K(s.E, s.u, s.y)
    return s.y


def _prepare_filter(case, seed):
    shape = _shape(case)
    x = _design(shape, seed)
    return State(case, ctx=_context(shape, case["r"]), x=x, dc=-(x + 0.05) ** 2 * torch.exp(_noise(shape, seed + 5, 4).reshape(-1)),
                 frozen=(_noise(shape, seed + 9, 8).reshape(-1) > 1.5).to(U8), xphys=torch.empty_like(x),
                 dxp=torch.empty_like(x), dcx=torch.empty_like(x))


def _run_filter(s):
    s.ctx.physical(s.x, s.frozen, s.case["beta"], ETA, s.xphys, s.dxp)
    s.ctx.filter_bwd(s.dc, s.dcx)
    return {"xphys": s.xphys, "dxp": s.dxp, "dcx": s.dcx}


def _prepare_update(case, seed):
    s = _prepare_filter(case, seed)
    shape, n = _shape(case), case["cases"]
    s.phi = torch.ones_like(s.x)
    s.x = torch.where(s.frozen != 0, torch.ones_like(s.x), s.x * 0.9 + 0.01)
    s.ctx.physical(s.x, s.frozen, case["beta"], ETA, s.xphys, s.dxp)
    s.U = _displacements(shape, seed, n) * (_clamped(shape) == 0)
    s.coef = [1.0 / (1 + c) for c in range(n)]
    s.vtarget = 0.3 * s.x.numel()
    s.dv, s.dvx, s.xnew, s.xphys_new = (torch.empty_like(s.x) for _ in range(4))
    return s


def _run_update(s):
    c, beta = s.ctx, s.case["beta"]
    c.sensitivity(s.U, s.coef, s.xphys, s.dxp, s.phi, P, EMIN, E0, s.dc, s.dv)
    c.filter_bwd(s.dc, s.dcx)
    c.filter_bwd(s.dv, s.dvx)
    c.oc_update(s.x, s.dcx, s.dvx, s.phi, s.frozen, MOVE, beta, ETA, s.vtarget, s.xnew)
    c.physical(s.xnew, s.frozen, beta, ETA, s.xphys_new, None)
    change, _, vol, ndes = c.design_stats(s.x, s.xnew, s.xphys_new, s.phi, s.frozen)
    return {"dc": s.dc, "dcx": s.dcx, "dvx": s.dvx, "xnew": s.xnew, "xphys": s.xphys_new, "change": change,
            "volume": vol, "ndes": ndes}


def _prepare_surface(case, seed):
    shape = _shape(case)
    most = 24 * math.prod(shape) // 10  # the mesh ends up in buffers of one size, as a viewer's are
    return State(case, grid=Grid(shape, 1.0, (0, 0, 0)), vertices=np.zeros((most, 3)),
                 faces=np.zeros((2 * most, 3), np.int64), f=_design(shape, seed, 8.0, 0.0).double().cpu().numpy())


def _run_surface(s):
    m = export.surface(s.grid, s.f, 0.5, log=_quiet)
    nv, nf = len(m.vertices), len(m.faces)
    s.vertices[:nv], s.faces[:nf] = m.vertices, m.faces
    s.vertices[nv:], s.faces[nf:] = 0, -1
    return {"vertices": s.vertices, "faces": s.faces, "counts": [nv, nf]}


@functools.lru_cache(maxsize=3)
def _ball(subdivisions):
    return geometry.icosphere(subdivisions, 1.0)


def _prepare_voxel(case, seed):
    """A lumpy closed body that fills most of the grid."""
    shape = np.array(_shape(case), float)
    v, f = _ball(case["subdivisions"])
    rng = np.random.default_rng(seed)
    k = rng.normal(0.0, 2.5, (6, 3))
    ph = rng.uniform(0, 2 * math.pi, 6)
    rad = 0.8 + 0.03 * np.sin(v @ k.T + ph).sum(axis=1)
    tri = (v * rad[:, None] * shape / 2 + shape / 2)[f]
    return State(case, grid=Grid(_shape(case), 1.0, (0, 0, 0)), tri=tri)


def _run_voxel(s):
    return geometry.voxel_fill(s.tri, s.grid, s=3)


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return globals()["_run_" + state.case["kind"]](state)


# ------------------------------------------------------------------ what a pass cannot do without

def work(case):
    """Inputs read once and outputs written once. A solve's flops: one K u per distinct case,
    about 210 operations an element in the cheapest known form of the element product (its
    solution has at least to meet its residual)."""
    nx, ny, nz = _shape(case)
    ne, nn = nx * ny * nz, (nx + 1) * (ny + 1) * (nz + 1)
    kind = case["kind"]
    taps = (2 * max(math.ceil(case.get("r", 1.5)) - 1, 1) + 1) ** 3
    if kind == "simp":
        given = 6 if case["part"] == "sixcase" else 1
        solved = 3 if case["part"] == "sixcase" else 1
        # x, phi, the active and frozen flags, F and U in; x, xphys, dcx and U out
        return {"bytes": 10 * ne + 12 * ne + given * (24 + 36) * nn, "flops": (solved * 420 + 8 * taps) * ne}
    if kind == "asbuilt":
        return {"bytes": 8 * ne + 24 * nn + 24 * nn + 8 * ne, "flops": (210 + 60) * ne}
    if kind == "ku":
        return {"bytes": 4 * ne + 24 * nn, "flops": 210 * ne}
    if kind == "filter":
        return {"bytes": (4 + 4 + 1 + 12) * ne, "flops": 4 * taps * ne}
    if kind == "update":
        return {"bytes": (4 * 4 + 1 + 5 * 4) * ne + case["cases"] * 24 * nn, "flops": (210 * case["cases"] + 8 * taps) * ne}
    if kind == "surface":
        # the field in, the mesh out: about one cut cell in eight of the 8 N_e upsampled ones,
        # a vertex (24 bytes) and two faces (48 bytes) each
        return {"bytes": 8 * ne + 72 * ne, "flops": 8 * 20 * ne}
    return {"bytes": 8 * ne + 72 * 20 * 4 ** case["subdivisions"], "flops": 27 * ne}


# ------------------------------------------------------------------ the same in 64 bits

def exact(case, seed):
    return globals()["_exact_" + case["kind"]](case, seed)


def _ke64():
    """Hex8 stiffness of a unit cube, unit modulus, corner = px + 2 py + 4 pz (2x2x2 Gauss)."""
    s = np.array([[(c >> d & 1) * 2 - 1 for d in range(3)] for c in range(8)], float)
    lam, mu = NU / ((1 + NU) * (1 - 2 * NU)), 1 / (2 * (1 + NU))
    D = np.diag([2 * mu] * 3 + [mu] * 3)
    D[:3, :3] += lam
    K = np.zeros((24, 24))
    for q in range(8):
        g = s[q] / math.sqrt(3)
        one = 1 + s * g
        dN = np.stack([s[:, 0] * one[:, 1] * one[:, 2], s[:, 1] * one[:, 0] * one[:, 2], s[:, 2] * one[:, 0] * one[:, 1]], 1) / 4
        B = np.zeros((6, 24))
        B[0, 0::3], B[1, 1::3], B[2, 2::3] = dN.T
        B[3, 0::3], B[3, 1::3] = dN[:, 1], dN[:, 0]
        B[4, 1::3], B[4, 2::3] = dN[:, 2], dN[:, 1]
        B[5, 0::3], B[5, 2::3] = dN[:, 2], dN[:, 0]
        K += B.T @ D @ B / 8
    return torch.tensor(K, device="cuda")


class _Solid64:
    """K u, energies and a Jacobi-CG solve in 64 bits with plain torch, on (nz+1, ny+1, nx+1, 3) fields."""

    def __init__(self, shape, E, free):
        self.shape, self.K = shape, _ke64()
        self.E = E.reshape(shape[::-1]).double()
        self.free = free.reshape(shape[2] + 1, shape[1] + 1, shape[0] + 1, 3)

    def _corner(self, c):
        nx, ny, nz = self.shape
        i, j, k = c & 1, c >> 1 & 1, c >> 2
        return slice(k, nz + k), slice(j, ny + j), slice(i, nx + i)

    def gather(self, u):
        return torch.cat([u[self._corner(c)] for c in range(8)], -1)

    def apply(self, u):
        f = (self.gather(u) @ self.K) * self.E[..., None]
        y = torch.zeros_like(u)
        for c in range(8):
            y[self._corner(c)] += f[..., 3 * c:3 * c + 3]
        return y * self.free

    def energy(self, u):
        g = self.gather(u.reshape(self.free.shape))
        return ((g @ self.K) * g).sum(-1).reshape(-1)

    def solve(self, F, rtol):
        b = F.reshape(self.free.shape) * self.free
        d = torch.zeros(self.free.shape[:3], device="cuda", dtype=F64)
        for c in range(8):
            d[self._corner(c)] += self.E * self.K[0, 0]
        dinv = torch.where(d > 0, 1 / d, torch.zeros_like(d))[..., None]
        x, r = torch.zeros_like(b), b.clone()
        z = dinv * r
        p, rz, bb = z.clone(), (r * z).sum(), (b * b).sum()
        for it in range(40000):
            q = self.apply(p)
            a = rz / (p * q).sum()
            x += a * p
            r -= a * q
            z = dinv * r
            new = (r * z).sum()
            p = z + (new / rz) * p
            rz = new
            if it % 100 == 99 and float((r * r).sum() / bb) < rtol ** 2:
                break
        return x.reshape(-1)


def _cone64(r):
    R = max(math.ceil(r) - 1, 1)
    return [(dx, dy, dz, r - math.sqrt(dx * dx + dy * dy + dz * dz)) for dz in range(-R, R + 1)
            for dy in range(-R, R + 1) for dx in range(-R, R + 1) if r - math.sqrt(dx * dx + dy * dy + dz * dz) > 0], R


class _Filter64:
    def __init__(self, shape, r, active):
        self.taps, self.R = _cone64(r)
        self.size, self.act = shape[::-1], active.reshape(shape[::-1]).double()
        self.Hs = self._conv(self.act)
        self.Hs = torch.where(self.Hs == 0, torch.ones_like(self.Hs), self.Hs)

    def _conv(self, v):
        (nz, ny, nx), R = self.size, self.R
        p = torch.nn.functional.pad(v, (R,) * 6)
        out = torch.zeros_like(v)
        for dx, dy, dz, w in self.taps:
            out += w * p[R + dz:R + dz + nz, R + dy:R + dy + ny, R + dx:R + dx + nx]
        return out

    def fwd(self, x):
        return (self._conv(x.reshape(self.size) * self.act) / self.Hs * self.act).reshape(-1)

    def bwd(self, d):
        return (self._conv(d.reshape(self.size) * self.act / self.Hs) * self.act).reshape(-1)

    def physical(self, x, frozen, beta):
        xt, act = self.fwd(x), self.act.reshape(-1)
        xp, g = xt, torch.ones_like(xt)
        if beta > 0:
            t0, t1 = math.tanh(beta * ETA), math.tanh(beta * (1 - ETA))
            th = torch.tanh(beta * (xt - ETA))
            xp, g = (t0 + th) / (t0 + t1), beta * (1 - th * th) / (t0 + t1)
        return torch.where(frozen, torch.ones_like(xp), xp) * act, g * act


def _oc64(flt, x, dcx, dvx, phi, frozen, beta, vtarget):
    act = flt.act.reshape(-1) > 0
    des = act & ~frozen
    scale = max(float(-dcx[des].mean()) / max(float(dvx[des].mean()), 1e-30), 1e-300)
    lo, hi, mv = scale * 1e-8, scale * 1e8, MOVE if beta <= 1 else MOVE / 2
    for _ in range(100):
        lam = math.sqrt(lo * hi)
        xn = x * torch.sqrt(torch.clamp(-dcx, min=0) / torch.clamp(dvx * lam, min=1e-300))
        xn = torch.minimum(torch.maximum(xn, torch.clamp(x - mv, min=0)), torch.clamp(x + mv, max=1))
        xn = torch.where(frozen, torch.ones_like(xn), xn) * act
        vol = float((phi * flt.physical(xn, frozen, beta)[0]).sum())
        lo, hi = (lam, hi) if vol > vtarget else (lo, lam)
        if hi / lo < 1 + 1e-9:
            break
    return xn


def _sens64(solid, us, coef, xphys, dxp, phi):
    pre = -P * xphys ** (P - 1) * (1 - EMIN) * E0 * phi
    dc = sum(c * pre * solid.energy(u) for c, u in zip(coef, us))
    return torch.clamp(dc, max=0) * dxp


def _exact_simp(case, seed):
    w = _workload(_key(case))
    if w.nelem > 260_000:
        return None   # the plain CG would take minutes
    dev = lambda a, t=F64: torch.as_tensor(np.ascontiguousarray(a), device="cuda").to(t)  # noqa: E731
    active, frozen, phi = dev(w.active, torch.bool), dev(w.frozen, torch.bool) & dev(w.active, torch.bool), dev(w.fill)
    phi = phi * active
    beta = case["beta"]
    des = active & ~frozen
    vtot = float(phi.sum())
    vt, vfz = case["vf"] * vtot, float(phi[frozen].sum())
    xs = torch.clamp(_design(w.shape, seed).double(), 0, 1)
    cur = float((phi * xs)[des].sum())
    x = torch.where(des, torch.clamp(xs * (vt - vfz) / cur, 0.001, 1.0), torch.ones_like(xs)) * active
    x = x.float().double()  # the design is float32 data
    flt = _Filter64(w.shape, max(case["r"], 1.5), active)
    xphys, dxp = flt.physical(x, frozen, beta)
    E = E0 * phi * (EMIN + xphys ** P * (1 - EMIN))
    used = dev(problems.used_nodes(w.shape, w.active), torch.bool)
    free = used[:, None].expand(-1, 3).clone().reshape(-1)
    free[dev(w.fixed, torch.int64)] = False
    solid = _Solid64(w.shape, E, free.double())
    us = {}
    for name, F in w.loads.items():  # -x is the negative of +x: solved once
        f = dev(F)
        for other, (g, u) in us.items():
            if torch.equal(f, -g):
                us[name] = (f, -u)
                break
        else:
            us[name] = (f, solid.solve(f, 1e-11))
    comp = [float((f * free * u).sum()) for f, u in us.values()]
    out = _sens64(solid, [u for _, u in us.values()], [1.0] * len(us), xphys, dxp, phi)
    dcx, dvx = flt.bwd(out), flt.bwd(phi * dxp)
    xn = _oc64(flt, x, dcx, dvx, phi, frozen, beta, vt)
    xp = flt.physical(xn, frozen, beta)[0]
    return {"x": xn, "xphys": xp, "dcx": dcx, "u": torch.stack([u for _, u in us.values()]), "compliance": comp,
            "volume": float((phi * xp).sum()) / vtot}


def _exact_asbuilt(case, seed):
    if case["nx"] * case["ny"] * case["nz"] > 120_000:
        return None
    w, Ee = _asbuilt_parts(case, seed)
    free = (_clamped(w.shape) == 0).double()
    solid = _Solid64(w.shape, Ee.float(), free)   # element scales are float32 data
    u = solid.solve(torch.as_tensor(w.loads["c"], device="cuda"), 1e-13)
    g = solid.gather(u.reshape(solid.free.shape)).reshape(-1, 8, 3)
    s = torch.tensor([[(c >> d & 1) * 2 - 1 for d in range(3)] for c in range(8)], device="cuda", dtype=F64) / 4
    G = torch.einsum("ecd,ck->edk", g, s)    # du_d / dx_k at the centre
    eps = (G + G.transpose(1, 2)) / 2
    lam, mu = NU / ((1 + NU) * (1 - 2 * NU)), 1 / (2 * (1 + NU))
    eye = torch.eye(3, device="cuda", dtype=F64)
    sig = Ee[:, None, None] * (lam * eps.diagonal(dim1=1, dim2=2).sum(-1)[:, None, None] * eye + 2 * mu * eps)
    dev = sig - sig.diagonal(dim1=1, dim2=2).mean(-1)[:, None, None] * eye
    return {"u": u[free > 0], "vm": torch.sqrt(1.5 * (dev * dev).sum((1, 2)))}


def _exact_ku(case, seed):
    shape = _shape(case)
    free = (_clamped(shape) == 0).double()
    solid = _Solid64(shape, _stiffness(shape, seed), free)
    u = (_displacements(shape, seed, 1)[0] * free).float().double()
    return solid.apply(u.reshape(solid.free.shape)).reshape(-1)


def _inputs64(case, seed):
    """The filter and the inputs of the filter and update cases, without the package."""
    shape = _shape(case)
    x = _design(shape, seed)
    dc = (-(x + 0.05) ** 2 * torch.exp(_noise(shape, seed + 5, 4).reshape(-1))).double()
    frozen = _noise(shape, seed + 9, 8).reshape(-1) > 1.5
    return _Filter64(shape, case["r"], torch.ones_like(x)), x, dc, frozen


def _exact_filter(case, seed):
    flt, x, dc, frozen = _inputs64(case, seed)
    xphys, dxp = flt.physical(x.double(), frozen, case["beta"])
    return {"xphys": xphys, "dxp": dxp, "dcx": flt.bwd(dc)}


def _exact_update(case, seed):
    shape, beta, n = _shape(case), case["beta"], case["cases"]
    flt, x, _, frozen = _inputs64(case, seed)
    x = torch.where(frozen, torch.ones_like(x), x * 0.9 + 0.01).double()
    xphys, dxp = flt.physical(x, frozen, beta)
    free = (_clamped(shape) == 0).double()
    solid = _Solid64(shape, torch.ones_like(x), free)
    us = _displacements(shape, seed, n) * free
    phi = torch.ones_like(x)
    dc = _sens64(solid, us, [1.0 / (1 + c) for c in range(n)], xphys, dxp, phi)
    dcx, dvx = flt.bwd(dc), flt.bwd(phi * dxp)
    xn = _oc64(flt, x, dcx, dvx, phi, frozen, beta, 0.3 * x.numel())
    xp = flt.physical(xn, frozen, beta)[0]
    des = ~frozen
    return {"dc": dc, "dcx": dcx, "dvx": dvx, "xnew": xn, "xphys": xp, "change": float((xn - x)[des].abs().max()),
            "volume": float(xp.sum()), "ndes": int(des.sum())}


def _exact_surface(case, seed):
    return None   # the numbering of a mesh is the library's own: compared vertex by vertex


def _exact_voxel(case, seed):
    return None   # fractions of 27 samples, compared bit for bit
