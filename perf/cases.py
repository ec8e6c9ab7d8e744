"""Performance cases of the level-step library, through its public entry points.

Each case is a dict of plain values; ``prepare`` builds what a program holds
(solver, fields and body from a seed, the first step taken, which builds a
body's operator), ``run`` takes one pass of it, ``work`` gives the bytes and
operations the pass cannot do without and ``exact`` the pass's outputs in 64
bits from plain torch.

Kinds:
  channel    D2Q9, force-driven, halfway bounce-back walls (LevelSolver)
  tgv        D2Q9 Taylor-Green box, periodic (LevelSolver)
  duct       D3Q19 / D3Q27 square duct, user_2 walls, uniform force (LevelSolver)
  cylinder   D2Q9 flow past a fixed cylinder, its force record every step
  airfoil    D2Q9 pitching NACA section (operator rebuilt every step), recorded
  sphere     D3Q19 / D3Q27 flow past a fixed sphere, recorded
  boxes      one level in several caller-filled boxes in AMReX's own array
             layout with stored macro fields (the drop-in inside AMReX)
  hierarchy  D2Q9 cylinder or D3Q19 sphere with refined levels
  batch      many D2Q9 cases advanced together by the batch engine
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from ilbmrex_b200 import capi, cases
from ilbmrex_b200.batch import Batch
from ilbmrex_b200.hierarchy import HierarchySolver, TwoLevelSolver
from ilbmrex_b200.lattice import D2Q9, D3Q19, D3Q27
from ilbmrex_b200.level import Context, LevelSolver, level_params

LATTICE = {9: D2Q9, 19: D3Q19, 27: D3Q27}
BYTES = {"f64": 8, "f32": 4, "f16": 2}
TORCH = {"f64": torch.float64, "f32": torch.float32, "f16": torch.float16}
F16_SCALE = 1024.0


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest call a program makes: one step of a small wall-bounded
        # level, where the launch and the host path are the time
        dict(name="channel_64x48_f64", kind="channel", q=9, storage="f64", nx=64, ny=48, nz=1, steps=1),
        # the Taylor-Green verification run (256 x 256, FP64, the parity form)
        dict(name="tgv_256_f64", kind="tgv", q=9, storage="f64", nx=256, ny=256, nz=1, steps=4),
        # the 2D cylinder deck on one level with its force record every step
        dict(name="cylinder_1024x512_f32", kind="cylinder", q=9, storage="f32", nx=1024, ny=512, nz=1,
             body=40.0, steps=10),
        # a moving body: the pitching airfoil on an odd-sized level
        dict(name="airfoil_501x255_f32", kind="airfoil", q=9, storage="f32", nx=501, ny=255, nz=1,
             body=80.0, steps=10),
        # the sphere in the parity form at half the benchmark's resolution
        dict(name="sphere_128x64x64_f64", kind="sphere", q=19, storage="f64", nx=128, ny=64, nz=64,
             body=16.0, steps=2),
        # the sphere's base level of the benchmark in the 2-byte form
        dict(name="sphere_256x128x128_f16", kind="sphere", q=19, storage="f16", nx=256, ny=128, nz=128,
             body=32.0, steps=2),
        # the sphere deck's own lattice (D3Q27), ragged sizes
        dict(name="sphere_150x75x83_q27_f32", kind="sphere", q=27, storage="f32", nx=150, ny=75, nz=83,
             body=20.0, steps=2),
        # the largest served request: a 128-wide duct four times as long
        dict(name="duct_512x128x128_f32", kind="duct", q=19, storage="f32", nx=512, ny=128, nz=128, steps=2),
        # the AMReX drop-in: an FP64 level cut into 12 boxes, stored macro fields
        dict(name="boxes_150x100x90_f64", kind="boxes", q=19, storage="f64", nx=150, ny=100, nz=90,
             cut=50, steps=1),
        # the benchmark: the sphere with one refined level, recorded every step
        dict(name="sphere_two_level_f32", kind="hierarchy", q=19, storage="f32", nx=256, ny=128, nz=128,
             body=32.0, nlev=2, steps=2),
        # the cylinder wake with two refined levels, replayed from a graph
        dict(name="cylinder_three_level_f32", kind="hierarchy", q=9, storage="f32", nx=1024, ny=512, nz=1,
             body=40.0, nlev=3, steps=10),
        # the batch engine on a mix of fixed and pitching bodies
        dict(name="batch_32_f32", kind="batch", q=9, storage="f32", nx=1024, ny=512, nz=1, ncase=32, steps=10),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["channel", "tgv", "duct", "cylinder", "airfoil", "sphere", "boxes", "hierarchy", "batch"])
    storage = rng.choice(["f64", "f32", "f32", "f16"])
    if kind in ("channel", "tgv"):
        nx = _log_int(rng, 33, 2048)
        return dict(kind=kind, q=9, storage=storage, nx=nx, ny=_log_int(rng, 33, 1024) if kind == "channel" else nx,
                    nz=1, steps=rng.choice([1, 4]))
    if kind == "duct":
        n = _log_int(rng, 24, 96)
        return dict(kind=kind, q=rng.choice([19, 27]), storage=storage, nx=_log_int(rng, n, 4 * n), ny=n, nz=n, steps=2)
    if kind == "cylinder":
        ny = _log_int(rng, 96, 512)
        return dict(kind=kind, q=9, storage=storage, nx=_log_int(rng, ny + 32, 1024), ny=ny, nz=1,
                    body=round(rng.uniform(0.1, 0.2) * ny, 2), steps=10)
    if kind == "airfoil":
        ny = _log_int(rng, 128, 512)
        return dict(kind=kind, q=9, storage=rng.choice(["f64", "f32"]), nx=_log_int(rng, ny + 64, 1024), ny=ny, nz=1,
                    body=round(rng.uniform(0.25, 0.4) * ny, 2), steps=10)
    if kind == "sphere":
        n = _log_int(rng, 48, 112)
        return dict(kind=kind, q=rng.choice([19, 27]), storage=storage, nx=_log_int(rng, n + 32, 2 * n), ny=n,
                    nz=max(48, n + rng.randint(-5, 5)), body=round(rng.uniform(0.2, 0.28) * 48 * (n / 48.0), 2), steps=2)
    if kind == "boxes":
        n = _log_int(rng, 40, 110)
        return dict(kind=kind, q=rng.choice([19, 27]), storage="f64", nx=_log_int(rng, n, 2 * n), ny=n,
                    nz=max(32, n - rng.randint(0, 9)), cut=max(rng.choice([32, 48, 64]), -(-n // 2)), steps=1)
    if kind == "hierarchy":
        if rng.random() < 0.5:
            n = _log_int(rng, 64, 112)
            return dict(kind=kind, q=19, storage=storage, nx=2 * n + rng.randint(0, 9), ny=n, nz=n,
                        body=round(rng.uniform(0.2, 0.25) * n, 2), nlev=2, steps=2)
        ny = _log_int(rng, 256, 512)
        return dict(kind=kind, q=9, storage=rng.choice(["f64", "f32"]), nx=2 * ny + rng.randint(0, 40), ny=ny, nz=1,
                    body=round(rng.uniform(0.06, 0.09) * ny, 2), nlev=rng.choice([2, 3]), steps=10)
    return dict(kind="batch", q=9, storage=rng.choice(["f32", "f64"]), nx=_log_int(rng, 256, 768), ny=_log_int(rng, 128, 384),
                nz=1, ncase=rng.randint(4, 24), steps=10)


# ---------------------------------------------------------------------------
# inputs: level and body descriptions with seeded positions and flow
# ---------------------------------------------------------------------------
def _modes(rng, dim, amp):
    """Three smooth velocity perturbations, each a product of one cosine per direction."""
    return [(amp * rng.uniform(0.3, 1.0), rng.integers(0, dim), rng.integers(1, 4, 3), rng.uniform(0, 2 * np.pi, 3))
            for _ in range(3)]


def _init(box, ext, dim, base, modes):
    """rho, u, v, w at the cell centres of a level box (``ext``: the domain's extent)."""
    shape, dx = box.shape, box.dx
    ax = [(box.prob_lo[d] + (np.arange(box.n_cell[d]) + 0.5) * dx) / ext[d] for d in range(3)]

    def fn():
        out = [np.full(shape, b) for b in (1.0,) + tuple(base)]
        for a, c, k, ph in modes:
            t = [np.cos(2 * np.pi * k[d] * ax[d] + ph[d]) if d < dim else np.ones(1) for d in range(3)]
            prod = t[2][:, None, None] * t[1][None, :, None] * t[0][None, None, :]
            out[1 + c] += a * prod
            out[0] += 0.1 * a * prod
        return tuple(out)

    return fn


def _single(c, rng):
    """(LevelCase, MarkerIB or None, init) of a single-level case."""
    nx, ny, nz, lat = c["nx"], c["ny"], c["nz"], LATTICE[c["q"]]
    U = 0.05 if lat.dim == 2 else 0.04
    jit = rng.uniform(-0.4, 0.4, 3)
    ib, base, amp = None, (0.0, 0.0, 0.0), 0.02
    if c["kind"] == "channel":
        case, _ = cases.channel_bounce_back(nx=nx, ny=ny, force=1e-5)
    elif c["kind"] == "tgv":
        case, _ = cases.taylor_green(nx, U0=0.02, tau=0.8)
    elif c["kind"] == "duct":
        case, _ = cases.square_duct(N=ny, L=nx, force=1e-5, lattice=lat)
    elif c["kind"] == "cylinder":
        case, ib, _ = cases.cylinder(nx=nx, ny=ny, D=c["body"], center=(0.25 * nx + jit[0], 0.5 * ny + jit[1]), U=U)
        base, amp = (U, 0.0, 0.0), 0.1 * U
    elif c["kind"] == "airfoil":
        case, ib, _ = cases.pitching_airfoil(nx=nx, ny=ny, chord=c["body"], pivot=(0.3 * nx + jit[0], 0.5 * ny + jit[1]),
                                             U=U)
        base, amp = (U, 0.0, 0.0), 0.1 * U
    else:
        case, ib, _ = cases.sphere(nx, ny, nz, D=c["body"], U=U, Re=60.0, lattice=lat,
                                   center=(0.3 * nx + jit[0], 0.5 * ny + jit[1], 0.5 * nz + jit[2]))
        base, amp = (U, 0.0, 0.0), 0.1 * U
    ext = [case.prob_hi[d] - case.prob_lo[d] for d in range(3)]
    return case, ib, _init(case, ext, lat.dim, base, _modes(rng, lat.dim, amp))


def _hierarchy(c, rng):
    """(HierarchyCase or TwoLevelCase, MarkerIB, inits)."""
    nx, ny, nz, D = c["nx"], c["ny"], c["nz"], c["body"]
    dim = 3 if c["q"] == 19 else 2
    U = 0.05 if dim == 2 else 0.04
    ctr = (0.25 * nx, 0.5 * ny, 0.5 * nz)
    if dim == 3:
        lo = [int(v - D) for v in ctr]
        hi = [int(ctr[0] + 2.0 * D), int(ctr[1] + D), int(ctr[2] + D)]
        hc, ib, _, _ = cases.sphere_two_level(nx, ny, nz, D=D, center=ctr, U=U, box_lo=lo, box_hi=hi)
        boxes = [hc.coarse, hc.fine_box()]
    else:
        hc, ib, _ = cases.cylinder_hierarchy(nx=nx, ny=ny, D=D, center=ctr[:2], U=U, nlev=c["nlev"], upstream=0.65,
                                             downstream=2.15, cross=1.15, inflow_uy=1e-4)
        boxes = [hc.box_case(l) for l in range(c["nlev"])]
    jit = rng.uniform(-0.2, 0.2, 3)                      # the body within the fixed boxes
    ib.x0, ib.y0, ib.z0 = ib.x0 + jit[0], ib.y0 + jit[1], ib.z0 + (jit[2] if dim == 3 else 0.0)
    ext = [hc.coarse.prob_hi[d] - hc.coarse.prob_lo[d] for d in range(3)]
    modes = _modes(rng, dim, 0.1 * U)
    return hc, ib, [_init(b, ext, dim, (U, 0.0, 0.0), modes) for b in boxes]


def _batch(c, rng):
    """[(LevelCase, MarkerIB, init)] of a batch: cylinders and airfoils in turn, sizes up to nx x ny."""
    out = []
    for n in range(c["ncase"]):
        nx = max(128, int(c["nx"] * (0.3 + 0.7 * ((37 * n + 11) % 64) / 63.0)))
        ny = max(96, int(c["ny"] * (0.3 + 0.7 * ((23 * n + 5) % 64) / 63.0)))
        kind = "airfoil" if n % 2 else "cylinder"
        body = max(12.0, min(0.15 * ny, 48.0)) if kind == "cylinder" else min(0.35 * ny, 0.4 * nx, 128.0)
        out.append(_single(dict(c, kind=kind, nx=nx, ny=ny, body=body), rng))
    return out


def _box_cuts(c):
    """Valid ranges (lo, hi) of the boxes of a level cut into pieces of about ``cut`` cells."""
    def axis(n):
        k = max(1, -(-n // c["cut"]))
        e = [round(n * i / k) for i in range(k + 1)]
        return [(e[i], e[i + 1] - 1) for i in range(k)]
    return [((x[0], y[0], z[0]), (x[1], y[1], z[1])) for z in axis(c["nz"]) for y in axis(c["ny"]) for x in axis(c["nx"])]


def _boxes_input(c, seed, device):
    """Populations [Q, nz, ny, nx] and macro fields [4, ...] of a periodic level in 64 bits: smooth flow
    plus the small deviations from equilibrium that a running flow carries."""
    lat = LATTICE[c["q"]]
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    n = (c["nz"], c["ny"], c["nx"])
    x = [torch.arange(m, device=device, dtype=torch.float64) * (2 * math.pi / m) for m in n]
    ph = torch.rand(12, generator=g, device=device, dtype=torch.float64) * 2 * math.pi
    u = [0.03 * torch.cos(x[0] + ph[d])[:, None, None] * torch.sin(x[1] + ph[3 + d])[None, :, None] *
         torch.cos(x[2] + ph[6 + d])[None, None, :] for d in range(3)]
    rho = 1.0 + 0.002 * torch.cos(x[0] + ph[9])[:, None, None] * torch.cos(x[2] + ph[10])[None, None, :].expand(n)
    f = torch.empty((lat.q,) + n, device=device, dtype=torch.float64)
    for q in range(lat.q):
        f[q] = _feq(lat, q, rho, u) + 1e-5 * lat.w[q] * torch.randn(n, generator=g, device=device, dtype=torch.float64)
    rho = f.sum(0)
    m = torch.stack([rho] + [sum(lat.c[q][d] * f[q] for q in range(lat.q)) / rho for d in range(3)])
    return f, m


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
_CONTEXTS = {}


def _context(q, storage):
    """One context per lattice and storage form, which a program's solvers share."""
    if (q, storage) not in _CONTEXTS:
        _CONTEXTS[q, storage] = Context(LATTICE[q], storage)
    return _CONTEXTS[q, storage]


class _Held:
    """A solver that gives its device objects back with the state."""

    def __init__(self, obj):
        self.obj = obj

    def __del__(self):
        try:
            self.obj.close()
        except Exception:
            pass


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    c = dict(case)
    st = dict(case=c)
    if c["kind"] == "boxes":
        return _prepare_boxes(c, seed, st)
    if c["kind"] == "hierarchy":
        hc, ib, inits = _hierarchy(c, rng)
        s = (TwoLevelSolver if c["q"] == 19 else HierarchySolver)(hc, c["storage"], ib=ib, graphs=c["q"] == 9)
        s.set_macro(*[i() for i in inits])
        s.step(1)
        s.ctx.sync()
        return dict(st, s=s, held=_Held(s))
    if c["kind"] == "batch":
        b = Batch(LATTICE[c["q"]], c["storage"])
        ids = [b.add(b.solver(k, ib, init), max_steps=100000) for k, ib, init in _batch(c, rng)]
        return dict(st, s=b, ids=ids, held=_Held(b))
    k, ib, init = _single(c, rng)
    s = LevelSolver(k, c["storage"], ib=ib, ctx=_context(c["q"], c["storage"]))
    s.set_macro(*init())
    s.step(1, record_force=ib is not None)
    s.ctx.sync()
    return dict(st, s=s, held=_Held(s))


def _prepare_boxes(c, seed, st):
    dev = torch.device("cuda")
    lat = LATTICE[c["q"]]
    ctx = _context(c["q"], c["storage"])
    f, m = _boxes_input(c, seed, dev)
    pad = lambda t, w: torch.nn.functional.pad(t[None], (w,) * 6, mode="circular")[0]
    f1, m2 = pad(f, 1), pad(m, 2)
    cuts = _box_cuts(c)
    arr, keep, lb = (capi.Box_t * len(cuts))(), [], []
    for b, (lo, hi) in zip(arr, cuts):
        n = [hi[d] - lo[d] + 1 for d in range(3)]
        cutout = lambda t, w: t[:, lo[2]:hi[2] + 1 + 2 * w, lo[1]:hi[1] + 1 + 2 * w, lo[0]:hi[0] + 1 + 2 * w].contiguous()
        fi, mi = cutout(f1, 1), cutout(m2, 2)
        fo, mo = torch.zeros_like(fi), torch.zeros_like(mi)
        keep.append((fi, fo, mi, mo))
        for d in range(3):
            b.lo[d], b.hi[d] = lo[d], hi[d]
        b.ngrow_f, b.ngrow_m = 1, 2
        b.fstride[:] = [n[0] + 2, (n[0] + 2) * (n[1] + 2), (n[0] + 2) * (n[1] + 2) * (n[2] + 2)]
        b.mstride[:] = [n[0] + 4, (n[0] + 4) * (n[1] + 4), (n[0] + 4) * (n[1] + 4) * (n[2] + 4)]
        b.f_in, b.f_out, b.macro_in, b.macro_out = (t.data_ptr() for t in (fi, fo, mi, mo))
        lb += [*lo, *hi]
    level = cases.LevelCase(lat, (c["nx"], c["ny"], c["nz"]), nu=0.05)
    p = level_params(level, uniform_force=False)
    lb = (ctypes.c_int * len(lb))(*lb)
    p.ghost_mode = capi.GHOST_CALLER
    p.level_boxes = ctypes.cast(lb, ctypes.POINTER(ctypes.c_int))
    p.nlevel_boxes = len(cuts)
    torch.cuda.synchronize()
    return dict(st, ctx=ctx, arr=arr, keep=keep, lb=lb, p=p)


def _narrow(rec, storage):
    """A force record is as exact as the populations it comes from."""
    return np.asarray(rec, dtype=np.float64 if storage == "f64" else np.float32)


def run(state):
    c, s = state["case"], state.get("s")
    if c["kind"] == "boxes":
        ctx = state["ctx"]
        capi.check(ctx.L.ilbm_level_step(ctx.h, state["arr"], len(state["keep"]), ctypes.byref(state["p"])), "level_step")
        return [(fo[:, 1:-1, 1:-1, 1:-1], mo[:, 2:-2, 2:-2, 2:-2]) for _, fo, _, mo in state["keep"]]
    if c["kind"] == "hierarchy":
        if c["q"] == 19:
            s.step(c["steps"], record_force=True, pipelined=True)   # a record every step, taken one step behind
        else:
            s.step(c["steps"])
            s.compute_ib_force()                                    # one record after the steps
        return dict(f=[lv.valid(lv.f, lv.gf) for lv in s.levels], force=s.F.valid(s.F.fb, s.F.gm)[:s.dim],
                    rec=_narrow(s.rec, c["storage"]))
    if c["kind"] == "batch":
        s.step(c["steps"])
        s.progress()                                                # the server's look at who is done
        return [m._valid(m.f, m.gf) for m in (s.members[i] for i in state["ids"])]
    if s.ib is None:
        s.step(c["steps"])
        return s._valid(s.f, s.gf)
    rec = s.run_recorded(c["steps"])
    return dict(f=s._valid(s.f, s.gf), force=s._valid(s.force_prev, s.gm)[:s.dim], rec=_narrow(rec, c["storage"]))


# ---------------------------------------------------------------------------
# work: each step reads and writes every population once
# ---------------------------------------------------------------------------
def work(case):
    c = dict(case)
    rng = np.random.default_rng(0)
    q, b = c["q"], BYTES[c["storage"]]
    if c["kind"] == "batch":
        cells = sum(k.cells for k, _, _ in _batch(c, rng))
    elif c["kind"] == "hierarchy":
        hc, _, _ = _hierarchy(c, rng)
        cells = (hc.coarse.cells + 2 * int(np.prod(hc.fine_n_cell[:hc.dim])) if hasattr(hc, "fine_n_cell")
                 else hc.updates_per_coarse_step())
    else:
        cells = c["nx"] * c["ny"] * c["nz"]
    per_cell = 2 * q * b + (64 if c["kind"] == "boxes" else 0)      # boxes: rho, u read and written too
    return {"bytes": float(per_cell * cells * c["steps"]), "flops": float(14 * q * cells * c["steps"])}


# ---------------------------------------------------------------------------
# exact: the same pass in 64 bits, plain torch
# ---------------------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _feq(lat, q, rho, u):
    cu = sum(lat.c[q][d] * u[d] for d in range(3))
    return lat.w[q] * rho * (1.0 + 3.0 * cu + 4.5 * cu * cu - 1.5 * sum(v * v for v in u))


class _Level:
    """One level in one box: populations and stored macro fields on its cells."""

    def __init__(self, lat, box, tau, dx, init, fill, force=(0.0, 0.0, 0.0)):
        self.lat, self.box, self.tau, self.dx, self.fill = lat, box, tau, dx, fill
        t = [torch.tensor(v, dtype=torch.float64, device=_dev()) for v in init]
        self.m = torch.stack(t)
        self.f = torch.stack([_feq(lat, q, self.m[0], self.m[1:]) for q in range(lat.q)])
        self.F = [torch.full_like(self.m[0], v) for v in force]

    def step(self):
        lat, m = self.lat, self.m
        u, F, om = m[1:], self.F, 1.0 / self.tau
        post = torch.empty_like(self.f)
        for q in range(lat.q):
            c = lat.c[q]
            cu = sum(c[d] * u[d] for d in range(3))
            si = sum(((c[d] - u[d]) * 3.0 + 9.0 * cu * c[d]) * F[d] for d in range(lat.dim))
            post[q] = self.f[q] - om * (self.f[q] - _feq(lat, q, m[0], u)) + lat.w[q] * (1.0 - 0.5 * om) * si
        self.f = self.fill(self, post)
        rho = self.f.sum(0)
        self.m = torch.stack([rho] + [(sum(lat.c[q][d] * self.f[q] for q in range(lat.q)) + 0.5 * F[d]) / rho
                                      if d < lat.dim else torch.zeros_like(rho) for d in range(3)])


def _pull(lat, P, n):
    """f_new from grown populations P: f_new(x, q) = P(x - c_q, q)."""
    out = torch.empty((lat.q,) + tuple(n), dtype=torch.float64, device=P.device)
    for q in range(lat.q):
        c = [int(v) for v in lat.c[q]]
        z0, y0, x0 = 1 - c[2], 1 - c[1], 1 - c[0]
        out[q] = P[q, z0:z0 + n[0], y0:y0 + n[1], x0:x0 + n[2]]
    return out


def _domain_fill(case):
    """Streaming of a level equal to its domain: periodic images, then per ghost user_2 / user_1 / ext_dir
    states on the nearest domain cell, else the nearest cell along the last foextrap direction."""
    lat, dim, n = case.lattice, case.dim, case.n_cell
    sh = tuple(case.shape)
    g = np.meshgrid(*[np.arange(-1, m + 1) for m in sh], indexing="ij")
    g = [g[2], g[1], g[0]]
    per = [case.periodic[d] or d >= dim for d in range(3)]
    out = [(g[d] < 0, g[d] >= n[d]) for d in range(3)]
    phys = sum(((out[d][0] | out[d][1]) if not per[d] else np.zeros(g[0].shape, bool)) for d in range(3)).astype(bool)
    clamp = [np.clip(g[d], 0, n[d] - 1) for d in range(3)]
    kind = np.zeros(g[0].shape, int)                     # 0 post-collision image, 1 copy, 2 ext_dir, 3 user_2, 4 bounce-back
    src = [np.where(phys, clamp[d], np.mod(g[d], n[d])) for d in range(3)]
    bval = np.zeros(g[0].shape + (4,))
    todo = phys.copy()
    for typ, code in ((cases.USER_2, 3), (cases.USER_1, 4), (cases.EXT_DIR, 2)):
        for d in range(dim):
            for side, bc, val in ((0, case.bc_lo[d], case.bc_lo_val[d]), (1, case.bc_hi[d], case.bc_hi_val[d])):
                if bc == typ and not per[d]:
                    hit = todo & out[d][side]
                    kind[hit], bval[hit] = code, val
                    todo &= ~hit
    for d in range(3):                                   # foextrap: periodic directions keep their image
        src[d] = np.where(todo, np.mod(g[d], n[d]) if per[d] else clamp[d], src[d])
    kind[todo] = 1
    dev = _dev()
    at = np.nonzero(phys)
    K = torch.tensor(kind[at], device=dev)
    S = [torch.tensor(src[d][at], device=dev) for d in (2, 1, 0)]
    BV = torch.tensor(bval[at], device=dev)
    at = tuple(torch.tensor(a, device=dev) for a in at)
    walls = [(d, side) for d in range(dim) for side, bc in ((0, case.bc_lo[d]), (1, case.bc_hi[d]))
             if bc == cases.USER_1 and not per[d]]
    opp = [lat.opposite(q) for q in range(lat.q)]

    def fill(lev, post):
        pad = torch.nn.functional.pad
        if dim == 3:
            P = pad(post[None], (1,) * 6, mode="circular")[0]
        else:
            P = pad(post[:, 0][None], (1,) * 4, mode="circular")[0][:, None].expand(-1, 3, -1, -1).clone()
        if K.numel():
            fs = lev.f[:, S[0], S[1], S[2]]
            rho = fs.sum(0)
            u = [sum(lat.c[q][d] * fs[q] for q in range(lat.q)) / rho for d in range(3)]
            rt = torch.where(K == 3, 2.0 * BV[:, 0] - rho, BV[:, 0])
            ut = [torch.where(K == 3, 2.0 * BV[:, 1 + d] - u[d], BV[:, 1 + d]) for d in range(3)]
            for q in range(lat.q):
                neq = _feq(lat, q, rt, ut) + fs[q] - _feq(lat, q, rho, u)
                P[(q,) + at] = torch.where((K == 2) | (K == 3), neq, fs[q])
        new = _pull(lat, P, post.shape[1:])
        for d, side in walls:                            # halfway bounce-back on user_1 faces
            for q in range(lat.q):
                if lat.c[q][d] != (1 if side else -1):
                    continue
                s = [slice(None)] * 3                    # not the cells whose link also leaves a periodic face
                for e in range(dim):
                    if e == d:
                        s[2 - e] = slice(n[e] - 1, n[e]) if side else slice(0, 1)
                    elif case.periodic[e] and lat.c[q][e]:
                        s[2 - e] = slice(0, n[e] - 1) if lat.c[q][e] > 0 else slice(1, n[e])
                new[(opp[q], *s)] = post[(q, *s)]
        return new

    return fill


class _Body:
    """The marker body with implicit velocity correction on a level whose cell (0, 0, 0) of the domain
    sits at ``origin`` in the level's box."""

    def __init__(self, ib, case, box_lo=(0, 0, 0)):
        self.ib, self.dim, self.h, self.lo, self.plo = ib, case.dim, case.dx, box_lo, case.prob_lo
        R, h = ib.R, case.dx
        if ib.geometry_type == 2:
            chord, th, mean, amp, freq, phase, pivot = ib.airfoil
            self.kin = (mean, amp, freq, phase)
            nh = max(math.ceil(1.5 * chord / h), 48)
            def prof(x):
                xc = np.clip(x / chord, 0.0, 1.0)
                return 5.0 * th * chord * (0.2969 * np.sqrt(xc) - 0.1260 * xc - 0.3516 * xc ** 2 + 0.2843 * xc ** 3 - 0.1036 * xc ** 4)
            up = 0.5 * chord * (1.0 - np.cos(np.pi * np.arange(nh + 1) / nh))
            dn = 0.5 * chord * (1.0 - np.cos(np.pi * np.arange(nh - 1, 0, -1) / nh))
            ref = np.stack([np.concatenate([up, dn]), np.concatenate([prof(up), -prof(dn)])])
            d = ref - np.roll(ref, -1, axis=1)
            self.dv = float(np.sqrt((d ** 2).sum(0)).sum()) / ref.shape[1] * h
            self.ref = ref - np.array([[pivot], [0.0]])
        elif self.dim == 2:
            n = max(math.ceil(2.0 * math.pi * R / h), 16)
            t = 2.0 * np.pi * np.arange(n) / n
            self.dv = 2.0 * math.pi * R * h / n
            self.x = np.stack([ib.x0 + R * np.cos(t), ib.y0 + R * np.sin(t)])
        else:
            vol = (R + 0.5 * h) ** 3 - (R - 0.5 * h) ** 3
            n = max(int(vol / (3.0 * h ** 3 / 4.0 / math.pi)), 32)
            self.dv = vol / (3.0 * n / 4.0 / math.pi)
            H = -1.0 + 2.0 * np.arange(n) / (n - 1.0)
            ph = np.zeros(n)
            for i in range(1, n - 1):
                ph[i] = math.fmod(ph[i - 1] + 3.809 / math.sqrt(n) / math.sqrt(1.0 - H[i] * H[i]), 2.0 * math.pi)
            th = np.arccos(H)
            self.x = np.stack([ib.x0 + R * np.sin(th) * np.cos(ph), ib.y0 + R * np.sin(th) * np.sin(ph), ib.z0 + R * np.cos(th)])
        self.lu = None

    def _place(self, time):
        if self.ib.geometry_type != 2:
            return self.x, np.zeros_like(self.x)
        mean, amp, freq, phase = self.kin
        p = 2.0 * math.pi * freq * time + phase
        a, om = mean + amp * math.sin(p), 2.0 * math.pi * freq * amp * math.cos(p)
        x = self.ib.x0 + math.cos(a) * self.ref[0] - math.sin(a) * self.ref[1]
        y = self.ib.y0 + math.sin(a) * self.ref[0] + math.cos(a) * self.ref[1]
        return np.stack([x, y]), np.stack([-om * (y - self.ib.y0), om * (x - self.ib.x0)])

    def force(self, lev, dt, time):
        """Sets the level's force and returns the marker force sum."""
        dim, h, dev = self.dim, self.h, _dev()
        x, ut = self._place(time)
        x, ut = torch.tensor(x, device=dev), torch.tensor(ut, device=dev)
        if self.lu is None or self.ib.geometry_type == 2:
            self.idx, self.w, A = [], [], self.dv
            for d in range(dim):
                c0 = torch.floor((x[d] - self.plo[d]) / h).long()
                ii = c0[:, None] + torch.arange(-2, 3, device=dev)
                r = (self.plo[d] + (ii.double() + 0.5) * h - x[d][:, None]).abs() / h
                s1 = torch.sqrt(torch.clamp(1.0 + 4.0 * r - 4.0 * r * r, min=0.0))
                s2 = torch.sqrt(torch.clamp(-7.0 + 12.0 * r - 4.0 * r * r, min=0.0))
                w = torch.where(r < 1.0, 0.125 * (3.0 - 2.0 * r + s1), torch.where(r < 2.0, 0.125 * (5.0 - 2.0 * r - s2), 0.0 * r)) / h
                base = int(ii.min())
                W = torch.zeros((x.shape[1], int(ii.max()) - base + 1), dtype=torch.float64, device=dev)
                W.scatter_(1, ii - base, w)
                A = A * (W @ W.T * h)
                self.idx.append(ii - self.lo[d])
                self.w.append(w)
            A = A + self.ib.ivc_diag_reg * torch.eye(x.shape[1], dtype=torch.float64, device=dev)
            self.lu = torch.linalg.lu_factor(A)
        n = x.shape[1]
        if dim == 3:
            K, J, I = self.idx[2][:, :, None, None], self.idx[1][:, None, :, None], self.idx[0][:, None, None, :]
            w = self.w[2][:, :, None, None] * self.w[1][:, None, :, None] * self.w[0][:, None, None, :]
        else:
            K, J, I = torch.zeros((1, 1, 1, 1), dtype=torch.long, device=dev), self.idx[1][:, None, :, None], self.idx[0][:, None, None, :]
            w = (self.w[1][:, :, None] * self.w[0][:, None, :])[:, None]
        K, J, I = (t.expand(w.shape) for t in (K, J, I))
        U = torch.stack([(w * lev.m[1 + d][K, J, I]).reshape(n, -1).sum(1) * h ** dim for d in range(dim)])
        Fm = torch.linalg.lu_solve(*self.lu, ((ut - U) / dt).T).T
        for d in range(dim):
            a = torch.zeros_like(lev.m[0])
            a.index_put_((K.reshape(-1), J.reshape(-1), I.reshape(-1)), (w * (Fm[d] * self.dv)[:, None, None, None]).reshape(-1), accumulate=True)
            lev.F[d] = dt * lev.m[0] * a
        s = np.zeros(3)
        s[:dim] = (Fm.sum(1) * self.dv).cpu().numpy()
        return s


class _Record:
    """The force record's arithmetic (time-centred body force, Cd / Cl)."""

    def __init__(self, ib, dim, dx):
        self.ib, self.dim, self.dx, self.prev = ib, dim, dx, None

    def take(self, lev, msum, dt):
        fe = np.zeros(3)
        for d in range(self.dim):
            fe[d] = -float(lev.F[d].sum()) * self.dx ** self.dim / dt
        ftc = fe if self.prev is None else 0.5 * (self.prev + fe)
        self.prev = fe
        r = np.zeros(18)
        U, R = self.ib.U0, self.ib.R
        den = 0.5 * U * U * (math.pi * R * R if self.dim == 3 else 2.0 * R)
        r[0:3], r[6:9], r[9:12], r[12:15], r[15:18] = ftc, fe, fe, -msum, fe
        r[3:3 + self.dim] = ftc[:self.dim] / den
        return r


def _stored(lat, f, storage):
    """Populations as the storage form holds them."""
    w = torch.tensor(lat.w, dtype=torch.float64, device=f.device).view(-1, 1, 1, 1)
    return f if storage == "f64" else (f - w) if storage == "f32" else (f - w) * (F16_SCALE / w)


def _exact_single(case, ib, init, c, steps):
    F = case.prescribed_force if ib is None and case.prescribed_force else (0.0, 0.0, 0.0)
    lev = _Level(case.lattice, case, case.tau, case.dx, init(), _domain_fill(case), F)
    body = _Body(ib, case) if ib is not None else None
    rec, recs, t = _Record(ib, case.dim, case.dx) if ib is not None else None, [], 0.0
    for _ in range(steps):
        if body is not None:
            ms = body.force(lev, case.dt, t)
            recs.append(rec.take(lev, ms, case.dt))
        lev.step()
        t += case.dt
    return lev, recs


def _exact_hierarchy(c, rng):
    hc, ib, inits = _hierarchy(c, rng)
    if hasattr(hc, "fine_lo"):
        hc = cases.HierarchyCase(hc.coarse, ((hc.fine_lo, hc.fine_hi),))
    lat, dim, nlev = hc.coarse.lattice, hc.dim, hc.nlev
    levs = []

    def cf_fill(l, mac):
        """Grown populations of level l: equilibrium of the level above's macro fields, limited-linear."""
        lo, hi = hc.box_lohi(l)
        clo, _ = hc.box_lohi(l - 1)
        ix = []
        for d in (2, 1, 0):
            ix.append(torch.arange(lo[d] - 1, hi[d] + 2, device=_dev()) if d < dim else torch.zeros(1, dtype=torch.long, device=_dev()))
        ci = [torch.div(i, 2, rounding_mode="floor") - clo[d] if d < dim else i for i, d in zip(ix, (2, 1, 0))]
        take = lambda t, z, y, x: t[:, z][:, :, y][:, :, :, x]
        cc = take(mac, *ci)
        v = cc.clone()
        for a, d in ((0, 2), (1, 1), (2, 0)):
            if d >= dim:
                continue
            up, dn = list(ci), list(ci)
            up[a], dn[a] = ci[a] + 1, ci[a] - 1
            r, l_ = take(mac, *up) - cc, cc - take(mac, *dn)
            cen = 0.5 * (r + l_)
            s = torch.minimum(cen.abs(), 2.0 * torch.minimum(r.abs(), l_.abs())) * torch.sign(cen)
            s = torch.where(r * l_ <= 0.0, torch.zeros_like(s), s)
            off = torch.where(ix[a] % 2 == 0, -0.25, 0.25).double()
            v += s * off.view([-1 if k == a else 1 for k in range(3)])[None]
        P = torch.stack([_feq(lat, q, v[0], v[1:]) for q in range(lat.q)])
        return P if dim == 3 else P.expand(-1, 3, -1, -1).clone()

    def fine_step_fill(lev, post):
        P = lev.ghost.clone()
        n = post.shape[1:]
        if dim == 3:
            P[:, 1:-1, 1:-1, 1:-1] = post
        else:
            P[:, :, 1:-1, 1:-1] = post
        return _pull(lat, P, n)

    for l in range(nlev):
        k = hc.level_case(l)
        levs.append(_Level(lat, hc.box_case(l), k.tau, k.dx, inits[l](), _domain_fill(hc.coarse) if l == 0 else fine_step_fill))
    top = nlev - 1
    lo, _ = hc.box_lohi(top)
    kt = hc.level_case(top)
    body, rec = _Body(ib, kt, lo), _Record(ib, dim, kt.dx)
    msum = [None]

    def average(l):
        clo, _ = hc.box_lohi(l)
        flo, fhi = hc.box_lohi(l + 1)
        s = [slice(flo[d] // 2 - clo[d], fhi[d] // 2 + 1 - clo[d]) if d < dim else slice(None) for d in (2, 1, 0)]
        for t, u in ((levs[l].f, levs[l + 1].f), (levs[l].m, levs[l + 1].m)):
            a = u[:, :, ::2, ::2] + u[:, :, 1::2, ::2] + u[:, :, ::2, 1::2] + u[:, :, 1::2, 1::2]
            t[:, s[0], s[1], s[2]] = (a[:, ::2] + a[:, 1::2]) * 0.125 if dim == 3 else a * 0.25

    def advance(l, t, dt):
        L = levs[l]
        old = L.m
        if l == top:
            msum[0] = body.force(L, dt, t)
        L.step()
        if l < top:
            for sub in range(2):
                levs[l + 1].ghost = cf_fill(l + 1, old if sub == 0 else 0.5 * (old + L.m))
                advance(l + 1, t + 0.5 * sub * dt, 0.5 * dt)
            average(l)

    for l in range(top - 1, -1, -1):
        average(l)
    t, r = 0.0, None
    every = c["q"] == 19
    for s in range(1 + c["steps"]):
        advance(0, t, hc.coarse.dt)
        t += hc.coarse.dt
        if (every and s > 0) or s == c["steps"]:
            r = rec.take(levs[top], msum[0], kt.dt)
    return dict(f=[_stored(lat, x.f, c["storage"]) for x in levs], force=torch.stack(levs[top].F[:dim]), rec=r)


def exact(case, seed):
    c = dict(case)
    rng = np.random.default_rng(seed)
    if c["kind"] == "boxes":
        f, m = _boxes_input(c, seed, _dev())
        lat = LATTICE[c["q"]]
        level = cases.LevelCase(lat, (c["nx"], c["ny"], c["nz"]), nu=0.05)
        lev = _Level(lat, level, level.tau, level.dx, [t.cpu().numpy() for t in m], _domain_fill(level))
        lev.f = f
        lev.step()
        return [tuple(t[:, lo[2]:hi[2] + 1, lo[1]:hi[1] + 1, lo[0]:hi[0] + 1] for t in (lev.f, lev.m)) for lo, hi in _box_cuts(c)]
    if c["kind"] == "hierarchy":
        return _exact_hierarchy(c, rng)
    if c["kind"] == "batch":
        return [_stored(D2Q9, _exact_single(k, ib, init, c, 1 + c["steps"])[0].f, c["storage"]) for k, ib, init in _batch(c, rng)]
    k, ib, init = _single(c, rng)
    lev, recs = _exact_single(k, ib, init, c, 1 + c["steps"])
    f = _stored(k.lattice, lev.f, c["storage"])
    if ib is None:
        return f
    return dict(f=f, force=torch.stack(lev.F[:k.dim]), rec=np.array(recs[1:]))
