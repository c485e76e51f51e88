"""Workloads of the PB multigrid library: what its users have it do.

Four kinds of call, each through the library's public boundary (the C ABI of
include/pmg_b200.h by multigrid_b200._lib, the pmgc kernels by
multigrid_b200.pmgc, the serving runtime by multigrid_b200.serve):

  solve    one PB solve on a problem handle that the program keeps: load the
           finest level (six device arrays, or the atoms with the GPU
           set-up), build the hierarchy, V-cycles / refinement steps or the
           MG-preconditioned CG to relative residual 1e-10, the potential
           into a device array;
  batch    several molecules of uneven sizes through a resident server;
  driver   the APBS iparm/rparm driver on coefficient maps;
  cycle    a V(2,2) cycle written with the pmgc kernels on the caller's own
           hierarchy (double with the coarsest CG, or float);
  build    two coarsenings with the pmgc builders (prolongation, Galerkin).

The molecules are synthetic (atoms uniform in a ball, radii U[1.2, 2.0] A,
charges N(0, 0.4) e) with the library's default physics: dielectric 2 inside
and 78.54 outside with a 1.4 A probe, 0.15 M salt, ion radius 2 A, 298.15 K.
Inputs and expected results are computed here with torch in 64 bits.
"""
import ctypes
import itertools
import math

import numpy as np
import torch

from multigrid_b200 import _lib, pmgc
from multigrid_b200.molecule import DEFAULT_PHYSICS, levels_for
from multigrid_b200.problem import PRECISIONS, physics_struct
from multigrid_b200.serve import Server

TOL = 1e-10       # relative residual of the solves
DRIVER_TOL = 1e-9  # relative L1 residual of the APBS driver
DEV = "cuda"

# grids whose coarsest level has at most 15 points per axis by the library's
# size rule
SOLVE_SIZES = (33, 41, 49, 57, 65, 81, 97, 113, 129, 161, 193)


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # a small molecule, the latency of one solve (65^3, 400 atoms)
        dict(name="solve-mixed-65", kind="solve", n=65, h=0.5, natoms=400,
             ball=12.0, precision="mixed", method="cycles", source="arrays"),
        # the headline: 257^3, 5000 atoms, mixed precision
        dict(name="solve-mixed-257", kind="solve", n=257, h=0.4, natoms=5000,
             ball=30.0, precision="mixed", method="cycles", source="arrays"),
        # the reference's all-double cycle on its own hierarchy, 161^3
        dict(name="solve-fp64-161", kind="solve", n=161, h=0.4, natoms=5000,
             ball=30.0, precision="fp64", method="cycles", source="arrays"),
        # double V-cycles inside the refinement loop, 129^3
        dict(name="solve-fp64fast-129", kind="solve", n=129, h=0.5,
             natoms=3000, ball=25.0, precision="fp64-fast", method="cycles",
             source="arrays"),
        # the MG-preconditioned CG as outer solver, 193^3
        dict(name="pcg-mixed-193", kind="solve", n=193, h=0.4, natoms=5000,
             ball=30.0, precision="mixed", method="pcg", source="arrays"),
        # from the atoms: GPU set-up, build and solve, 129^3
        dict(name="atoms-mixed-129", kind="solve", n=129, h=0.5, natoms=3000,
             ball=25.0, precision="mixed", method="cycles", source="atoms"),
        # a screening batch: eight molecules of 65^3 to 129^3 on one server
        dict(name="batch-mixed-8", kind="batch", count=8, smallest=65,
             largest=129, h=0.5, precision="mixed"),
        # the APBS driver, 65^3, 4 levels, CG on the coarsest (9^3)
        dict(name="driver-cg-65", kind="driver", nx=65, ny=65, nz=65, nlev=4,
             h=0.5, natoms=400, ball=12.0, solver="cg"),
        # an oblong focusing box, banded solve on the coarsest (6 x 5 x 7)
        dict(name="driver-band-81", kind="driver", nx=81, ny=65, nz=97,
             nlev=5, h=0.5, natoms=400, ball=12.0, solver="band"),
        # a host code's own V-cycle on a large oblong grid, double
        dict(name="cycle-double-257", kind="cycle", nx=257, ny=225, nz=241,
             nlev=5, h=0.4, natoms=4000, ball=28.0, dtype="double"),
        # the same in float on a small grid: launches count
        dict(name="cycle-float-49", kind="cycle", nx=33, ny=41, nz=49,
             nlev=3, h=0.5, natoms=60, ball=5.0, dtype="float"),
        # operators of a hierarchy built by the caller, two coarsenings
        dict(name="build-129", kind="build", nx=129, ny=113, nz=97, h=0.5,
             natoms=1500, ball=18.0),
    ]


def _log_choice(rng, seq):
    """A member of a sorted sequence, uniform over the logarithm."""
    v = math.exp(rng.uniform(math.log(seq[0]), math.log(seq[-1])))
    return min(seq, key=lambda s: abs(math.log(s / v)))


def _molecule_of(rng, n, h):
    """(atoms, ball radius) that an n-point axis of spacing h has room for."""
    ball = max(4.0, ((n - 1) * h - 10.0) / 2 - 2.0)
    ball = round(min(ball, 30.0) * rng.uniform(0.7, 1.0), 2)
    return max(10, int(5000 * (ball / 30.0) ** 3 * rng.uniform(0.7, 1.0))), ball


def draw(rng):
    kind = rng.choice(("solve", "solve", "solve", "batch", "driver", "cycle",
                       "cycle", "build"))
    h = round(rng.uniform(0.4, 0.55), 3)
    if kind == "solve":
        precision = rng.choice(("mixed", "mixed", "fp64", "fp64-fast"))
        method = rng.choice(("cycles", "cycles", "pcg"))
        sizes = [s for s in SOLVE_SIZES if precision == "mixed" or s <= 161]
        n = _log_choice(rng, sizes)
        natoms, ball = _molecule_of(rng, n, h)
        return dict(kind=kind, n=n, h=h, natoms=natoms, ball=ball,
                    precision=precision, method=method,
                    source=rng.choice(("arrays", "arrays", "atoms")))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(2, 8), smallest=65,
                    largest=rng.choice((97, 129)), h=h,
                    precision=rng.choice(("mixed", "mixed", "fp64-fast")))
    if kind == "driver":
        # multiples of 16 plus one, three or four levels of exact coarsening
        dims = [16 * rng.randint(2, 6) + 1 for _ in range(3)]
        solver = rng.choice(("cg", "band"))
        natoms, ball = _molecule_of(rng, min(dims), h)
        return dict(kind=kind, nx=dims[0], ny=dims[1], nz=dims[2],
                    nlev=5 if solver == "band" else rng.choice((4, 5)), h=h,
                    natoms=natoms, ball=ball, solver=solver)
    if kind == "cycle":
        big = rng.random() < 0.5
        unit, most, nlev = (16, 12, 5) if big else (8, 10, 4)
        dims = [unit * rng.randint(4, most) + 1 for _ in range(3)]
        natoms, ball = _molecule_of(rng, min(dims), h)
        return dict(kind=kind, nx=dims[0], ny=dims[1], nz=dims[2], nlev=nlev,
                    h=h, natoms=natoms, ball=ball,
                    dtype=rng.choice(("double", "float")))
    dims = [4 * rng.randint(8, 36) + 1 for _ in range(3)]
    natoms, ball = _molecule_of(rng, min(dims), h)
    return dict(kind=kind, nx=dims[0], ny=dims[1], nz=dims[2], h=h,
                natoms=natoms, ball=ball)


# ---------------------------------------------------------------------------
# the fine level from atoms, with torch
# ---------------------------------------------------------------------------
def make_atoms(seed, natoms, ball, center):
    """natoms x 5 (x, y, z, radius, charge), uniform in a ball; integer net
    charge."""
    rng = np.random.default_rng(seed)
    p = rng.normal(size=(natoms, 3))
    p *= (ball * rng.uniform(size=(natoms, 1)) ** (1 / 3) /
          np.linalg.norm(p, axis=1, keepdims=True))
    q = rng.normal(0.0, 0.4, size=natoms)
    q += (np.round(q.sum()) - q.sum()) / natoms
    return np.ascontiguousarray(np.column_stack(
        [p + np.asarray(center), rng.uniform(1.2, 2.0, size=natoms), q]))


def case_atoms(case, seed):
    dims = grid_dims(case)
    center = [case["h"] * (dims[2 - a] - 1) / 2 for a in range(3)]
    return make_atoms(seed, case["natoms"], case["ball"], center)


def grid_dims(case):
    """(nx, ny, nz)"""
    if "n" in case:
        return case["n"], case["n"], case["n"]
    return case["nx"], case["ny"], case["nz"]


def _constants():
    """(kappa [1/A], eps0 in e^2 / (kT A)) of the default physics."""
    kb, e, eps, na = 1.380649e-23, 1.60217663e-19, 8.8541878128e-12, 6.0221408e23
    t = DEFAULT_PHYSICS["temperature"]
    inv_sq = (e * e / (kb * t) * 2 * 1000 * DEFAULT_PHYSICS["ionic_strength"]
              * na / (DEFAULT_PHYSICS["eps_out"] * eps))
    return math.sqrt(inv_sq) * 1e-10, eps * 1e-10 / (e * e) * kb * t


def _mark(mask, h, centers, radii):
    """mask (n0, n1, n2) set on the grid points within radii of centers."""
    if not len(centers):
        return
    w = int(2 * float(radii.max()) / h) + 2
    step = max(1, 12_000_000 // w ** 3)
    ar = torch.arange(w, device=mask.device)
    for c, r in zip(centers.split(step), radii.split(step)):
        ix, d2, ok = [], [], []
        for a in range(3):
            i = torch.ceil((c[:, a] - r) / h).long()[:, None] + ar
            ix.append(i)
            d2.append((i * h - c[:, a:a + 1]) ** 2)
            ok.append((i >= 0) & (i < mask.shape[a]))
        far = (d2[0][:, :, None, None] + d2[1][:, None, :, None] +
               d2[2][:, None, None, :])
        hit = ((far <= (r * r)[:, None, None, None]) & ok[0][:, :, None, None]
               & ok[1][:, None, :, None] & ok[2][:, None, None, :])
        at = ((ix[0][:, :, None, None] * mask.shape[1] +
               ix[1][:, None, :, None]) * mask.shape[2] +
              ix[2][:, None, None, :])
        mask.view(-1)[at[hit]] = True


def _probe_centers(at, probe):
    """Centres of the probe spheres: 96 points of a Fibonacci lattice on
    every inflated atom sphere that no other inflated sphere contains."""
    s = torch.arange(96, device=at.device, dtype=torch.float64)
    zz = 1 - 2 * (s + 0.5) / 96
    rr = (1 - zz * zz).clamp_min(0).sqrt()
    ang = math.pi * (3.0 - math.sqrt(5.0)) * s
    u = torch.stack([rr * torch.cos(ang), rr * torch.sin(ang), zz], 1)
    big = at[:, 3] + probe
    pc = at[:, None, :3] + big[:, None, None] * u[None]
    free = torch.empty(len(at), 96, dtype=torch.bool, device=at.device)
    step = max(1, 30_000_000 // (96 * len(at)))
    lim = big * big * (1 - 1e-12)
    every = torch.arange(len(at), device=at.device)
    for q in range(0, len(at), step):
        p = pc[q:q + step]
        d2 = sum((p[:, :, None, a] - at[None, None, :, a]) ** 2
                 for a in range(3))
        own = every[q:q + step, None, None] == every[None, None, :]
        free[q:q + step] = ~((d2 < lim) & ~own).any(2)
    return pc[free]


def _two_valued(mask, yes, no):
    out = torch.full(mask.shape, no, dtype=torch.float64, device=mask.device)
    return out.masked_fill_(mask, yes)


def fine_level(dims, h, atoms):
    """The class's finest level: dict of (nz, ny, nx) doubles on the GPU.
    oE oN uC: eps / h^2 at the points half a step along x, y, z; kap:
    kappa^2 eps_out outside the ion spheres; oC the six faces plus kap on the
    interior; f trilinear charges; x0 Debye-Hueckel values on the shell.
    Atom coordinate 0 runs along the slowest axis (z)."""
    nx, ny, nz = dims
    shape = (nz, ny, nx)
    at = torch.from_numpy(atoms).to(DEV)
    kappa, eps0 = _constants()
    ph = DEFAULT_PHYSICS
    probes = _probe_centers(at, ph["probe_radius"])
    face = []
    for axis in range(3):  # 0 -> uC, 1 -> oN, 2 -> oE
        off = torch.zeros(3, dtype=torch.float64, device=DEV)
        off[axis] = 0.5 * h
        inside = torch.zeros(shape, dtype=torch.bool, device=DEV)
        sas, carved = torch.zeros_like(inside), torch.zeros_like(inside)
        _mark(inside, h, at[:, :3] - off, at[:, 3])
        _mark(sas, h, at[:, :3] - off, at[:, 3] + ph["probe_radius"])
        _mark(carved, h, probes - off, torch.full(
            (len(probes),), ph["probe_radius"], dtype=torch.float64,
            device=DEV))
        face.append(_two_valued(inside | (sas & ~carved),
                                ph["eps_in"] / (h * h),
                                ph["eps_out"] / (h * h)))
    uC, oN, oE = face
    ion = torch.zeros(shape, dtype=torch.bool, device=DEV)
    _mark(ion, h, at[:, :3], at[:, 3] + ph["ion_radius"])
    kap = _two_valued(ion, 0.0, kappa * kappa * ph["eps_out"])
    oC = torch.zeros(shape, dtype=torch.float64, device=DEV)
    c = (slice(1, -1),) * 3
    oC[c] = ((uC[c] + uC[:-2, 1:-1, 1:-1]) + (oN[c] + oN[1:-1, :-2, 1:-1]) +
             (oE[c] + oE[1:-1, 1:-1, :-2]) + kap[c])
    # charges: the eight corners of every atom's cell
    f = np.zeros(shape)
    s = atoms[:, :3] / h
    lo = np.floor(s).astype(np.int64)
    for corner in itertools.product((0, 1), repeat=3):
        b = np.asarray(corner)
        wt = np.prod(np.where(b, s - lo, lo + 1 - s), axis=1)
        np.add.at(f, tuple((lo + b).T), atoms[:, 4] / eps0 * wt / h ** 3)
    f = torch.from_numpy(f).to(DEV)
    # boundary: sum over atoms on the shell
    x0 = torch.zeros(shape, dtype=torch.float64, device=DEV)
    shell = torch.ones(shape, dtype=torch.bool, device=DEV)
    shell[c] = False
    pts = shell.nonzero()
    val = torch.zeros(len(pts), dtype=torch.float64, device=DEV)
    pref = 4 * math.pi * eps0 * ph["eps_out"]
    for q in range(0, len(at), 48):
        a = at[q:q + 48]
        d = sum((pts[:, None, e] * h - a[None, :, e]) ** 2
                for e in range(3)).sqrt()
        val += (a[:, 4] / (pref * (1 + kappa * a[:, 3])) *
                torch.exp(-kappa * (d - a[:, 3])) / d).sum(1)
    x0[shell] = val
    return dict(oC=oC, oE=oE, oN=oN, uC=uC, f=f, x0=x0, kap=kap)


# ---------------------------------------------------------------------------
# the pmgc operations with torch, 64 bits: operators as lists of (nz, ny, nx)
# arrays, 4 (7-point) or 14 diagonals; couplings are positive
# ---------------------------------------------------------------------------
# upper neighbour of diagonal s = 1..13: oE oN uC oNE oNW uE uW uN uS uNE uNW
# uSE uSW, as (dx, dy, dz)
UPPER = ((0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (-1, 1, 0),
         (1, 0, 1), (-1, 0, 1), (0, 1, 1), (0, -1, 1), (1, 1, 1), (-1, 1, 1),
         (1, -1, 1), (-1, -1, 1))
ALL27 = tuple((x, y, z) for z in (-1, 0, 1) for y in (-1, 0, 1)
              for x in (-1, 0, 1))
PLANE = ((0, 0), (0, 1), (0, -1), (1, 0), (-1, 0), (1, 1), (-1, 1), (1, -1),
         (-1, -1))


def pslot(d):
    """Row of the prolongation weight of fine offset d in the list of 27."""
    return (0, 9, 18)[(0, 1, -1).index(d[2])] + PLANE.index((d[0], d[1]))


def _add(a, b):
    return tuple(x + y for x, y in zip(a, b))


def _neg(a):
    return tuple(-x for x in a)


class Points:
    """A strided set of points of a grid: view(a, d) is array a at the
    points moved by d = (dx, dy, dz)."""

    def __init__(self, start, step, count):  # (x, y, z) each
        self.start, self.step, self.count = start, step, count

    def view(self, a, d=(0, 0, 0)):
        sl = []
        for q in (2, 1, 0):
            s = self.start[q] + d[q]
            sl.append(slice(s, s + (self.count[q] - 1) * self.step + 1,
                            self.step))
        return a[tuple(sl)]


def interior(shape):
    return Points((1, 1, 1), 1, tuple(s - 2 for s in reversed(shape)))


def couplings(op):
    """[(offset e, diagonal, offset where its value is read)] of a stencil."""
    out = []
    for s in range(1, len(op)):
        e = UPPER[s]
        out += [(e, s, (0, 0, 0)), (_neg(e), s, _neg(e))]
    return out


def neighbour_sum(op, x, pts):
    out = 0
    for e, s, w in couplings(op):
        out = out + pts.view(op[s], w) * pts.view(x, e)
    return out


def residual64(op, f, x):
    r = torch.zeros_like(x)
    p = interior(x.shape)
    p.view(r).copy_(p.view(f) + neighbour_sum(op, x, p) -
                    p.view(op[0]) * p.view(x))
    return r


def smooth64(op, f, x, sweeps, adjoint):
    """Red-black (7-point) or eight-colour (27-point) Gauss-Seidel; colours
    of 1-based indices."""
    n = tuple(reversed(x.shape))
    if len(op) == 4:
        k, j, i = torch.meshgrid(*[torch.arange(s, device=x.device)
                                   for s in x.shape], indexing="ij")
        par = interior(x.shape).view((i + j + k + 3) % 2)
        for c in list((1, 0) if adjoint else (0, 1)) * sweeps:
            p = interior(x.shape)
            new = (p.view(f) + neighbour_sum(op, x, p)) / p.view(op[0])
            p.view(x).copy_(torch.where(par == c, new, p.view(x)))
        return
    for c in list(range(7, -1, -1) if adjoint else range(8)) * sweeps:
        bits = (c & 1, c >> 1 & 1, c >> 2 & 1)
        # the 0-based interior index i has 1-based parity (i + 1) % 2
        start = tuple(1 if (1 + 1) % 2 == b else 2 for b in bits)
        count = tuple((n[a] - 2 - start[a]) // 2 + 1 for a in range(3))
        if min(count) < 1:
            continue
        p = Points(start, 2, count)
        p.view(x).copy_((p.view(f) + neighbour_sum(op, x, p)) / p.view(op[0]))


def fine_points(coarse_shape):
    """The fine images of the coarse interior points."""
    return Points((2, 2, 2), 2, tuple(s - 2 for s in reversed(coarse_shape)))


def restrict64(r, P):
    out = torch.zeros_like(P[0])
    pf, pc = fine_points(out.shape), interior(out.shape)
    pc.view(out).copy_(sum(pc.view(P[pslot(d)]) * pf.view(r, d)
                           for d in ALL27))
    return out


def interpolate64(xc, P, fine_shape):
    """Every fine point but the last of each axis; coarse points inject."""
    out = torch.zeros(fine_shape, dtype=xc.dtype, device=xc.device)
    cells = tuple(s - 1 for s in reversed(xc.shape))
    for o in itertools.product((0, 1), repeat=3):
        to = Points(o, 2, cells)
        if o == (0, 0, 0):
            to.view(out).copy_(Points((0, 0, 0), 1, cells).view(xc))
            continue
        acc = 0
        for c in itertools.product(*[(0, 1) if v else (0,) for v in o]):
            d = tuple(v - 2 * b for v, b in zip(o, c))
            frm = Points(c, 1, cells)
            acc = acc + frm.view(P[pslot(d)]) * frm.view(xc)
        to.view(out).copy_(acc)
    return out


def prolongation64(op, coarse_shape):
    """Operator-based weights (27, nz, ny, nx): faces, then edges, then
    corners; couplings along the axes not interpolated across are lumped
    onto the diagonal. uPE of the 27-point form reads the coupling of f to
    (0, 1, -1) where the rule has (-1, 0, -1), as the reference does."""
    P = torch.zeros((27,) + tuple(coarse_shape), dtype=op[0].dtype,
                    device=op[0].device)
    pf, pc = fine_points(coarse_shape), interior(coarse_shape)
    at = {e: (s, w) for e, s, w in couplings(op)}
    w = {(0, 0, 0): torch.ones_like(pc.view(P[0]))}
    for d in sorted(ALL27, key=lambda v: sum(map(abs, v))):
        if d == (0, 0, 0):
            continue
        num, lump = 0, 0
        for e in ALL27:
            if e == (0, 0, 0) or e not in at:
                continue
            if not any(e[a] for a in range(3) if d[a]):
                s, o = at[e]
                lump = lump + pf.view(op[s], _add(d, o))
            elif all(e[a] in (0, -d[a]) for a in range(3) if d[a]):
                read = e
                if len(op) == 14 and d == (1, 0, 1) and e == (-1, 0, -1):
                    read = (0, 1, -1)
                s, o = at[read]
                v = tuple(d[a] + e[a] if d[a] else 0 for a in range(3))
                num = num + pf.view(op[s], _add(d, o)) * w[v]
        w[d] = num / (pf.view(op[0], d) - lump)
    for d in ALL27:
        pc.view(P[pslot(d)]).copy_(w[d])
    return P


def galerkin64(op, P):
    """A_c(C, C+D) = sum_{d, e} P_d(C) A_f(c+d, c+d+e) P_{d+e-2D}(C+D)."""
    shape = P.shape[1:]
    out = torch.zeros((14,) + tuple(shape), dtype=P.dtype, device=P.device)
    pf, pc = fine_points(shape), interior(shape)
    cs = [((0, 0, 0), 0, (0, 0, 0))] + couplings(op)
    for s, D in enumerate(UPPER):
        acc = torch.zeros_like(pc.view(P[0]))
        for d in ALL27:
            inner = 0
            for e, q, o in cs:
                t = tuple(d[a] + e[a] - 2 * D[a] for a in range(3))
                if max(map(abs, t)) > 1:
                    continue
                term = pf.view(op[q], _add(d, o)) * pc.view(P[pslot(t)], D)
                inner = inner + (term if q == 0 else -term)
            if not isinstance(inner, int):
                acc += pc.view(P[pslot(d)]) * inner
        pc.view(out[s]).copy_(acc if s == 0 else -acc)
    return out


def solve64(op, f, x, rtol, atol=0.0):
    """Conjugate gradients with the diagonal as preconditioner on the
    interior, from x (its shell holds the boundary values)."""
    x = x.clone()
    p = interior(x.shape)
    dinv = 1.0 / p.view(op[0])
    r = p.view(residual64(op, f, x)).clone()
    z = dinv * r
    v = torch.zeros_like(x)
    p.view(v).copy_(z)
    rz = (r * z).sum()
    stop = max(rtol * float(r.norm()), atol)
    for it in range(20000):
        if it % 20 == 0 and float(r.norm()) <= stop:
            break
        pv = p.view(v)
        ap = p.view(op[0]) * pv - neighbour_sum(op, v, p)
        alpha = rz / (pv * ap).sum()
        p.view(x).add_(alpha * pv)
        r -= alpha * ap
        z = dinv * r
        new = (r * z).sum()
        pv.mul_(new / rz).add_(z)
        rz = new
    return x


def hierarchy64(fine, nlev):
    """[operator per level], [P to level L from L + 1], finest first."""
    ops = [[fine[k] for k in ("oC", "oE", "oN", "uC")]]
    Ps = []
    for _ in range(nlev - 1):
        shape = tuple((s - 1) // 2 + 1 for s in ops[-1][0].shape)
        Ps.append(prolongation64(ops[-1], shape))
        ops.append(list(galerkin64(ops[-1], Ps[-1])))
    return ops, Ps


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


class Handle:
    """A problem handle of the C ABI."""

    def __init__(self, n, h, precision):
        self.n = n
        # the class's levels for its own cycle, the deepest otherwise
        base, nlev = (levels_for(n, 5, 9) if precision == "fp64"
                      else levels_for(n, 12, 5))
        self.h = ctypes.c_void_p()
        _lib.check("pmg_problem_create", _lib.lib.pmg_problem_create(
            base, nlev, h * (n - 1), PRECISIONS[precision], None,
            ctypes.byref(self.h)))

    def __del__(self):
        if self.h and _lib is not None:  # None while the interpreter exits
            _lib.lib.pmg_problem_destroy(self.h)


def _level_arrays(case, seed):
    return fine_level(grid_dims(case), case["h"], case_atoms(case, seed))


def _batch(case, seed):
    """Grid sizes spread over the range by index, molecules by seed."""
    sizes = [s for s in (65, 97, 129)
             if case["smallest"] <= s <= case["largest"]]
    out = []
    for q in range(case["count"]):
        n = sizes[(5 * q) % len(sizes)]
        ball = ((n - 1) * case["h"] - 10.0) / 2 - 2.0
        natoms = max(10, int(5000 * (ball / 30.0) ** 3))
        c = case["h"] * (n - 1) / 2
        out.append((n, make_atoms(1000 * seed + q, natoms, ball, (c, c, c))))
    return out


def _torch_dtype(case):
    return torch.float64 if case["dtype"] == "double" else torch.float32


def _cycle_inputs(case, seed):
    """The caller's hierarchy, right-hand side and start, in its type."""
    fine = _level_arrays(case, seed)
    ops, Ps = hierarchy64(fine, case["nlev"])
    t = _torch_dtype(case)
    return ([[a.to(t).contiguous() for a in op] for op in ops],
            [P.to(t) for P in Ps], fine["f"].to(t), fine["x0"].to(t))


def prepare(case, seed):
    kind = case["kind"]
    state = dict(case=case)
    if kind == "solve":
        n = case["n"]
        state["problem"] = Handle(n, case["h"], case["precision"])
        state["out"] = torch.empty((n, n, n), dtype=torch.float64, device=DEV)
        if case["source"] == "atoms":
            state["atoms"] = case_atoms(case, seed)
            state["physics"] = physics_struct(DEFAULT_PHYSICS)
        else:
            fine = _level_arrays(case, seed)
            state["fine"] = [fine[k] for k in ("oC", "oE", "oN", "uC", "f",
                                               "x0")]
    elif kind == "batch":
        state["server"] = Server(40 << 30, max_inflight=case["count"])
        state["work"] = []
        for n, atoms in _batch(case, seed):
            base, nlev = levels_for(n)
            state["work"].append((base, nlev, case["h"] * (n - 1), atoms,
                                  torch.empty((n, n, n), dtype=torch.float64,
                                              device=DEV)))
    elif kind == "driver":
        nx, ny, nz = grid_dims(case)
        f = _level_arrays(case, seed)
        h2 = case["h"] ** 2
        line = [torch.arange(m, dtype=torch.float64, device=DEV) * case["h"]
                for m in (nx, ny, nz)]
        x0 = f["x0"]
        state["maps"] = line + [
            torch.stack([x0[:, :, 0], x0[:, :, -1]]).contiguous(),
            torch.stack([x0[:, 0, :], x0[:, -1, :]]).contiguous(),
            torch.stack([x0[0], x0[-1]]).contiguous(),
            f["oE"] * h2, f["oN"] * h2, f["uC"] * h2, f["kap"], f["f"]]
        iparm, rparm = [0] * 25, [0.0] * 12
        iparm[2:6] = [nx, ny, nz, case["nlev"]]
        iparm[6] = iparm[7] = 2                  # nu1, nu2
        iparm[9], iparm[10] = 100, 1             # itmax, istop
        iparm[16], iparm[17] = 1, 2              # operator-based, Galerkin
        iparm[19] = 1                            # red-black Gauss-Seidel
        iparm[20] = 1 if case["solver"] == "band" else 0
        rparm[0] = DRIVER_TOL
        state["iparm"], state["rparm"] = iparm, rparm
        state["u"] = torch.zeros((nz, ny, nx), dtype=torch.float64,
                                 device=DEV)
    elif kind == "cycle":
        ops, Ps, f, x0 = _cycle_inputs(case, seed)
        state.update(ops=ops, Ps=Ps, x0=x0)
        state["f"] = [f] + [torch.zeros_like(P[0]) for P in Ps]
        state["x"] = [torch.zeros_like(a) for a in state["f"]]
        state["r"] = [torch.zeros_like(a) for a in state["f"]]
        state["e"] = [torch.zeros_like(a) for a in state["f"]]
    else:
        fine = _level_arrays(case, seed)
        state["op"] = [fine[k] for k in ("oC", "oE", "oN", "uC")]
        c1 = tuple((s - 1) // 2 + 1 for s in fine["oC"].shape)
        c2 = tuple((s - 1) // 2 + 1 for s in c1)
        z = dict(dtype=torch.float64, device=DEV)
        state["P1"], state["A1"] = (torch.zeros((27,) + c1, **z),
                                    torch.zeros((14,) + c1, **z))
        state["P2"], state["A2"] = (torch.zeros((27,) + c2, **z),
                                    torch.zeros((14,) + c2, **z))
    torch.cuda.synchronize()
    return state


def _dims(a):
    return a.shape[-1], a.shape[-2], a.shape[-3]


def run(state):
    return {"solve": _run_solve, "batch": _run_batch, "driver": _run_driver,
            "cycle": _run_cycle, "build": _run_build}[
                state["case"]["kind"]](state)


def _run_solve(s):
    lib, p = _lib.lib, s["problem"]
    if "atoms" in s:
        _lib.check("pmg_problem_set_atoms", lib.pmg_problem_set_atoms(
            p.h, s["atoms"].ctypes.data_as(_lib.PD), len(s["atoms"]),
            ctypes.byref(s["physics"])))
    else:
        _lib.check("pmg_problem_set_fine", lib.pmg_problem_set_fine(
            p.h, *[_ptr(a) for a in s["fine"]]))
    _lib.check("pmg_build_hierarchy", lib.pmg_build_hierarchy(p.h, 0))
    count, rel = ctypes.c_int(), ctypes.c_double()
    solve = (lib.pmg_pcg_solve if s["case"]["method"] == "pcg"
             else lib.pmg_solve)
    _lib.check("pmg_solve", solve(p.h, TOL, 100, ctypes.byref(count),
                                  ctypes.byref(rel), None))
    _lib.check("pmg_get_potential", lib.pmg_get_potential(p.h,
                                                          _ptr(s["out"])))
    return s["out"]


def _run_batch(s):
    for base, nlev, box, atoms, out in s["work"]:
        s["server"].submit(base, nlev, box, None,
                           precision=s["case"]["precision"], out=out, tol=TOL,
                           atoms=atoms, physics=DEFAULT_PHYSICS)
    for c in s["server"].drain(len(s["work"])):
        if not c.ok:
            raise RuntimeError(c.message)
    return [w[4] for w in s["work"]]


def _run_driver(s):
    pmgc.Vmgdriv(s["iparm"], s["rparm"], s["u"], *s["maps"])
    return s["u"]


def _smooth(op, f, x, sweeps, adjoint=0, zero=False):
    if len(op) == 4:
        pmgc.Vgsrb7x(*_dims(x), op[0], None, f, *op[1:], x, sweeps, adjoint,
                     zero)
    else:
        pmgc.Vgsrb27x(*_dims(x), op, None, f, x, sweeps, zero, adjoint)


def _run_cycle(s):
    ops, Ps, f, x, r, e = (s[k] for k in ("ops", "Ps", "f", "x", "r", "e"))
    x[0].copy_(s["x0"])
    last = len(ops) - 1
    for L in range(last):
        _smooth(ops[L], f[L], x[L], 2, zero=L > 0)
        if L == 0:
            pmgc.Vmresid7_1s(*_dims(x[0]), ops[0][0], None, f[0], *ops[0][1:],
                             x[0], r[0])
        else:
            pmgc.Vmresid27_1s(*_dims(x[L]), ops[L], None, f[L], x[L], r[L])
        pmgc.Vrestrc2(*_dims(r[L]), *_dims(f[L + 1]), r[L], f[L + 1], Ps[L])
    if s["case"]["dtype"] == "double":
        x[last].zero_()
        pmgc.cg_level(*_dims(x[last]), ops[last], f[last], x[last])
    else:  # the float cycle ends in sweeps
        _smooth(ops[last], f[last], x[last], 8, zero=True)
    for L in range(last - 1, -1, -1):
        pmgc.VinterpPMG2(*_dims(x[L + 1]), *_dims(x[L]), x[L + 1], e[L],
                         Ps[L])
        x[L].add_(e[L])
        _smooth(ops[L], f[L], x[L], 2, adjoint=1)
    return x


def _run_build(s):
    n0, n1, n2 = _dims(s["op"][0]), _dims(s["P1"]), _dims(s["P2"])
    pmgc.VbuildPb_op7(*n0, *n1, *s["op"], list(s["P1"]))
    pmgc.VbuildG_7(*n0, *n1, list(s["P1"]), *s["op"], list(s["A1"]))
    pmgc.VbuildPb_op27(*n1, *n2, list(s["A1"]), list(s["P2"]))
    pmgc.VbuildG_27(*n1, *n2, list(s["P2"]), list(s["A1"]), list(s["A2"]))
    return [s["P1"], s["A1"], s["P2"], s["A2"]]


# ---------------------------------------------------------------------------
# what a pass cannot do without, and its exact result
# ---------------------------------------------------------------------------
def work(case):
    """Inputs read once, outputs written once. Operations: a V(2,2) cycle
    counts 7-point work on the finest level (five stencil visits, 14
    operations each) and 27-point work below (an eighth of the points, 54
    operations); the solves count twenty cycles, the preconditioned CG
    fourteen, the driver fifteen."""
    kind = case["kind"]
    if kind == "batch":
        parts = [work(dict(kind="solve", n=n, source="atoms", method="cycles",
                           natoms=len(a))) for n, a in _batch(case, 0)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    nx, ny, nz = grid_dims(case)
    n3 = nx * ny * nz
    cycle = 5 * 14 * n3 + 5 * 54 * n3 / 7
    if kind == "solve":
        count = 14 if case["method"] == "pcg" else 20
        b = 8 * n3 * (7 if case["source"] == "arrays" else 1)
        return dict(bytes=b, flops=count * cycle)
    if kind == "driver":
        return dict(bytes=8 * n3 * 6, flops=15 * cycle)
    if kind == "cycle":
        size = 8 if case["dtype"] == "double" else 4
        # finest 4 + f + x0 + x, each coarse level 14 + 27 + x
        return dict(bytes=size * n3 * (7 + 42 / 7), flops=cycle)
    # four diagonals in, 41 arrays out per coarsening; three operations for
    # each of the 430 (7-point) or 1270 (27-point) terms of the fourteen
    # entries
    return dict(bytes=8 * n3 * (4 + 41 / 8 + 41 / 64),
                flops=3 * n3 * (430 / 8 + 1270 / 64))


def exact(case, seed):
    kind = case["kind"]
    if kind in ("solve", "driver"):
        f = _level_arrays(case, seed)
        return solve64([f[k] for k in ("oC", "oE", "oN", "uC")], f["f"],
                       f["x0"], 1e-14)
    if kind == "batch":
        out = []
        for n, atoms in _batch(case, seed):
            f = fine_level((n, n, n), case["h"], atoms)
            out.append(solve64([f[k] for k in ("oC", "oE", "oN", "uC")],
                               f["f"], f["x0"], 1e-14))
        return out
    if kind == "build":
        f = _level_arrays(case, seed)
        (_, A1, A2), (P1, P2) = hierarchy64(f, 3)
        return [P1, torch.stack(A1), P2, torch.stack(A2)]
    ops, Ps, f0, x0 = _cycle_inputs(case, seed)
    ops = [[a.double() for a in op] for op in ops]
    Ps = [P.double() for P in Ps]
    f, x = [f0.double()], [x0.double().clone()]
    for L, P in enumerate(Ps):
        smooth64(ops[L], f[L], x[L], 2, 0)
        f.append(restrict64(residual64(ops[L], f[L], x[L]), P))
        x.append(torch.zeros_like(f[-1]))
    if case["dtype"] == "double":
        x[-1] = solve64(ops[-1], f[-1], x[-1], 0.0, atol=1e-10)
    else:
        smooth64(ops[-1], f[-1], x[-1], 8, 0)
    for L in range(len(Ps) - 1, -1, -1):
        x[L] += interpolate64(x[L + 1], Ps[L], x[L].shape)
        smooth64(ops[L], f[L], x[L], 2, 1)
    return x
