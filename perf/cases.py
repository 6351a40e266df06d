"""Performance cases: what a program that uses this package has it compute.

The package applies H-matrices of displacement-discontinuity cracks, builds
their blocks on the device, solves with them and evaluates fields around the
solution.  The cases run those calls on synthetic cracks of the sizes of the
repository's tests and benchmark (2DS0 segment cracks, 3DR0 rectangle cracks,
a 3DT0 penny-shaped crack), with a cluster tree, an admissibility test and
low-rank blocks of the ranks those matrices have; block entries are random
with the decay and the dominant diagonal of the kernels.

A case is a dict: ``op`` names the call and the other keys its sizes and
options.  ``prepare`` makes the inputs and the handle a program keeps,
``run`` is one pass, ``exact`` the same values in 64 bits by plain torch.
"""
from __future__ import annotations

import functools
import math
from types import SimpleNamespace

import numpy as np
import torch

from bigwham_dev_b200 import HmatGpu
from bigwham_dev_b200.autograd import hmatvec
from bigwham_dev_b200.devbuild import DeviceKernels, factor_layout
from bigwham_dev_b200.fields import R0Fields, S0Fields
from bigwham_dev_b200.meshes import penny_crack_3d, straight_crack_2d
from bigwham_dev_b200.solve import Gmres

DEV = "cuda"
ESIZE = {"fp64": 8, "fp32": 4, "bf16": 2}


def listed():
    return [
        # the smallest call: one straight crack, a step of a time loop (latency, launches)
        dict(name="matvec_2d_256_fp64", op="matvec", mesh="2d", nx=256, ny=1, prec="fp64"),
        # the reference's own call: host arrays in and out, as scipy's solvers use it
        dict(name="matvec_host_3d_64_fp64", op="matvec", mesh="3d", nx=64, ny=64, prec="fp64", host=True),
        # an irregular mesh with ragged leaves and blocks (132,690 DoF penny), 16-bit storage
        dict(name="matvec_penny_bf16", op="matvec", mesh="penny", nx=78, ny=1, prec="bf16"),
        # the headline product: 196,608 DoF, 32-bit storage, larger than any cache
        dict(name="matvec_3d_256_fp32", op="matvec", mesh="3d", nx=256, ny=256, prec="fp32"),
        # a gradient step of an inversion: forward product and its adjoint through autograd
        dict(name="adjoint_3d_128_fp32", op="adjoint", mesh="3d", nx=128, ny=128, prec="fp32"),
        # a population of independent cracks applied by one call (48 cracks, 256 to 16,384 segments)
        dict(name="batch_2d_48_bf16", op="batch", count=48, lo=256, hi=16384, prec="bf16"),
        # a few load cases at once, 32-bit storage
        dict(name="matmat_3d_96_fp32_8", op="matmat", mesh="3d", nx=96, ny=96, prec="fp32", cols=8),
        # many right-hand sides on the tensor cores, as the inner operator of a block solve
        dict(name="matmat_3d_96_bf16_64", op="matmat", mesh="3d", nx=96, ny=96, prec="bf16", cols=64),
        # stresses and displacements on a grid of points around a crack
        dict(name="fields_2d_4000", op="fields2", n=4000, points=50000),
        dict(name="fields_3d_64", op="fields3", nx=64, ny=64, points=20000),
        # the blocks of a crack computed on the device: full-rank assembly and compression
        dict(name="build_3d_64", op="build", nx=64, ny=64),
        # a whole solve: restarted GMRES with the diagonal preconditioner
        dict(name="gmres_3d_64_fp64", op="gmres", mesh="3d", nx=64, ny=64, prec="fp64", restart=30),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["matvec"] * 4 + ["adjoint", "batch", "matmat", "matmat", "fields2", "fields3", "build", "gmres"])
    prec = rng.choice(["fp64", "fp32", "bf16"])
    if op == "matvec":
        mesh = rng.choice(["2d", "3d", "3d", "penny"])
        c = dict(op=op, mesh=mesh, nx=_log_int(rng, 200, 16384), ny=1, prec=prec)
        if mesh == "3d":
            c.update(nx=_log_int(rng, 20, 180), ny=_log_int(rng, 20, 180))
        if mesh == "penny":
            c.update(nx=_log_int(rng, 10, 64))
        if rng.random() < 0.25:
            c["host"] = True
        elif rng.random() < 0.25:
            c["permuted"] = True
        return c
    if op in ("adjoint", "gmres"):
        top = 128 if op == "adjoint" else 64
        c = dict(op=op, mesh="3d", nx=_log_int(rng, 20, top), ny=_log_int(rng, 20, top), prec=prec)
        if op == "gmres":
            c.update(restart=rng.choice([20, 30, 50]), prec="fp64")
        return c
    if op == "batch":
        lo = _log_int(rng, 100, 400)
        return dict(op=op, count=rng.randint(4, 40), lo=lo, hi=lo * rng.randint(2, 32), prec=prec)
    if op == "matmat":
        return dict(op=op, mesh="3d", nx=_log_int(rng, 20, 90), ny=_log_int(rng, 20, 90), prec=prec,
                    cols=rng.randint(2, 16) if prec != "bf16" else rng.randint(2, 130))
    if op == "fields2":
        return dict(op=op, n=_log_int(rng, 100, 4000), points=_log_int(rng, 200, 50000))
    if op == "fields3":
        return dict(op=op, nx=_log_int(rng, 8, 64), ny=_log_int(rng, 8, 64), points=_log_int(rng, 200, 20000))
    return dict(op=op, nx=_log_int(rng, 16, 60), ny=_log_int(rng, 16, 60))


# ---------------------------------------------------------------------------- meshes and block patterns
@functools.lru_cache(maxsize=64)
def _centres(mesh, nx, ny):
    """Collocation points (n, dim) of a crack."""
    if mesh == "2d":
        coor, _ = straight_crack_2d(nx)
        return 0.5 * (coor[1:] + coor[:-1])
    if mesh == "penny":
        coor, conn = penny_crack_3d(1.0 / nx)
        return coor[conn].mean(axis=1)
    x, y = (np.linspace(-1.0, 1.0, n, endpoint=False) + 1.0 / n for n in (nx, ny))
    X, Y = np.meshgrid(x, y)
    return np.column_stack([X.ravel(), Y.ravel(), np.zeros(X.size)])


def _tree(pts, leaf):
    """Cluster tree by median bisection along the widest box axis: permutation,
    node ranges, children (-1: leaf) and boxes."""
    perm = np.arange(len(pts))
    rng, kids = [(0, len(pts))], []
    k = 0
    while k < len(rng):
        a, b = rng[k]
        if b - a <= leaf:
            kids.append((-1, -1))
        else:
            p = pts[perm[a:b]]
            axis = int(np.argmax(p.max(0) - p.min(0)))
            perm[a:b] = perm[a:b][np.argsort(p[:, axis], kind="stable")]
            m = a + (b - a) // 2
            kids.append((len(rng), len(rng) + 1))
            rng += [(a, m), (m, b)]
        k += 1
    # a node's points are final once its descendants are sorted; boxes do not depend on the order
    lo = np.array([pts[perm[a:b]].min(0) for a, b in rng])
    hi = np.array([pts[perm[a:b]].max(0) for a, b in rng])
    return perm, np.array(rng), np.array(kids), lo, hi


@functools.lru_cache(maxsize=96)
def _pattern(mesh, nx, ny, leaf, eta=3.0):
    """Block partition of a crack: permutation, full-rank and admissible blocks
    (rows i0, j0, i1, j1 in points) and the distance of each block's clusters
    in leaf diameters."""
    pts = _centres(mesh, nx, ny)
    perm, rng, kids, lo, hi = _tree(pts, leaf)
    diam = np.linalg.norm(hi - lo, axis=1)
    unit = max(float(np.median(diam[kids[:, 0] < 0])), 1e-300)
    a = b = np.zeros(1, np.int64)
    fr, lr = [], []
    while a.size:
        gap = np.maximum(0.0, np.maximum(lo[a] - hi[b], lo[b] - hi[a]))
        dist = np.linalg.norm(gap, axis=1)
        adm = np.maximum(diam[a], diam[b]) <= eta * dist
        la, lb = kids[a, 0] < 0, kids[b, 0] < 0
        full = ~adm & la & lb
        far = np.linalg.norm(0.5 * (lo[a] + hi[a] - lo[b] - hi[b]), axis=1) / unit
        for sel, out in ((full, fr), (adm, lr)):
            out.append(np.column_stack([rng[a[sel], 0], rng[b[sel], 0], rng[a[sel], 1], rng[b[sel], 1], far[sel]]))
        rest = ~adm & ~full
        a, b, la, lb = a[rest], b[rest], la[rest], lb[rest]
        na, nb = [], []
        for i in (0, 1):
            for j in (0, 1):
                keep = ~((la & (i == 1)) | (lb & (j == 1)))
                na.append(np.where(la, a, kids[a, i])[keep])
                nb.append(np.where(lb, b, kids[b, j])[keep])
        a, b = np.concatenate(na), np.concatenate(nb)
    fr, lr = np.concatenate(fr), np.concatenate(lr)
    return perm.astype(np.int64), fr[:, :4].astype(np.int64), lr[:, :4].astype(np.int64), fr[:, 4], lr[:, 4]


def _shape(mesh):
    """dof per point and leaf size of a mesh family."""
    return {"2d": (2, 32), "3d": (3, 32), "penny": (3, 64)}[mesh]


@functools.lru_cache(maxsize=96)
def _ranked(mesh, nx, ny):
    """The pattern with the ranks the compressed blocks have: 10 on a 2D crack,
    33 to 80 (multiples of 3) on the 3D ones, larger for larger blocks."""
    dof, leaf = _shape(mesh)
    perm, fr, lr, dfr, dlr = _pattern(mesh, nx, ny, leaf)
    side = np.minimum(lr[:, 2] - lr[:, 0], lr[:, 3] - lr[:, 1])
    if mesh == "2d":
        r = np.full(len(lr), 10)
    else:
        level = np.log2(np.maximum(side / leaf, 1.0)).astype(np.int64)
        base = 13 if mesh == "3d" else 11
        r = 3 * (base + level + np.random.default_rng(7).integers(0, 7, len(lr)))
    r = np.minimum(r, dof * side)
    return dof, perm, fr, np.column_stack([lr, r]), dfr, dlr


def _sizes(mesh, nx, ny):
    """(unknowns, stored entries) of a crack's H-matrix."""
    d, perm, fr, lr, _, _ = _ranked(mesh, nx, ny)
    m, n = d * (lr[:, 2] - lr[:, 0]), d * (lr[:, 3] - lr[:, 1])
    e = d * d * int(((fr[:, 2] - fr[:, 0]) * (fr[:, 3] - fr[:, 1])).sum()) + int((lr[:, 4] * (m + n)).sum())
    return d * len(perm), e


def _hmatrix(mesh, nx, ny, seed):
    """Flat form of a crack's H-matrix with random blocks on the device."""
    d, perm, fr, lr, dfr, dlr = _ranked(mesh, nx, ny)
    g = torch.Generator(device=DEV).manual_seed(seed)

    def normal(sizes, scale):
        size = torch.as_tensor(sizes, device=DEV)
        total = int(sizes.sum())
        v = torch.randn(total, dtype=torch.float64, device=DEV, generator=g)
        return v.mul_(torch.repeat_interleave(torch.as_tensor(scale, device=DEV), size, output_size=total))

    # entries decay with the cube (2D: square) of the distance in leaf diameters
    power = 2.0 if mesh == "2d" else 3.0
    m, n = d * (fr[:, 2] - fr[:, 0]), d * (fr[:, 3] - fr[:, 1])
    fr_data = normal(m * n, 0.012 / (1.0 + dfr) ** power)
    off = np.concatenate([[0], np.cumsum(m * n)])
    for k in np.flatnonzero((fr[:, 0] == fr[:, 1]) & (fr[:, 2] == fr[:, 3])):
        fr_data[off[k]:off[k + 1]:int(m[k]) + 1] += 1.0
    m, n, r = d * (lr[:, 2] - lr[:, 0]), d * (lr[:, 3] - lr[:, 1]), lr[:, 4]
    sizes = np.column_stack([m * r, r * n]).ravel()
    amp = 0.012 / (1.0 + dlr) ** power
    lr_data = normal(sizes, np.column_stack([1.0 / np.sqrt(np.maximum(r, 1)), amp]).ravel())
    nd = d * len(perm)
    return dict(dof=d, n_rows=nd, n_cols=nd, fr=fr, lr=lr, fr_data=fr_data, lr_data=lr_data, perm0=perm, perm1=perm)


def _vector(n, seed, cols=None):
    g = torch.Generator(device=DEV).manual_seed(seed + 1000003)
    shape = (n,) if cols is None else (cols, n)
    v = torch.rand(shape, dtype=torch.float64, device=DEV, generator=g).mul_(2.0).sub_(1.0)
    return v if cols is None else v.t()


def _members(c):
    """Segment counts of a batch's cracks, spread over their logarithm."""
    r = np.random.default_rng(3)
    return [int(v) for v in np.round(np.exp(r.uniform(math.log(c["lo"]), math.log(c["hi"]), c["count"])))]


# ---------------------------------------------------------------------------- elements
def _segments(n, seed):
    """A bent crack of n segments: coordinates and connectivity."""
    r = np.random.default_rng(seed)
    x = np.linspace(-1.0, 1.0, n + 1) + r.uniform(-0.2, 0.2, n + 1) / n
    coor = np.column_stack([x, 0.2 * np.sin(2.0 * x) + 0.01 * r.standard_normal()])
    return coor, np.column_stack([np.arange(n), np.arange(1, n + 1)])


def _rectangles(nx, ny, seed, rotation):
    """Element records (centre, rotation, normal, half sides) of a rectangle
    crack whose spacing varies along both sides."""
    r = np.random.default_rng(seed)
    gx, gy = (np.concatenate([[0.0], np.cumsum(r.uniform(0.8, 1.2, n))]) for n in (nx, ny))
    gx, gy = 2.0 * gx / gx[-1] - 1.0, 2.0 * gy / gy[-1] - 1.0
    X, Y = np.meshgrid(0.5 * (gx[1:] + gx[:-1]), 0.5 * (gy[1:] + gy[:-1]))
    A, B = np.meshgrid(0.5 * np.diff(gx), 0.5 * np.diff(gy))
    cp = np.column_stack([X.ravel(), Y.ravel(), np.zeros(X.size)]) @ rotation  # local = rotation global
    one = np.ones((X.size, 1))
    rec = np.hstack([cp, one * rotation.reshape(1, 9), one * rotation[2:3], A.reshape(-1, 1), B.reshape(-1, 1)])
    return np.ascontiguousarray(rec)


def _skew():
    a, b = 0.4, 0.7
    Rz = np.array([[math.cos(a), math.sin(a), 0], [-math.sin(a), math.cos(a), 0], [0, 0, 1.0]])
    Rx = np.array([[1.0, 0, 0], [0, math.cos(b), math.sin(b)], [0, -math.sin(b), math.cos(b)]])
    return Rx @ Rz


YOUNG, POISSON = 1.0, 0.25


def _points(c, seed):
    """Observation points off the crack and the DD of every element."""
    dim = 2 if c["op"] == "fields2" else 3
    ne = c["n"] if dim == 2 else c["nx"] * c["ny"]
    g = torch.Generator(device=DEV).manual_seed(seed)
    p = torch.rand((c["points"], dim), dtype=torch.float64, device=DEV, generator=g).mul_(3.0).sub_(1.5)
    dd = torch.rand(dim * ne, dtype=torch.float64, device=DEV, generator=g).add_(0.5)
    return p, dd


# ---------------------------------------------------------------------------- the cases
def prepare(case, seed):
    c, op = case, case["op"]
    s = SimpleNamespace(c=c)
    if op in ("matvec", "adjoint", "matmat", "gmres"):
        flat = _hmatrix(c["mesh"], c["nx"], c["ny"], seed)
        n = flat["n_rows"]
        if op == "matmat" and c["prec"] == "bf16":  # the tensor-core layout is made from host blocks
            flat["fr_data"], flat["lr_data"] = flat["fr_data"].cpu().numpy(), flat["lr_data"].cpu().numpy()
            s.h = HmatGpu.from_flat(**flat, precisions=("bf16",), matmat=True)
        else:
            s.h = HmatGpu.from_device_flat(**flat, precisions=(c["prec"],), transpose=op == "adjoint")
        s.x = _vector(n, seed, c.get("cols"))
        if c.get("host"):
            s.x = s.x.cpu().numpy()
        if op == "adjoint":
            s.x.requires_grad_(True)
            s.w = _vector(n, seed + 1)
        if op == "gmres":
            minv = 1.0 / torch.from_numpy(s.h.diagonal()).to(DEV)
            s.solver = Gmres(lambda x, y: s.h.matvec(x, c["prec"], out=y), n, c["restart"], minv)
    elif op == "batch":
        members = []
        for k, n in enumerate(_members(c)):
            f = _hmatrix("2d", n, 1, seed + 7919 * k)
            f["fr_data"], f["lr_data"] = f["fr_data"].cpu().numpy(), f["lr_data"].cpu().numpy()
            members.append(SimpleNamespace(**f))
        s.h = HmatGpu.batch(members, precisions=(c["prec"],))
        s.x = _vector(s.h.n_cols, seed)
    elif op == "fields2":
        s.f = S0Fields(*_segments(c["n"], seed), YOUNG, POISSON)
        s.p, s.dd = _points(c, seed)
    elif op == "fields3":
        s.f = R0Fields(_rectangles(c["nx"], c["ny"], seed, _skew()), YOUNG, POISSON)
        s.p, s.dd = _points(c, seed)
    else:
        s.rec = _rectangles(c["nx"], c["ny"], seed, np.eye(3))
        s.perm, s.fr, s.lr, _, _ = _pattern("3d", c["nx"], c["ny"], 32)
        s.k = DeviceKernels()
    return s


def _written(data, size, limit, width=None):
    """The entries of each block that hold factors, zeros in the room left over:
    the first `limit` of every `width` entries (default: of the whole block)."""
    size, limit = (torch.as_tensor(v, device=DEV) for v in (size, limit))
    total = data.numel()
    pos = torch.arange(total, device=DEV) - torch.repeat_interleave(size.cumsum(0) - size, size, output_size=total)
    if width is not None:
        pos %= torch.repeat_interleave(torch.as_tensor(width, device=DEV), size, output_size=total)
    return data.masked_fill_(pos >= torch.repeat_interleave(limit, size, output_size=total), 0.0)


def _build(s):
    """Full-rank blocks and low-rank factors of a crack, in the flat layout of
    the device entries."""
    G, cap = YOUNG / (2.0 * (1.0 + POISSON)), 48
    fr = s.k.assemble_fr(s.rec, G, POISSON, s.fr, s.perm)
    fa, fb, rank, err = s.k.aca(s.rec, G, POISSON, s.lr, s.perm, 1e-5, cap)
    n0, n1, capk, a_off, b_off = factor_layout(s.lr, cap)
    r = rank.astype(np.int64)
    return {"fr": fr, "a": _written(fa, np.diff(a_off), r * 3 * n0), "b": _written(fb, np.diff(b_off), r, 3 * capk),
            "rank": rank, "err": err}


def run(state):
    s, c = state, state.c
    op = c["op"]
    if op in ("matvec", "batch"):
        return s.h.matvec(s.x, c["prec"], permuted=c.get("permuted", False))
    if op == "adjoint":
        y = hmatvec(s.x, s.h, c["prec"])
        (g,) = torch.autograd.grad(y, s.x, s.w)
        return y, g
    if op == "matmat":
        return s.h.matmat(s.x, c["prec"])
    if op == "gmres":
        return s.solver.solve(s.x, tol=1e-8)[0]
    if op in ("fields2", "fields3"):
        return s.f.fields(s.p, s.dd)
    return _build(s)


def work(case):
    """Stored entries read once, vectors read and written once.  Fields and
    builds are arithmetic: per element-point pair about 150 (2D) or 700 (3D)
    floating-point operations, functions counted by their polynomials."""
    c, op = case, case["op"]
    if op in ("matvec", "adjoint", "matmat", "gmres"):
        n, e = _sizes(c["mesh"], c["nx"], c["ny"])
        passes = {"adjoint": 2, "gmres": 2 * c.get("restart", 0)}.get(op, 1)
        cols = c.get("cols", 1)
        return {"bytes": passes * (e * ESIZE[c["prec"]] + 16 * n * cols), "flops": 2 * e * cols * passes}
    if op == "batch":
        both = [_sizes("2d", k, 1) for k in _members(c)]
        return {"bytes": sum(e * ESIZE[c["prec"]] + 16 * n for n, e in both), "flops": 2 * sum(e for _, e in both)}
    if op == "fields2":
        return {"bytes": 56 * (c["n"] + c["points"]), "flops": 150 * c["n"] * c["points"]}
    ne = c["nx"] * c["ny"]
    if op == "fields3":
        return {"bytes": 160 * ne + 96 * c["points"], "flops": 700 * ne * c["points"]}
    _, fr, lr, _, _ = _pattern("3d", c["nx"], c["ny"], 32)
    pairs = int(((fr[:, 2] - fr[:, 0]) * (fr[:, 3] - fr[:, 1])).sum())
    r, side = 45, int((lr[:, 2] - lr[:, 0] + lr[:, 3] - lr[:, 1]).sum())
    return {"bytes": 72 * pairs + 24 * r * side + 136 * ne, "flops": 500 * (pairs + side * r // 3) + 6 * r * r * side}


def tolerance(case):
    """About four times the error against 64 bits that each path shows."""
    c, op = case, case["op"]
    if op == "gmres":
        return {"rel": 4e-8}  # stops at a residual of 1e-8
    if op == "build":
        return {"rel": 4e-9, "max": 4e-6, "differ": 0.002}  # factors amplify rounding by 1 / eps
    if op in ("fields2", "fields3"):
        return {"rel": 1e-13}
    if op == "matmat" and c["prec"] == "bf16":
        return {"rel": 1e-2}  # right-hand sides and phase-1 products in 16 bits too
    return {"rel": {"fp64": 2e-15, "fp32": 7e-7, "bf16": 5e-3}[c["prec"]]}


# ---------------------------------------------------------------------------- 64-bit values
def _apply(flat, x, transpose=False, permuted=False):
    """H x block by block in float64, original ordering unless permuted."""
    d = flat["dof"]
    p = (d * torch.as_tensor(flat["perm0"], device=DEV)[:, None] + torch.arange(d, device=DEV)).reshape(-1)
    v = x if permuted else x[p]
    y = torch.zeros_like(v)
    at = 0
    for i0, j0, i1, j1 in (flat["fr"] * d).tolist():
        m, n = i1 - i0, j1 - j0
        a = flat["fr_data"][at:at + m * n].view(n, m)  # the transposed block
        if transpose:
            y[j0:j1] += a @ v[i0:i1]
        else:
            y[i0:i1] += a.t() @ v[j0:j1]
        at += m * n
    at = 0
    for (i0, j0, i1, j1), r in zip((flat["lr"][:, :4] * d).tolist(), flat["lr"][:, 4].tolist()):
        m, n = i1 - i0, j1 - j0
        a = flat["lr_data"][at:at + m * r].view(r, m)
        b = flat["lr_data"][at + m * r:at + r * (m + n)].view(n, r)
        if transpose:
            y[j0:j1] += b @ (a @ v[i0:i1])
        else:
            y[i0:i1] += a.t() @ (b.t() @ v[j0:j1])
        at += r * (m + n)
    if permuted:
        return y
    out = torch.empty_like(y)
    out[p] = y
    return out


def _fields2(coor, conn, p, dd):
    """Constant-DD segment solution (Crouch and Starfield), plane strain."""
    coor, conn = torch.as_tensor(coor, device=DEV), torch.as_tensor(conn, device=DEV)
    v0, v1 = coor[conn[:, 0]], coor[conn[:, 1]]
    t = v1 - v0
    a = 0.5 * t.norm(dim=1)
    t = t / t.norm(dim=1, keepdim=True)
    nrm = torch.stack([-t[:, 1], t[:, 0]], 1)
    G, nu = YOUNG / (2.0 * (1.0 + POISSON)), POISSON
    c = 1.0 / (4.0 * math.pi * (1.0 - nu))
    ds, dn = dd[0::2], dd[1::2]
    S, U = [], []
    for q in p.split(2000):
        r = q[:, None, :] - 0.5 * (v0 + v1)
        x, y = (r * t).sum(2), (r * nrm).sum(2)
        xm, xp = x - a, x + a
        r1, r2 = xm * xm + y * y, xp * xp + y * y
        fx = 0.5 * c * (r1.log() - r2.log())
        fy = -c * (torch.atan2(y, xm) - torch.atan2(y, xp))
        fxy = c * (y / r1 - y / r2)
        fyy = -c * (xm / r1 - xp / r2)
        fxyy = c * ((xm * xm - y * y) / (r1 * r1) - (xp * xp - y * y) / (r2 * r2))
        fyyy = 2.0 * c * y * (xm / (r1 * r1) - xp / (r2 * r2))
        sxx = 2 * G * (ds * (2 * fxy + y * fxyy) + dn * (fyy + y * fyyy))
        syy = 2 * G * (ds * (-y * fxyy) + dn * (fyy - y * fyyy))
        sxy = 2 * G * (ds * (fyy + y * fyyy) + dn * (-y * fxyy))
        ux = ds * (2 * (1 - nu) * fy + y * fyy) - dn * ((1 - 2 * nu) * fx + y * fxy)
        uy = ds * ((1 - 2 * nu) * fx - y * fxy) + dn * (2 * (1 - nu) * fy - y * fyy)
        (tx, ty), (nx, ny) = t.t(), nrm.t()
        S.append(torch.stack([(sxx * tx * tx + syy * nx * nx + 2 * sxy * tx * nx).sum(1),
                              (sxx * ty * ty + syy * ny * ny + 2 * sxy * ty * ny).sum(1),
                              (sxx * tx * ty + syy * nx * ny + sxy * (tx * ny + nx * ty)).sum(1)], 1))
        U.append(torch.stack([(ux * tx + uy * nx).sum(1), (ux * ty + uy * ny).sum(1)], 1))
    return torch.cat(S), torch.cat(U)


def _fields3(rec, p, dd):
    """Rectangular DD: Kelvin's solution from the derivatives of the integral
    of 1 / R over the rectangle, summed over its corners."""
    rec = torch.as_tensor(rec, device=DEV)
    cp, R, a, b = rec[:, :3], rec[:, 3:12].view(-1, 3, 3), rec[:, 15], rec[:, 16]
    G, nu = YOUNG / (2.0 * (1.0 + POISSON)), POISSON
    D = dd.view(-1, 3)
    S, U = [], []
    for q in p.split(400):
        x, y, z = torch.einsum("eij,pej->ipe", R, q[:, None, :] - cp)
        d = {}

        def add(key, value):
            d[key] = d[key] + value if key in d else value

        for sx in (1.0, -1.0):
            for sy in (1.0, -1.0):
                s, X, Y = sx * sy, x + sx * a, y + sy * b
                r = (X * X + Y * Y + z * z).sqrt()
                for k, (P, Q) in {"x": (X, Y), "y": (Y, X)}.items():  # terms in ln(Q + r) and their mirror
                    w = torch.where(Q >= 0, r + Q, (P * P + z * z) / (r - Q))
                    e = (r * w - P * P * (2 * r + Q) / r) / (r * r * w * w)
                    add(k, s * w.log())
                    add(k * 2, s * P / (r * w))
                    add(k + "z", s * z / (r * w))
                    add(k * 3, s * e)
                    add(k * 2 + "z", -s * P * z * (2 * r + Q) / (r ** 3 * w * w))
                    add(k + "zz", s * (r * w - z * z * (2 * r + Q) / r) / (r * r * w * w))
                add("z", -s * torch.atan(X * Y / (z * r)))
                add("xy", s / r)
                add("zz", s * X * Y * (X * X + Y * Y + 2 * z * z) / (r * (X * X + z * z) * (Y * Y + z * z)))
                add("xxy", -s * X / r ** 3)
                add("xyy", -s * Y / r ** 3)
                add("xyz", -s * z / r ** 3)
        zzz = -(d["xxz"] + d["yyz"])
        C, c, k1, k2 = G / (4 * math.pi * (1 - nu)), 1 / (8 * math.pi * (1 - nu)), 2 * (1 - nu), 1 - 2 * nu
        d0, d1, d2 = D.t()
        xx = d0 * (2 * d["xz"] - z * d["xxx"]) + d1 * (2 * nu * d["yz"] - z * d["xxy"])
        xx = C * (xx + d2 * (d["zz"] + k2 * d["yy"] - z * d["xxz"]))
        yy = d0 * (2 * nu * d["xz"] - z * d["xyy"]) + d1 * (2 * d["yz"] - z * d["yyy"])
        yy = C * (yy + d2 * (d["zz"] + k2 * d["xx"] - z * d["yyz"]))
        zz = C * (-d0 * z * d["xzz"] - d1 * z * d["yzz"] + d2 * (d["zz"] - z * zzz))
        xy = d0 * ((1 - nu) * d["yz"] - z * d["xxy"]) + d1 * ((1 - nu) * d["xz"] - z * d["xyy"])
        xy = C * (xy - d2 * (k2 * d["xy"] + z * d["xyz"]))
        xz = d0 * (d["zz"] + nu * d["yy"] - z * d["xxz"]) - d1 * (nu * d["xy"] + z * d["xyz"]) - d2 * z * d["xzz"]
        yz = -d0 * (nu * d["xy"] + z * d["xyz"]) + d1 * (d["zz"] + nu * d["xx"] - z * d["yyz"]) - d2 * z * d["yzz"]
        xz, yz = C * xz, C * yz
        T = torch.stack([xx, xy, xz, xy, yy, yz, xz, yz, zz], -1).view(*xx.shape, 3, 3)
        T = torch.einsum("eki,pekl,elj->pij", R, T, R)
        S.append(torch.stack([T[:, 0, 0], T[:, 1, 1], T[:, 2, 2], T[:, 0, 1], T[:, 0, 2], T[:, 1, 2]], 1))
        u = c * torch.stack([
            d0 * (k1 * d["z"] - z * d["xx"]) - d1 * z * d["xy"] - d2 * (k2 * d["x"] + z * d["xz"]),
            -d0 * z * d["xy"] + d1 * (k1 * d["z"] - z * d["yy"]) - d2 * (k2 * d["y"] + z * d["yz"]),
            d0 * (k2 * d["x"] - z * d["xz"]) + d1 * (k2 * d["y"] - z * d["yz"]) + d2 * (k1 * d["z"] - z * d["zz"])], -1)
        U.append(torch.einsum("eki,pek->pi", R, u))
    return torch.cat(S), torch.cat(U)


def _assembled(rec, fr, perm):
    """Full-rank blocks of a planar crack: tractions at the receiver's centre
    due to unit DDs of the source, from the corner distances in the plane."""
    G, nu = YOUNG / (2.0 * (1.0 + POISSON)), POISSON
    C = G / (4 * math.pi * (1 - nu))
    rec = torch.as_tensor(rec[perm], device=DEV)
    out = []
    for i0, j0, i1, j1 in fr.tolist():
        rcv, src = rec[i0:i1], rec[j0:j1]
        x, y = (rcv[None, :, k] - src[:, None, k] for k in (0, 1))  # (source, receiver)
        a, b = src[:, None, 15], src[:, None, 16]
        xx = yy = xy = 0.0
        for sx in (1.0, -1.0):
            for sy in (1.0, -1.0):
                X, Y = x + sx * a, y + sy * b
                r = torch.hypot(X, Y)
                # X / (r (r + Y)) = (r - Y) / (r X), which does not cancel for Y < 0
                xx = xx + sx * sy * torch.where(Y >= 0, X / (r * (r + Y)), (r - Y) / (r * X))
                yy = yy + sx * sy * torch.where(X >= 0, Y / (r * (r + X)), (r - X) / (r * Y))
                xy = xy + sx * sy / r
        zz = -(xx + yy)
        o = torch.zeros_like(zz)
        K = torch.stack([torch.stack([C * (zz + nu * yy), -C * nu * xy, o], -1),
                         torch.stack([-C * nu * xy, C * (zz + nu * xx), o], -1),
                         torch.stack([o, o, C * zz], -1)], -2)  # (source, receiver, traction, DD)
        out.append(K.permute(0, 3, 1, 2).reshape(-1))  # column-major: (source, DD) columns
    return torch.cat(out)


def exact(case, seed):
    c, op = case, case["op"]
    if op == "fields2":
        return _fields2(*_segments(c["n"], seed), *_points(c, seed))
    if op == "fields3":
        return _fields3(_rectangles(c["nx"], c["ny"], seed, _skew()), *_points(c, seed))
    if op == "build":
        perm, fr, _, _, _ = _pattern("3d", c["nx"], c["ny"], 32)
        full = _assembled(_rectangles(c["nx"], c["ny"], seed, np.eye(3)), fr, perm)
        return {"fr": full, "a": None, "b": None, "rank": None, "err": None}
    if op == "batch":
        flats = [_hmatrix("2d", n, 1, seed + 7919 * k) for k, n in enumerate(_members(c))]
        x = _vector(sum(f["n_cols"] for f in flats), seed)
        return torch.cat([_apply(f, v) for f, v in zip(flats, x.split([f["n_cols"] for f in flats]))])
    flat = _hmatrix(c["mesh"], c["nx"], c["ny"], seed)
    x = _vector(flat["n_rows"], seed, c.get("cols"))
    if op == "gmres":
        dense = _apply(flat, torch.eye(flat["n_rows"], dtype=torch.float64, device=DEV))
        return torch.linalg.solve(dense, x)
    y = _apply(flat, x, permuted=c.get("permuted", False))
    if op == "adjoint":
        return y, _apply(flat, _vector(flat["n_rows"], seed + 1), transpose=True)
    return y.cpu().numpy() if c.get("host") else y
