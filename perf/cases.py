"""The work that users of this package have it do, as timed cases.

Every case calls the public entry points the way a program does: whole solves
(CG, GMRES, full multigrid, batches, the differentiable solve) and the single
level operations a user's own driver is built from (operator, smoother,
transfer, V-cycle, right-hand-side assembly).  ``exact`` restates each of them
in 64-bit torch from the definitions (dense 1D matrices and their Kronecker
structure), without the package.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import gputensorproductsmoother_b200 as tps

DTYPES = {"fp64": torch.float64, "fp32": torch.float32}
ITERATIONS = 6  # CG iterations of a constant-coefficient solve to 1e-10 (5..7 over degrees and sizes)


def listed():
    return [
        # the smallest whole solve: 2D Q2 on 64^2 cells, uniform nodal data;
        # hundreds of launches on a few thousand unknowns
        {"name": "cg_2d_q2_64", "kind": "cg", "dim": 2, "degree": 2, "cells": 64, "precision": "fp64"},
        # the headline solve: 3D Q4, 64^3 cells, FP32 V-cycle under the FP64 CG
        {"name": "cg_3d_q4_64", "kind": "cg", "dim": 3, "degree": 4, "cells": 64, "precision": "fp32"},
        # the high-order solve: 3D Q7, 32^3 cells
        {"name": "cg_3d_q7_32", "kind": "cg", "dim": 3, "degree": 7, "cells": 32, "precision": "fp32"},
        # many right-hand sides on one mesh plus meshes of uneven size, solved together
        {"name": "batch_3d_q3", "kind": "batch", "degree": 3, "cells": 32, "copies": 32, "others": 12,
         "precision": "fp32"},
        # forward and backward of the differentiable solve, per-cell coefficient, FP64, 3 * 2^4 cells
        {"name": "adjoint_3d_q4_48", "kind": "adjoint", "dim": 3, "degree": 4, "cells": 48},
        # the Poisson program's own driver (left-preconditioned GMRES), 3 * 2^3 cells
        {"name": "gmres_3d_q3_24", "kind": "gmres", "dim": 3, "degree": 3, "cells": 24,
         "precision": "fp64_rounded"},
        # one full-multigrid pass with Dirichlet data, 5 * 2^3 cells
        {"name": "fmg_3d_q2_40", "kind": "fmg", "dim": 3, "degree": 2, "cells": 40, "precision": "fp32"},
        # a V-cycle as a preconditioner in a user's own Krylov loop, large 2D mesh of 3 * 2^7 cells
        {"name": "vcycle_2d_q5_384", "kind": "vcycle", "dim": 2, "degree": 5, "cells": 384, "precision": "fp32"},
        # the operator of that loop, FP64, 3D Q4 on 64^3 cells
        {"name": "vmult_3d_q4_64", "kind": "vmult", "dim": 3, "degree": 4, "cells": 64, "dtype": "fp64"},
        # pre- and post-smoothing of a user's own multigrid on caller-owned vectors
        {"name": "smooth_3d_q4_64", "kind": "smooth", "dim": 3, "degree": 4, "cells": 64, "dtype": "fp32"},
        # the grid transfers of that multigrid, both ways
        {"name": "transfer_3d_q3_48", "kind": "transfer", "dim": 3, "degree": 3, "cells": 48, "dtype": "fp64"},
        # right-hand-side assembly for a general f at the Gauss points
        {"name": "assemble_3d_q4_48", "kind": "assemble", "dim": 3, "degree": 4, "cells": 48},
    ]


# what may be drawn per kind: dimensions, most unknowns (log-uniform sizes up to it)
RANGES = {
    "cg": ((2, 3, 3), 12e6),
    "batch": ((3,), 1.2e6),
    "adjoint": ((2, 3, 3), 3e6),
    "gmres": ((2, 3, 3), 3e6),
    "fmg": ((2, 3, 3), 6e6),
    "vcycle": ((2, 3), 12e6),
    "vmult": ((2, 3, 3), 17e6),
    "smooth": ((2, 3, 3), 17e6),
    "transfer": ((2, 3, 3), 17e6),
    "assemble": ((2, 3, 3), 8e6),
}


def draw(rng):
    """One more case: the kinds of the list in turn at random, any degree, cells m * 2^l with
    m = 2, 3 or 5, sizes log-uniform from a few hundred unknowns to the kind's largest."""
    kind = rng.choice(sorted(RANGES))
    dims, most = RANGES[kind]
    dim, degree = rng.choice(dims), rng.randint(1, 7)
    if kind == "adjoint":
        degree = rng.randint(2, 5)
    # coarsest meshes whose dense coarse solve stays small
    bases = [m for m in (2, 3, 5) if m == 2 or (m * degree - 1) ** dim <= 1400]
    sizes = sorted({m << l for m in bases for l in range(1, 11) if (m * degree << l) ** dim <= most})
    target = math.exp(rng.uniform(math.log(300.0), math.log(most)))
    near = sorted(sizes, key=lambda n: abs(math.log((n * degree + 1) ** dim / target)))
    c = {"kind": kind, "dim": dim, "degree": degree, "cells": rng.choice(near[:2])}
    if kind == "batch":
        del c["dim"]
        c["copies"], c["others"] = rng.randint(2, 16), rng.randint(1, 8)
    if kind in ("cg", "batch", "fmg", "vcycle"):
        c["precision"] = rng.choice(["fp32", "fp32", "fp64"])
    elif kind == "gmres":
        c["precision"] = rng.choice(["fp64_rounded", "fp32", "fp64"])
    elif kind in ("vmult", "smooth", "transfer"):
        c["dtype"] = rng.choice(["fp64", "fp32"])
    return c


# ---- 1D data from the definitions -------------------------------------------

def _nodes(k):
    if k == 1:
        return np.array([0.0, 1.0])
    inner = np.polynomial.legendre.Legendre.basis(k).deriv().roots()
    return np.concatenate([[0.0], np.sort(0.5 * (inner + 1.0)), [1.0]])


def _basis(k, x):
    """Values and derivatives of the k+1 Lagrange polynomials at x: (len(x), k+1) each."""
    t = _nodes(k)
    V, D = np.ones((len(x), k + 1)), np.zeros((len(x), k + 1))
    for i in range(k + 1):
        others = [m for m in range(k + 1) if m != i]
        for m in others:
            V[:, i] *= (x - t[m]) / (t[i] - t[m])
        for d in others:
            p = np.full(len(x), 1.0 / (t[i] - t[d]))
            for m in others:
                if m != d:
                    p *= (x - t[m]) / (t[i] - t[m])
            D[:, i] += p
    return V, D


def _gauss(k):
    x, w = np.polynomial.legendre.leggauss(k + 1)
    return 0.5 * (x + 1.0), 0.5 * w


def _cell_matrices(k):
    x, w = _gauss(k)
    V, D = _basis(k, x)
    return (V * w[:, None]).T @ V, (D * w[:, None]).T @ D


def _global(cell, k, n):
    A = np.zeros((n * k + 1, n * k + 1))
    for c in range(n):
        A[c * k:c * k + k + 1, c * k:c * k + k + 1] += cell
    return A


def _gpu(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def _mass_stiffness(k, n):
    M, S = _cell_matrices(k)
    return _gpu(_global(M / n, k, n)), _gpu(_global(S * n, k, n))


def _along(A, v, axis):
    """A applied to v along one axis."""
    return torch.movedim(torch.tensordot(A, v, dims=([1], [axis])), 0, axis)


def _kron(mats, v):
    for axis, A in enumerate(mats):
        v = _along(A, v, axis)
    return v


def _grid(v, dim, n1):
    return v.reshape((n1,) * dim)


def _inner(dim):
    return (slice(1, -1),) * dim


def _zero_boundary(v):
    out = torch.zeros_like(v)
    out[_inner(v.dim())] = v[_inner(v.dim())]
    return out


# ---- inputs -----------------------------------------------------------------

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)


def _uniform(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64) * 2.0 - 1.0


def _rhs(g, dim, k, n):
    """b = M f for i.i.d. uniform nodal values f, Dirichlet rows zero (flat)."""
    M, _ = _mass_stiffness(k, n)
    f = _zero_boundary(_uniform(g, *((n * k + 1,) * dim)))
    return _zero_boundary(_kron([M] * dim, f)).reshape(-1).contiguous()


def _smooth_field(g, dim, n1):
    """Eight random sine modes at equidistant points (a smooth field that vanishes on the boundary)."""
    t = torch.linspace(0.0, 1.0, n1, dtype=torch.float64, device="cuda")
    amp, freq = _uniform(g, 8), torch.randint(1, 9, (8, dim), generator=g, device="cuda")
    s = torch.sin(math.pi * freq[:, :, None] * t)
    spec = "az,ay,ax,a->zyx" if dim == 3 else "ay,ax,a->yx"
    return torch.einsum(spec, *[s[:, d] for d in range(dim)], amp).reshape(-1).contiguous()


def _kappa(g, dim, n):
    return torch.exp(0.5 * torch.randn(n ** dim, generator=g, device="cuda", dtype=torch.float64))


def _batch_systems(case):
    """(3, degree, cells) per system: copies of one mesh, then meshes of a few sizes in turn."""
    n = case["cells"]
    cells = [n] * case["copies"]
    sizes = sorted({max(4, q) for q in (n // 4, 5 * n // 16, 3 * n // 8, 5 * n // 8, 3 * n // 4, n, 5 * n // 4,
                                        3 * n // 2)})
    sizes = [q for q in sizes if _coarse_fits(3, case["degree"], q)]
    return [(3, case["degree"], q) for q in cells + [sizes[(3 * i) % len(sizes)] for i in range(case["others"])]]


def _coarse_fits(dim, k, n):
    m = tps.split_cells(n)[0]
    return m == 2 or (m * k - 1) ** dim <= 1400


def _inputs(case, seed):
    kind, k, n = case["kind"], case["degree"], case["cells"]
    g = _generator(seed)
    if kind == "batch":
        return {"b": [_rhs(g, d, q, m) for d, q, m in _batch_systems(case)]}
    dim, n1 = case["dim"], case["cells"] * case["degree"] + 1
    dt = DTYPES[case.get("dtype", "fp64")]
    if kind in ("cg", "gmres", "vcycle"):
        return {"b": _rhs(g, dim, k, n)}
    if kind == "adjoint":
        f = _uniform(g, n1 ** dim)
        return {"kappa": _kappa(g, dim, n), "f": f, "target": 0.01 * _smooth_field(g, dim, n1)}
    if kind == "fmg":
        levels = _levels(n)
        t = {q: torch.linspace(0.0, 1.0, q * k + 1, dtype=torch.float64, device="cuda") for q in levels}
        bnd = []
        for q in levels:  # Dirichlet values of x + 2 y (+ z) at the boundary nodes
            v = t[q] + 2.0 * t[q][:, None]
            v = v + t[q][:, None, None] if dim == 3 else v
            bnd.append((v - _zero_boundary(v)).reshape(-1).contiguous())
        return {"rhs": [_rhs(g, dim, k, q) for q in levels], "bnd": bnd}
    if kind in ("vmult", "smooth"):
        return {"x": _uniform(g, n1 ** dim).to(dt), "b": _rhs(g, dim, k, n).to(dt)}
    if kind == "transfer":
        nc1 = n // 2 * k + 1
        return {"fine": _uniform(g, n1 ** dim).to(dt), "coarse": _uniform(g, nc1 ** dim).to(dt)}
    if kind == "assemble":
        return {"fq": _uniform(g, n ** dim, (k + 1) ** dim)}
    raise ValueError(kind)


def _levels(n):
    m, levels = tps.split_cells(n)
    return [m << l for l in range(levels)]


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    kind = case["kind"]
    if kind == "batch":
        s["solver"] = tps.BatchSolver(_batch_systems(case))
        return s
    P = tps.PoissonProblem(case["dim"], case["degree"], case["cells"], kappa=s.get("kappa"))
    s["problem"] = P
    dt = DTYPES[case.get("dtype", "fp64")]
    if kind in ("cg", "gmres", "fmg", "vcycle"):
        s["solver"] = tps.MultigridSolvers(P)
    if kind == "vcycle":
        s["out"] = P.new_vector()
    if kind == "vmult":
        s["op"], s["out"] = tps.LaplaceOperator(P), P.new_vector(dtype=dt)
    if kind == "smooth":
        s["op"], s["out"] = tps.PatchSmoother(P), P.new_vector(dtype=dt)
    if kind == "transfer":
        L = P.n_levels - 1
        s["op"], s["up"], s["down"] = tps.MGTransferCUDA(P), P.new_vector(dtype=dt), P.new_vector(L - 1, dtype=dt)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "cg":
        return s["solver"].solve_cg(s["b"], precision=case["precision"])[0]
    if kind == "batch":
        return s["solver"].solve(s["b"], precision=case["precision"])[0]
    if kind == "adjoint":
        f, kappa = s["f"].detach().requires_grad_(True), s["kappa"].detach().requires_grad_(True)
        u = tps.autograd.solve(s["problem"], f, kappa)
        (0.5 * ((u - s["target"]) ** 2).sum()).backward()
        return u.detach(), f.grad, kappa.grad
    if kind == "gmres":
        return s["solver"].solve_gmres(s["b"], precision=case["precision"])[0]
    if kind == "fmg":
        return s["solver"].solve_fmg(s["rhs"], s["bnd"], precision=case["precision"])[0]
    if kind == "vcycle":
        s["solver"].vmult(s["out"], s["b"], precision=case["precision"])
        return s["out"]
    if kind == "vmult":
        s["op"].vmult(s["out"], s["x"])
        return s["out"]
    if kind == "smooth":
        s["op"].vmult(s["out"], s["b"])
        s["op"].step(s["out"], s["b"], reverse=True)
        return s["out"]
    if kind == "transfer":
        L = s["problem"].n_levels - 1
        s["down"].zero_()
        s["op"].restrict_and_add(L, s["down"], s["fine"])
        s["op"].prolongate(L, s["up"], s["coarse"])
        return s["down"], s["up"]
    return s["problem"].assemble_rhs(s["fq"])


# ---- the work a pass cannot do without --------------------------------------

def _operator_flops(dim, k, n):
    """Banded 1D contractions (k + 2 entries a row on average): 4 of them in 2D, 7 in 3D."""
    return (4 if dim == 2 else 7) * 2.0 * (k + 2) * (n * k + 1) ** dim


def _sweep_flops(dim, k, n):
    """Every patch: its box residual (ring columns only) and the fast diagonalisation of its interior."""
    m = 2 * k - 1
    return (n - 1) ** dim * m ** dim * (2.0 * m * 2 * dim + 2.0 * 2 * (2 * dim - 1))


def _vcycle_flops(dim, k, n):
    """Two sweeps and a residual per level (the transfers are small beside them)."""
    return sum(2 * _sweep_flops(dim, k, q) + _operator_flops(dim, k, q) for q in _levels(n)[1:])


def _cg_flops(dim, k, n, iterations):
    """Per iteration a V-cycle, q = A p and the vector updates."""
    return iterations * (_vcycle_flops(dim, k, n) + _operator_flops(dim, k, n) + 12.0 * (n * k + 1) ** dim)


def work(case):
    kind, k, n = case["kind"], case["degree"], case["cells"]
    size = 4 if case.get("dtype") == "fp32" else 8
    if kind == "batch":
        parts = _batch_systems(case)
        return {"bytes": sum(16.0 * (m * q + 1) ** d for d, q, m in parts),
                "flops": sum(_cg_flops(d, q, m, ITERATIONS) for d, q, m in parts)}
    dim = case["dim"]
    N, Nc = float((n * k + 1) ** dim), float((n // 2 * k + 1) ** dim)
    b = 2.0 * size * N  # one vector in, one out
    if kind in ("cg", "gmres"):
        f = _cg_flops(dim, k, n, ITERATIONS)
    elif kind == "adjoint":  # two solves to 1e-13; f, target, kappa in, u and the gradients out
        b, f = 8.0 * (4 * N + 2 * n ** dim), _cg_flops(dim, k, n, 2 * 2 * ITERATIONS)
    elif kind == "fmg":
        b = sum(8.0 * (q * k + 1) ** dim for q in _levels(n)) + 8.0 * N
        f = sum(_vcycle_flops(dim, k, q) + _operator_flops(dim, k, q) for q in _levels(n))
    elif kind == "vcycle":
        f = _vcycle_flops(dim, k, n)
    elif kind == "vmult":
        f = _operator_flops(dim, k, n)
    elif kind == "smooth":
        f = 2 * _sweep_flops(dim, k, n)
    elif kind == "transfer":
        b, f = size * (2 * N + 2 * Nc), 2 * 2.0 * (k + 1) * dim * N
    else:
        b = 8.0 * ((n * (k + 1)) ** dim + N)
        f = 2.0 * (k + 1) * dim * (n * (k + 1)) ** dim
    return {"bytes": b, "flops": f}


def tolerance(case):
    """About four times what the results are off the 64-bit restatement over these ranges."""
    kind = case["kind"]
    if kind in ("cg", "batch"):
        return {"rel": 2e-9}  # solved to a relative residual of 1e-10: up to 4e-10 off
    if kind == "adjoint":
        return {"rel": 1e-11}  # solved to 1e-13: up to 1e-12 off
    if kind == "gmres":
        return {"rel": 2e-6}  # the preconditioned residual reduced by 1e-9: up to 4e-7 off
    if "fp32" in (case.get("precision"), case.get("dtype")):
        # FP32 residuals of fine 2D meshes: 1.4e-5 at Q5 384^2; two sweeps: 9e-7 at 2D Q7 320^2;
        # one operator or transfer: 2e-7
        return {"rel": 6e-5 if kind in ("vcycle", "fmg") else 4e-6 if kind == "smooth" else 1e-6}
    return {"rel": 1e-12 if kind in ("vcycle", "fmg") else 1e-13}


# ---- the same results in 64-bit torch, from the definitions ------------------

def _apply_operator(M, S, v):
    """(S x M x .. + M x S x .. + ..) v."""
    dim = v.dim()
    return sum(_kron([S if a == d else M for a in range(dim)], v) for d in range(dim))


class _Direct:
    """A^{-1} on the interior by the eigenvectors of the global 1D pencil (S, M)."""

    def __init__(self, k, n, dim):
        M, S = (A[1:-1, 1:-1] for A in _mass_stiffness(k, n))
        C = torch.linalg.cholesky(M)
        K = torch.linalg.solve_triangular(C, torch.linalg.solve_triangular(C, S, upper=False).T, upper=False)
        lam, Q = torch.linalg.eigh(0.5 * (K + K.T))
        self.V = torch.linalg.solve_triangular(C.T, Q, upper=True)  # V^T M V = 1, V^T S V = lam
        self.den = sum(lam.reshape([-1 if a == d else 1 for a in range(dim)]) for d in range(dim))
        self.dim = dim

    def __call__(self, b):
        """x with zero boundary for the grid right-hand side b."""
        w = _kron([self.V.T.contiguous()] * self.dim, b[_inner(self.dim)].contiguous()) / self.den
        x = torch.zeros_like(b)
        x[_inner(self.dim)] = _kron([self.V] * self.dim, w)
        return x


class _Level:
    """Level operations of one mesh on grids (axes z, y, x)."""

    def __init__(self, dim, k, n):
        self.dim, self.k, self.n, self.n1 = dim, k, n, n * k + 1
        self.M, self.S = _mass_stiffness(k, n)

    def residual(self, x, b):
        return _zero_boundary(b - _apply_operator(self.M, self.S, x))

    def windows(self, v, colour):
        """The boxes of one colour's patches as a view: (patches.., box..)."""
        k = self.k
        for d in range(self.dim):  # bit 0 of the colour is the parity in x, the last axis
            off = ((colour >> (self.dim - 1 - d)) & 1) * k
            v = v.narrow(d, off, max(self.n1 - off, 0))
        if min(v.shape) < 2 * k + 1:
            return None
        for d in range(self.dim):
            v = v.unfold(d, 2 * k + 1, 2 * k)
        return v

    def sweep(self, x, b, reverse=False):
        """One coloured multiplicative vertex-patch sweep on x, in place."""
        dim, k = self.dim, self.k
        Mc, Sc = _cell_matrices(k)
        Mp, Sp = _gpu(_global(Mc / self.n, k, 2)), _gpu(_global(Sc * self.n, k, 2))
        solve = _patch_direct(Mp, Sp, dim)
        inner = (slice(None),) * dim + _inner(dim)
        colours = range(1 << dim)
        for c in reversed(colours) if reverse else colours:
            X = self.windows(x, c)
            if X is None:
                continue
            B = self.windows(b, c)
            shape = X.shape
            flat = X.reshape((-1,) + shape[dim:])
            r = B.reshape((-1,) + shape[dim:])[(slice(None),) + _inner(dim)] \
                - _batched_operator(Mp, Sp, flat)[(slice(None),) + _inner(dim)]
            new = flat[(slice(None),) + _inner(dim)] + solve(r)
            X[inner] = new.reshape(shape[:dim] + new.shape[1:])
        return x


def _batched(mats, v):
    for axis, A in enumerate(mats):
        v = _along(A, v, axis + 1)
    return v


def _batched_operator(M, S, v):
    dim = v.dim() - 1
    return sum(_batched([S if a == d else M for a in range(dim)], v) for d in range(dim))


def _patch_direct(Mp, Sp, dim):
    M, S = Mp[1:-1, 1:-1], Sp[1:-1, 1:-1]
    C = torch.linalg.cholesky(M)
    K = torch.linalg.solve_triangular(C, torch.linalg.solve_triangular(C, S, upper=False).T, upper=False)
    lam, Q = torch.linalg.eigh(0.5 * (K + K.T))
    V = torch.linalg.solve_triangular(C.T, Q, upper=True)
    den = sum(lam.reshape([-1 if a == d else 1 for a in range(dim)]) for d in range(dim))
    Vt = V.T.contiguous()
    return lambda r: _batched([V] * dim, _batched([Vt] * dim, r) / den)


def _interpolation(k, nc):
    """(2 nc k + 1, nc k + 1): nodal interpolation to the mesh of half the cell size."""
    t = _nodes(k)
    P = np.zeros((2 * nc * k + 1, nc * k + 1))
    for half in (0, 1):
        V, _ = _basis(k, 0.5 * (t + half))
        for c in range(nc):
            r = (2 * c + half) * k
            P[r:r + k + 1, c * k:c * k + k + 1] = V
    return _gpu(P)


def _prolongate(k, nc, coarse):
    return _zero_boundary(_kron([_interpolation(k, nc)] * coarse.dim(), coarse))


def _restrict(k, nc, fine):
    return _zero_boundary(_kron([_interpolation(k, nc).T.contiguous()] * fine.dim(), _zero_boundary(fine)))


def _vcycle(dim, k, levels, b, symmetric):
    """x from zero by one V-cycle with one sweep before and after (colours reversed after if symmetric)."""
    n = levels[-1]
    if len(levels) == 1:
        return _Direct(k, n, dim)(b)
    lev = _Level(dim, k, n)
    x = lev.sweep(torch.zeros_like(b), b)
    r = _restrict(k, levels[-2], lev.residual(x, b))
    x = x + _prolongate(k, levels[-2], _vcycle(dim, k, levels[:-1], r, symmetric))
    return lev.sweep(x, b, reverse=symmetric)


def _solve(dim, k, n, b):
    return _Direct(k, n, dim)(_grid(b, dim, n * k + 1)).reshape(-1)


class _Varying:
    """-div(kappa grad u) with one coefficient per cell, applied cell by cell."""

    def __init__(self, dim, k, n, kappa):
        self.dim, self.k, self.n = dim, k, n
        M, S = _cell_matrices(k)
        self.M, self.S = _gpu(M / n), _gpu(S * n)
        self.kappa = kappa.reshape((n,) * dim + (1,) * dim)

    def cells(self, v):
        for d in range(self.dim):
            v = v.unfold(d, self.k + 1, self.k)
        return v

    def local(self, v):
        """The unit-coefficient cell matrices on the cells of v."""
        w = self.cells(v)
        flat = w.reshape((-1,) + w.shape[self.dim:])
        return _batched_operator(self.M, self.S, flat).reshape(w.shape)

    def __call__(self, v):
        w = self.kappa * self.local(v)
        out = torch.zeros_like(v)
        k = self.k
        for colour in range(1 << self.dim):  # cells of one colour share no node
            par = [(colour >> d) & 1 for d in range(self.dim)]
            if min(self.n - p for p in par) < 1:
                continue
            o = out
            for d in range(self.dim):
                o = o.narrow(d, par[d] * k, out.shape[d] - par[d] * k)
            for d in range(self.dim):
                o = o.unfold(d, k + 1, 2 * k)
            o += w[tuple(slice(p, None, 2) for p in par)]
        return _zero_boundary(out)

    def solve(self, b):
        """CG preconditioned with the unit-coefficient solve, to rounding."""
        pre = _Direct(self.k, self.n, self.dim)
        b = _zero_boundary(b)
        x, r = torch.zeros_like(b), b.clone()
        z = pre(r)
        p, rz = z.clone(), (r * z).sum()
        for _ in range(400):
            q = self(p)
            a = rz / (p * q).sum()
            x += a * p
            r -= a * q
            if float(r.norm()) <= 3e-15 * float(b.norm()):
                break
            z = pre(r)
            new = (r * z).sum()
            p = z + (new / rz) * p
            rz = new
        return x


def exact(case, seed):
    kind, k, n = case["kind"], case["degree"], case["cells"]
    s = _inputs(case, seed)
    if kind == "batch":
        return [_solve(d, q, m, b) for (d, q, m), b in zip(_batch_systems(case), s["b"])]
    dim, n1 = case["dim"], n * k + 1
    if kind in ("cg", "gmres"):
        return _solve(dim, k, n, s["b"])
    if kind == "adjoint":
        A = _Varying(dim, k, n, s["kappa"])
        M, _ = _mass_stiffness(k, n)
        u = A.solve(_kron([M] * dim, _grid(s["f"], dim, n1)))
        lam = A.solve(u - _grid(s["target"], dim, n1))
        e = (A.cells(lam) * A.local(u)).flatten(dim).sum(-1)
        return u.reshape(-1), _kron([M] * dim, lam).reshape(-1), -e.reshape(-1)
    if kind == "fmg":
        levels = _levels(n)
        x = _solve(dim, k, levels[0], s["rhs"][0]).reshape((levels[0] * k + 1,) * dim)
        for l in range(1, len(levels)):
            q = levels[l]
            c = x + _grid(s["bnd"][l - 1], dim, levels[l - 1] * k + 1)
            x = _prolongate(k, levels[l - 1], c)
            r = _Level(dim, k, q).residual(x, _grid(s["rhs"][l], dim, q * k + 1))
            x = x + _vcycle(dim, k, levels[:l + 1], r, False)
        return (x + _grid(s["bnd"][-1], dim, n1)).reshape(-1)
    if kind == "vcycle":
        return _vcycle(dim, k, _levels(n), _grid(s["b"], dim, n1), False).reshape(-1)
    if kind == "vmult":
        x = _grid(s["x"].double(), dim, n1)
        M, S = _mass_stiffness(k, n)
        y = x.clone()
        y[_inner(dim)] = _apply_operator(M, S, x)[_inner(dim)]
        return y.reshape(-1)
    if kind == "smooth":
        lev, b = _Level(dim, k, n), _grid(s["b"].double(), dim, n1)
        x = lev.sweep(torch.zeros_like(b), b)
        return lev.sweep(x, b, reverse=True).reshape(-1)
    if kind == "transfer":
        fine = _grid(s["fine"].double(), dim, n1)
        coarse = _grid(s["coarse"].double(), dim, n // 2 * k + 1)
        return (_restrict(k, n // 2, fine).reshape(-1),
                _prolongate(k, n // 2, _zero_boundary(coarse)).reshape(-1))
    x, w = _gauss(k)
    V, _ = _basis(k, x)
    B = np.zeros((n1, n * (k + 1)))
    for c in range(n):
        B[c * k:c * k + k + 1, c * (k + 1):(c + 1) * (k + 1)] = (V * (w / n)[:, None]).T
    fq = s["fq"].reshape((n,) * dim + (k + 1,) * dim)
    order = [a for d in range(dim) for a in (d, dim + d)]
    grid = fq.permute(order).reshape((n * (k + 1),) * dim)
    return _zero_boundary(_kron([_gpu(B)] * dim, grid)).reshape(-1)
