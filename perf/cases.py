"""The calls a program built on this library makes, as measurable cases.

A finite-element program assembles K, eliminates its fixed DOFs, factors an
ILU(k) preconditioner and runs a Krylov solve; a program with its own assembly
hands K over and uses the SpMV and the preconditioner from its own solver; an
inverse problem adds the adjoint; a parameter study solves many small systems
as one batch.  Every case is one of these calls, through delfem_b200.lib and
delfem_b200.adjoint, on the meshes of delfem_b200.meshes with jittered nodes,
seeded coefficients and seeded loads.

A case is {"op", "kind", sizes, options}.  kind names the element: "poisson"
(1x1 blocks), "solid2d" (2x2), "solid3d" (3x3), "helmholtz" (complex).  n is
the grid side of the planar kinds and the ring count of the disk; nx, ny, nz
are the hexahedra of the box.
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

from delfem_b200 import adjoint, lib, meshes

NU = 0.3
LAM3, MYU3 = NU / ((1 + NU) * (1 - 2 * NU)), 1.0 / (2 * (1 + NU))
LAM2, MYU2 = NU / (1 - NU * NU), 1.0 / (2 * (1 + NU))  # plane stress, E = 1
WAVE = 2 * 3.1416 / 20
BLOCK = {"poisson": 1, "solid2d": 2, "solid3d": 3, "helmholtz": 1}
SOLVERS = {"pcg": lib.solve_pcg, "bicgstab": lib.solve_pbicgstab, "pcocg": lib.solve_pcocg,
           "pcg_mixed": lib.solve_pcg_mixed, "cg": lib.solve_cg}


def listed():
    return [
        # a small model's product inside a host-driven solver: one launch and its latency
        {"name": "spmv_2d_small", "op": "spmv", "kind": "poisson", "n": 32},
        # the product of the 1 M DOF cantilever: the whole matrix streams from HBM
        {"name": "spmv_3d", "op": "spmv", "kind": "solid3d", "nx": 200, "ny": 40, "nz": 40},
        # a preconditioner with fill, applied from a program's own solver
        {"name": "apply_3d_ilu1", "op": "apply", "kind": "solid3d", "nx": 100, "ny": 20, "nz": 20, "fill": 1,
         "patches": False},
        # a new K in the old pattern (a load or time step): numeric factor and first application
        {"name": "refactor_3d", "op": "refactor", "kind": "solid3d", "nx": 200, "ny": 40, "nz": 40, "fill": 0,
         "patches": True},
        # the same step's assembly: element matrices and residual at the current field, elimination
        {"name": "assemble_3d", "op": "assemble", "kind": "solid3d", "nx": 200, "ny": 40, "nz": 40},
        # 2-D diffusion solve: many short levels, everything in L2
        {"name": "pcg_2d", "op": "solve", "method": "pcg", "kind": "poisson", "n": 256, "tol": 1e-10,
         "patches": False},
        # the 1 M DOF cantilever solve, the largest of the ordinary solves
        {"name": "pcg_3d", "op": "solve", "method": "pcg", "kind": "solid3d", "nx": 200, "ny": 40, "nz": 40,
         "tol": 1e-10, "patches": True},
        # the mixed-precision solve (FP32 factor inside FP64 residual replacement) at half resolution
        {"name": "mixed_3d", "op": "solve", "method": "pcg_mixed", "kind": "solid3d", "nx": 100, "ny": 20, "nz": 20,
         "tol": 1e-8, "patches": True},
        # the unsymmetric solver on plane elasticity, an odd size
        {"name": "bicgstab_2d", "op": "solve", "method": "bicgstab", "kind": "solid2d", "n": 75, "tol": 1e-11,
         "patches": False},
        # complex symmetric Helmholtz solve with an absorbing boundary
        {"name": "cocg_disk", "op": "solve", "method": "pcocg", "kind": "helmholtz", "n": 64, "tol": 1e-10,
         "patches": False},
        # a parameter study: uneven small diffusion problems in one batched solve
        {"name": "batch_2d", "op": "batch", "kind": "poisson", "count": 96, "lo": 16, "hi": 192, "tol": 1e-10},
        # two steps of an inverse problem: assembly, factor, forward solve, adjoint solve, gradient
        {"name": "adjoint_2d", "op": "adjoint", "kind": "solid2d", "n": 64},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def size(kind, hi2, hi3):
        if kind == "solid3d":
            nx = log_int(15, hi3)
            return {"nx": nx, "ny": max(3, round(nx * rng.uniform(0.15, 0.25))),
                    "nz": max(3, round(nx * rng.uniform(0.15, 0.25)))}
        return {"n": log_int(12, 80) if kind == "helmholtz" else log_int(16, hi2)}

    op = rng.choice(["spmv", "spmv", "apply", "apply", "refactor", "assemble", "solve", "solve", "solve", "solve",
                     "batch", "adjoint"])
    if op == "batch":
        lo = log_int(8, 32)
        return {"op": op, "kind": "poisson", "count": rng.randint(16, 96), "lo": lo, "hi": log_int(lo + 8, 192),
                "tol": 1e-10}
    if op == "adjoint":
        return {"op": op, "kind": "solid2d", "n": log_int(12, 64)}
    if op == "solve":
        method, kind = rng.choice([("pcg", "poisson"), ("pcg", "solid2d"), ("pcg", "solid3d"), ("pcg_mixed", "poisson"),
                                   ("pcg_mixed", "solid3d"), ("bicgstab", "poisson"), ("bicgstab", "solid2d"),
                                   ("pcocg", "helmholtz"), ("cg", "poisson")])
        hi2 = 80 if kind == "solid2d" else 256
        # the FP32 factor holds elasticity above 1e-10
        tol = 1e-11 if method == "bicgstab" else 1e-8 if (method, kind) == ("pcg_mixed", "solid3d") else 1e-10
        return {"op": op, "method": method, "kind": kind, **size(kind, hi2, 110), "tol": tol,
                "patches": kind == "solid3d" and rng.random() < 0.5}
    kind = rng.choice(["poisson", "solid2d", "solid3d", "helmholtz"])
    case = {"op": op, "kind": kind, **size(kind, 400, 160)}
    if op in ("apply", "refactor"):
        case["fill"] = rng.choice([0, 0, 1])
        case["patches"] = kind == "solid3d" and rng.random() < 0.5
    return case


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=32)
def _mesh(kind, n, nx, ny, nz):
    if kind == "solid3d":
        return meshes.box_tet(nx, ny, nz)
    if kind == "helmholtz":
        return meshes.unit_disk_tri(n, numbering="bands")
    return meshes.unit_square_tri(n, bnd="left" if kind == "solid2d" else "all")


@functools.lru_cache(maxsize=8)
def _batch_mesh(count, lo, hi):
    return meshes.concat([meshes.unit_square_tri(int(k)) for k in meshes.batch_sizes(count, lo, hi, 3)])


def _case_mesh(case):
    if case["op"] == "batch":
        return _batch_mesh(case["count"], case["lo"], case["hi"])[0]
    return _mesh(case["kind"], case.get("n", 0), case.get("nx", 0), case.get("ny", 0), case.get("nz", 0))


def _spacing(case):
    """Node spacing along each axis (a column per node where it differs)."""
    if case["op"] == "batch":
        off = _batch_mesh(case["count"], case["lo"], case["hi"])[1]
        side = np.sqrt(np.diff(off)) - 1
        return np.repeat(1.0 / side, np.diff(off))[:, None]
    if case["kind"] == "solid3d":
        return np.array([1.0 / case["nx"], 0.2 / case["ny"], 0.2 / case["nz"]])
    return 1.0 / case["n"]


class _Inputs:
    """Jittered mesh, coefficients and loads of one seed, the same for prepare() and exact()."""

    def __init__(self, case, seed):
        m = _case_mesh(case)
        rng = np.random.default_rng(seed)
        self.kind, self.b = case["kind"], BLOCK[case["kind"]]
        self.xw = 2 if self.kind == "helmholtz" else self.b
        h = _spacing(case)
        self.coord = m.coord + 0.1 * h * rng.uniform(-1.0, 1.0, m.coord.shape)
        self.elem, self.bnd, self.nnode = m.elem, m.bnd, m.nnode
        self.fixed = np.unique(m.bnd.ravel()) if self.kind != "helmholtz" else np.zeros(0, np.int64)
        self.coef = rng.lognormal(0.0, 0.5, m.elem.shape[0]) if self.kind in ("poisson", "solid2d") else None
        scale = np.prod(np.broadcast_to(h, m.coord.shape), axis=1)[:, None]
        self.load = (scale * rng.standard_normal((m.nnode, self.xw))).ravel()
        if self.kind == "helmholtz":
            self.load = self.load + meshes.gaussian_source_load(m).ravel()
        self.u = 0.01 * rng.standard_normal(m.nnode * self.xw) if case["op"] == "assemble" else None
        self.flags = np.zeros((m.nnode, self.b), np.int32)
        self.flags[self.fixed] = 1


def _cuda(a):
    return None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda()


@functools.lru_cache(maxsize=1)
def _context():
    return lib.Context(0)


class _State:
    pass


class _View:
    """n doubles of the matrix A's device memory; a tensor made of it keeps A alive."""

    def __init__(self, A, ptr, n):
        self.A = A
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": (n,), "typestr": "<f8", "version": 3}


def _values(A):
    """The matrix's device values as tensors."""
    d, o = ctypes.c_void_p(), ctypes.c_void_p()
    lib.check(lib.lib().dfm_mat_values_device(A.h, ctypes.byref(d), ctypes.byref(o)))
    return (torch.as_tensor(_View(A, d.value, A.N * A.vw), device="cuda"),
            torch.as_tensor(_View(A, o.value, A.ncrs * A.vw), device="cuda"))


def _assemble(s):
    if s.kind == "poisson":
        s.G.assemble_poisson(s.A, 1.0, 1.0, s.rhs, coef=s.coef, u=s.u, load=s.load)
    elif s.kind == "solid2d":
        s.G.assemble_solid2d(s.A, LAM2, MYU2, 1.0, 0.0, -1.0, s.rhs, coef=s.coef, u=s.u, load=s.load)
    elif s.kind == "solid3d":
        s.G.assemble_solid3d(s.A, LAM3, MYU3, 1.0, 0.0, 0.0, -1.0, s.rhs, u=s.u, load=s.load)
    else:
        s.G.assemble_helmholtz(s.A, WAVE, s.rhs, u=s.u, load=s.load)
        return
    lib.apply_dirichlet(s.A, s.flags, s.rhs)


def _spmv_values(case, seed, nnode, ncrs):
    """Block values and vectors of the SpMV cases, on the device."""
    kind = case["kind"]
    vw, xw = (2, 2) if kind == "helmholtz" else (BLOCK[kind] ** 2, BLOCK[kind])
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda n: torch.randn(n, dtype=torch.float64, device="cuda", generator=g)  # noqa: E731
    return r(nnode * vw), r(ncrs * vw), r(nnode * xw), r(nnode * xw)


def prepare(case, seed):
    ctx = _context()
    s = _State()
    s.case, s.kind = case, case["kind"]
    op = case["op"]
    if op == "adjoint":
        I = _Inputs(case, seed)
        n = case["n"]
        m = _case_mesh(case)
        s.problem = adjoint.PlaneStressProblem(ctx, I.coord, I.elem, I.fixed, meshes.right_edge_traction(m, n), LAM2,
                                               MYU2, tol=1e-12)
        s.theta, s.idx, s.target = (_cuda(a) for a in _adjoint_inputs(case, seed))
        return s
    if op == "spmv":
        m = _case_mesh(case)
        G = lib.Mesh(ctx, m.coord, m.elem)
        rp, ci = G.pattern()
        s.A = lib.Matrix(ctx, rp, ci, BLOCK[s.kind], lib.COMPLEX if s.kind == "helmholtz" else lib.REAL)
        d, o, s.x, s.y = _spmv_values(case, seed, m.nnode, ci.size)
        s.A.set_values(d, o)
        return s
    I = _Inputs(case, seed)
    cplx = s.kind == "helmholtz"
    s.G = lib.Mesh(ctx, I.coord, I.elem, I.bnd if cplx else None)
    rp, ci = s.G.pattern()
    s.A = lib.Matrix(ctx, rp, ci, I.b, lib.COMPLEX if cplx else lib.REAL)
    s.coef, s.u, s.load, s.flags = _cuda(I.coef), _cuda(I.u), _cuda(I.load), _cuda(I.flags.ravel())
    s.rhs = torch.empty(I.nnode * I.xw, dtype=torch.float64, device="cuda")
    if op == "assemble":
        s.values = _values(s.A)
        return s
    _assemble(s)
    s.r, s.x = s.rhs.clone(), torch.zeros_like(s.rhs)
    if case.get("method") == "cg":
        return s
    s.M = lib.ILU(s.A, case.get("fill", 0))
    if case.get("patches"):
        s.M.set_sweep_partition(*lib.sweep_partition_patches(
            I.coord, torch.cuda.get_device_properties(0).multi_processor_count))
    s.M.factor()
    if op == "batch":
        s.B = lib.Batch(s.M, _batch_mesh(case["count"], case["lo"], case["hi"])[1].astype(np.uint32))
    return s


def _adjoint_inputs(case, seed):
    """Two moduli fields, the observed DOFs and their target values."""
    m = _case_mesh(case)
    rng = np.random.default_rng([seed, 1])
    theta = rng.lognormal(0.0, 0.5, (2, m.elem.shape[0]))
    obs = np.sort(rng.choice(m.nnode, size=min(256, m.nnode), replace=False))
    idx = np.concatenate([2 * obs, 2 * obs + 1])
    return theta, idx, rng.standard_normal(idx.size)


def run(s):
    op = s.case["op"]
    if op == "spmv":
        return s.A.spmv(1.0, s.x, 0.0, s.y)
    if op == "assemble":
        _assemble(s)
        return {"rhs": s.rhs, "diag": s.values[0], "off": s.values[1]}
    if op == "apply":
        return s.M.apply(s.rhs, s.x)
    if op == "refactor":
        s.M.factor()
        return s.M.apply(s.rhs, s.x)
    if op == "batch":
        s.B.solve(s.rhs, s.x, tol=s.case["tol"], maxit=20000)
        return s.x
    if op == "solve":
        s.r.copy_(s.rhs)
        solver = SOLVERS[s.case["method"]]
        if s.case["method"] == "cg":
            solver(s.A, s.r, s.x, tol=s.case["tol"], maxit=20000, allow=(lib.OK,))
        else:
            solver(s.A, s.M, s.r, s.x, tol=s.case["tol"], maxit=20000, allow=(lib.OK,))
        return s.x
    out = []
    for k in range(2):  # two steps: K(theta) is assembled and factored anew in each
        theta = s.theta[k].clone().requires_grad_(True)
        u = adjoint.elastic_solve(theta, s.problem)
        loss = 0.5 * torch.sum((u[s.idx] - s.target) ** 2)
        loss.backward()
        out += [u.detach(), theta.grad]
    return out


# -------------------------------------------------------------------- work
def work(case):
    m = _case_mesh(case)
    n, ne = m.nnode, m.elem.shape[0]
    b = BLOCK[case["kind"]]
    cplx = case["kind"] == "helmholtz"
    bb, xw = (2, 2) if cplx else (b * b, b)
    # blocks off the diagonal: two per edge; a triangulated disc has n + ne - 1 edges
    if case["kind"] == "solid3d":
        x, y, z = case["nx"], case["ny"], case["nz"]
        axis = x * (y + 1) * (z + 1) + (x + 1) * y * (z + 1) + (x + 1) * (y + 1) * z
        face = x * y * (z + 1) + x * (y + 1) * z + (x + 1) * y * z
        ncrs = 2 * (axis + face + x * y * z)
    else:
        parts = case["count"] if case["op"] == "batch" else 1
        ncrs = 2 * (n + ne - parts)
    flop = 8 if cplx else 2 * b * b
    matrix = 8 * bb * (n + ncrs) + 4 * (ncrs + n + 1)
    vec = 8 * n * xw
    op = case["op"]
    if op == "spmv":
        return {"bytes": matrix + 2 * vec, "flops": flop * (n + ncrs)}
    if op == "assemble":
        elem = ne * m.elem.shape[1] * 4 + m.coord.size * 8
        return {"bytes": matrix + elem + 3 * vec + 4 * n * b, "flops": 40 * ne * m.elem.shape[1] ** 2 * bb / 4}
    if op == "apply":
        return {"bytes": matrix + 2 * vec, "flops": flop * (n + ncrs)}
    if op == "refactor":  # K read, factor written and read by the sweeps; about 3 updates per lower block
        return {"bytes": 3 * matrix + 2 * vec, "flops": flop * (n + ncrs) + 3 * 2 * b ** 3 * ncrs / 2}
    if op == "adjoint":  # per step: K written and read by two solves, the gradient written
        return {"bytes": 2 * (3 * matrix + 6 * vec + 16 * ne), "flops": 2 * 4 * flop * (n + ncrs)}
    fine = 1 if case.get("method") == "cg" else 2  # K and its factor, each once
    return {"bytes": fine * matrix + 2 * vec, "flops": fine * flop * (n + ncrs)}


# ------------------------------------------------------------------- exact
class _Plain:
    """K (block values at sorted (row, col) keys) and the residual, assembled in plain torch."""

    def __init__(self, I, coef):
        dev = "cuda"
        kind = I.kind
        N, e = I.nnode, torch.from_numpy(I.elem.astype(np.int64)).to(dev)
        p = torch.from_numpy(I.coord).to(dev)[e]
        nno, ndim = e.shape[1], p.shape[2]
        # gradients of the P1 shape functions from the edge matrix
        J = p[:, 1:] - p[:, :1]
        g = torch.linalg.inv(J).transpose(1, 2)
        G = torch.cat([-g.sum(1, keepdim=True), g], 1)
        vol = torch.linalg.det(J) / (2.0 if ndim == 2 else 6.0)
        dd = torch.einsum("eai,eci->eac", G, G)
        if coef is not None:
            coef = torch.as_tensor(coef, device=dev)
        dt = torch.complex128 if kind == "helmholtz" else torch.float64
        b = I.b
        if kind == "poisson":
            K = ((coef * vol)[:, None, None] * dd)[..., None, None]
        elif kind == "helmholtz":
            k = 2 * 3.1416 / WAVE
            mass = (torch.ones(3, 3, device=dev, dtype=torch.float64) + torch.eye(3, device=dev)) / 12.0
            K = (vol[:, None, None] * (dd - k * k * mass))[..., None, None].to(dt)
        else:
            lam, myu = (LAM3, MYU3) if ndim == 3 else (LAM2, MYU2)
            K = lam * torch.einsum("eai,ecj->eacij", G, G) + myu * torch.einsum("eaj,eci->eacij", G, G)
            K = K + myu * dd[..., None, None] * torch.eye(b, device=dev, dtype=torch.float64)
            K = K * (vol if coef is None else vol * coef)[:, None, None, None, None]
        key = (e[:, :, None] * N + e[:, None, :]).reshape(-1)
        val = K.reshape(-1, b, b)
        if kind == "helmholtz":
            q = torch.from_numpy(I.bnd.astype(np.int64)).to(dev)
            c = torch.from_numpy(I.coord).to(dev)[q]
            ln = torch.linalg.norm(c[:, 0] - c[:, 1], dim=1)
            t1, t2 = 1j * k / 6.0 * ln, 1j * (-1.0 / (2.0 * ln * k))
            same = torch.eye(2, device=dev, dtype=torch.bool)
            S = torch.where(same, (2 * t1 + t2)[:, None, None], (t1 - t2)[:, None, None])
            key = torch.cat([key, (q[:, :, None] * N + q[:, None, :]).reshape(-1)])
            val = torch.cat([val, S.reshape(-1, 1, 1)])
        self.N, self.b = N, b
        self.key, inv = torch.unique(key, return_inverse=True)
        self.val = torch.zeros(self.key.numel(), b, b, device=dev, dtype=dt).index_add_(0, inv, val.to(dt))
        self.row, self.col = self.key // N, self.key % N
        # residual: body force, nodal load, minus K u
        f = torch.zeros(N, b, device=dev, dtype=dt)
        if kind == "poisson":
            body = torch.ones(1, device=dev, dtype=torch.float64)
        elif kind == "solid2d":
            body = torch.tensor([0.0, -1.0], device=dev, dtype=torch.float64)
        elif kind == "solid3d":
            body = torch.tensor([0.0, 0.0, -1.0], device=dev, dtype=torch.float64)
        else:
            body = torch.zeros(1, device=dev, dtype=torch.float64)
        f.index_add_(0, e.reshape(-1), ((vol / nno)[:, None, None] * body).expand(-1, nno, -1).reshape(-1, b).to(dt))
        if I.u is not None:
            f -= self.mul(self.vec(torch.from_numpy(I.u).to(dev))).reshape(N, b)
        self.rhs = f.reshape(-1) + self.vec(torch.from_numpy(I.load).to(dev))
        self.fixed = torch.from_numpy(I.flags.ravel() != 0).to(dev)

    def vec(self, x):
        return torch.view_as_complex(x.reshape(-1, 2)) if self.val.is_complex() else x

    def flat(self, x):
        return torch.view_as_real(x).reshape(-1) if x.is_complex() else x.reshape(-1)

    def mul(self, x):
        y = torch.einsum("sij,sj->si", self.val, x.reshape(self.N, self.b)[self.col])
        return torch.zeros(self.N, self.b, device=x.device, dtype=y.dtype).index_add_(0, self.row, y).reshape(-1)

    def eliminate(self):
        if self.val.is_complex():
            return self
        fx = self.fixed.reshape(self.N, self.b)
        one = fx[self.row][:, :, None] & (self.row == self.col)[:, None, None] \
            & torch.eye(self.b, device=fx.device, dtype=torch.bool)
        self.val[fx[self.row][:, :, None] | fx[self.col][:, None, :]] = 0.0
        self.val[one] = 1.0
        self.rhs = torch.where(self.fixed, torch.zeros_like(self.rhs), self.rhs)
        return self

    def csr(self):
        b, N = self.b, self.N
        k = torch.arange(b, device=self.key.device)
        r = (self.row[:, None, None] * b + k[None, :, None]).expand(-1, b, b).reshape(-1)
        c = (self.col[:, None, None] * b + k[None, None, :]).expand(-1, b, b).reshape(-1)
        return torch.sparse_coo_tensor(torch.stack([r, c]), self.val.reshape(-1), (N * b, N * b)).coalesce() \
            .to_sparse_csr()

    def solve(self, rhs, most=20000):
        """Dense for the small and the complex systems, else conjugate gradients to rounding."""
        n = self.N * self.b
        if n <= 4000 or self.val.is_complex():
            return torch.linalg.solve(self.csr().to_dense(), rhs)
        K = self.csr()
        d = 1.0 / self.flat(torch.diagonal(self.val[self.row == self.col], dim1=1, dim2=2))
        x = torch.zeros_like(rhs)
        for _ in range(2):  # the second round removes the drift of the first one's residual
            r = rhs - K @ x
            z = d * r
            p, rz = z.clone(), torch.dot(r, z)
            stop = 1e-15 * float(torch.linalg.norm(rhs))
            for it in range(most):
                q = K @ p
                a = rz / torch.dot(p, q)
                x += a * p
                r -= a * q
                if it % 50 == 49 and float(torch.linalg.norm(r)) < stop:
                    break
                z = d * r
                new = torch.dot(r, z)
                p = z + (new / rz) * p
                rz = new
        return x


def exact(case, seed):
    op = case["op"]
    if op in ("apply", "refactor"):  # defined by the factor's own elimination order: no closed value
        return None
    if op == "spmv":
        m = _case_mesh(case)
        N = m.nnode
        e = torch.from_numpy(m.elem.astype(np.int64)).cuda()
        key = torch.unique((e[:, :, None] * N + e[:, None, :]).reshape(-1))
        row, col = key // N, key % N
        row, col = row[row != col], col[row != col]
        d, o, x, _ = _spmv_values(case, seed, N, row.numel())
        if case["kind"] == "helmholtz":
            d, o, x = (torch.view_as_complex(t.reshape(-1, 2)) for t in (d, o, x))
        b = BLOCK[case["kind"]]
        X = x.reshape(N, b)
        y = torch.einsum("nij,nj->ni", d.reshape(N, b, b), X)
        y.index_add_(0, row, torch.einsum("sij,sj->si", o.reshape(-1, b, b), X[col]))
        return torch.view_as_real(y).reshape(-1) if y.is_complex() else y.reshape(-1)
    if case["kind"] == "helmholtz" and op == "solve" and case["n"] > 72:
        return None
    I = _Inputs(case, seed)
    if op == "adjoint":
        theta, idx, target = _adjoint_inputs(case, seed)
        m = _case_mesh(case)
        I.load = meshes.right_edge_traction(m, case["n"]).ravel()
        idx, target = torch.from_numpy(idx).cuda(), torch.from_numpy(target).cuda()
        out = []
        for k in range(2):
            P = _Plain(I, theta[k])
            # the problem has no body force: the load alone, on the free DOFs
            f = torch.where(P.fixed, 0.0, torch.from_numpy(I.load).cuda())
            P.eliminate()
            u = P.solve(f)
            gu = torch.zeros_like(u).index_put_((idx,), u[idx] - target)
            lam = P.solve(torch.where(P.fixed, torch.zeros_like(gu), gu))
            e = torch.from_numpy(I.elem.astype(np.int64)).cuda()
            p = torch.from_numpy(I.coord).cuda()[e]
            J = p[:, 1:] - p[:, :1]
            g = torch.linalg.inv(J).transpose(1, 2)
            G = torch.cat([-g.sum(1, keepdim=True), g], 1)
            vol = torch.linalg.det(J) / 2.0
            du = torch.einsum("eai,eaj->eij", G, u.reshape(-1, 2)[e])   # d u_j / d x_i
            dl = torch.einsum("eai,eaj->eij", G, lam.reshape(-1, 2)[e])
            tr = lambda t: t.diagonal(dim1=1, dim2=2).sum(1)  # noqa: E731
            en = LAM2 * tr(du) * tr(dl) + MYU2 * ((du * dl).sum((1, 2)) + (du * dl.transpose(1, 2)).sum((1, 2)))
            out += [u, -vol * en]
        return out
    P = _Plain(I, I.coef)
    P.eliminate()
    if op == "assemble":
        on = P.row == P.col
        return {"rhs": P.flat(P.rhs), "diag": P.flat(P.val[on]), "off": P.flat(P.val[~on])}
    return P.flat(P.solve(P.rhs))
