"""Performance cases of the assemble + sparse-Krylov framework.

Each case is one piece of work that a program using the package does, through
the package's public entry points, on the generators the package ships (2D
perturbed triangles, 3D Kuhn tetrahedra).  A case is a dict of plain values:

  op "vector"    the DistributedVector operations of a hand-written solver
  op "spmv"      DistributedMatrix.imul
  op "assemble"  value-only re-assembly into a resident pattern and A u (the
                 residual evaluation of an outer loop)
  op "corrected" cell gradients, the Corrected laplacian's assembly and A u
  op "factor"    value-only refactorisation and one preconditioner apply
  op "steady"    mesh in hand: assembly, factorisation and a complete solve
  op "step"      one implicit Euler step on resident objects: re-assembly,
                 refactorisation, solve from the previous solution
  op "batch"     many independent problems solved as one block-diagonal system

`dim` 2: side^2 squares of two triangles; 3: side^3 hexahedra of six
tetrahedra.  `order`: "natural" row order, "boxes" (box-colour ordering applied
in the matrix's numbering) or "permuted" (the permuted system).
"""
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "finite-volumes-rs_b200"))

import fvb200 as fv  # noqa: E402
from fvb200.batch import BatchCG, MeshBatch  # noqa: E402

JITTER = {2: 0.2, 3: 0.15}
SIGMA = {2: 1.0, 3: 0.5}
VELOCITY = (1.0, 0.5, 0.25)
DT = {2: 1e-3, 3: 2e-3}


def listed():
    return [
        # the smallest call: vector operations of a solver written on the package's vectors
        {"name": "vector_10k", "op": "vector", "n": 10007},
        # the smallest complete solve (2,048 cells, the smallest problem of the batched workload), as the smoke run does it
        {"name": "steady_square32", "op": "steady", "dim": 2, "side": 32, "order": "natural", "precond": "ic", "tol": 1e-12},
        # a small 3D convection-diffusion solve (24,576 cells)
        {"name": "steady_cube16", "op": "steady", "dim": 3, "side": 16, "order": "natural", "precond": "ilu", "tol": 1e-8},
        # the plain 2D diffusion workload (131,072 cells) in the reference's own row order
        {"name": "steady_square256", "op": "steady", "dim": 2, "side": 256, "order": "natural", "precond": "ic", "tol": 1e-8},
        # a time loop on a mid-size 2D mesh (65,522 cells), box order as the permuted system
        {"name": "step_square181", "op": "step", "dim": 2, "side": 181, "order": "permuted", "precond": "ic", "tol": 1e-8},
        # the time loop of the large 3D workload (5.3M cells)
        {"name": "step_cube96", "op": "step", "dim": 3, "side": 96, "order": "permuted", "precond": "ilu", "tol": 1e-8},
        # matrix-vector product of the large 3D matrix
        {"name": "spmv_cube96", "op": "spmv", "dim": 3, "side": 96},
        # re-assembly of the large 3D convection-diffusion operator
        {"name": "assemble_cube96", "op": "assemble", "dim": 3, "side": 96},
        # non-orthogonal correction on an odd-sized 2D mesh (263,538 cells)
        {"name": "corrected_square363", "op": "corrected", "dim": 2, "side": 363},
        # refactorisation and apply of ILU(0) in natural order (1.57M cells)
        {"name": "factor_cube64", "op": "factor", "dim": 3, "side": 64, "order": "natural", "precond": "ilu"},
        # batched 2D diffusion solves, FP64
        {"name": "batch_square_fp64", "op": "batch", "dim": 2, "side": 128, "problems": 24, "precision": "fp64", "tol": 1e-8},
        # batched 3D convection-diffusion solves, FP32 inside FP64 refinement
        {"name": "batch_cube_mixed", "op": "batch", "dim": 3, "side": 24, "problems": 10, "precision": "mixed", "tol": 1e-10},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    op = rng.choice(["vector", "spmv", "assemble", "corrected", "factor", "steady", "steady", "step", "step", "batch"])
    if op == "vector":
        return {"op": op, "n": _log_int(rng, 10, 8_000_000)}
    dim = rng.choice([2, 3])
    if op == "spmv":
        return {"op": op, "dim": dim, "side": _log_int(rng, 8, 1024) if dim == 2 else _log_int(rng, 4, 96)}
    if op == "assemble":
        return {"op": op, "dim": dim, "side": _log_int(rng, 8, 1024) if dim == 2 else _log_int(rng, 4, 96)}
    if op == "corrected":
        return {"op": op, "dim": dim, "side": _log_int(rng, 8, 700) if dim == 2 else _log_int(rng, 4, 56)}
    if op == "factor":
        return {"op": op, "dim": dim, "side": _log_int(rng, 8, 700) if dim == 2 else _log_int(rng, 4, 72),
                "order": rng.choice(["natural", "boxes", "permuted"]), "precond": "ic" if dim == 2 else "ilu"}
    if op == "steady":
        return {"op": op, "dim": dim, "side": _log_int(rng, 8, 230) if dim == 2 else _log_int(rng, 4, 40),
                "order": rng.choice(["natural", "natural", "boxes"]),
                "precond": rng.choice(["ic" if dim == 2 else "ilu"] * 4 + ["diag"]),
                "tol": rng.choice([1e-8, 1e-12]) if dim == 2 else 1e-8}
    if op == "step":
        return {"op": op, "dim": dim, "side": _log_int(rng, 8, 500) if dim == 2 else _log_int(rng, 4, 90),
                "order": rng.choice(["natural", "boxes", "permuted"]), "precond": "ic" if dim == 2 else "ilu", "tol": 1e-8}
    precision = rng.choice(["fp64", "mixed"])
    return {"op": op, "dim": dim, "side": _log_int(rng, 24, 128) if dim == 2 else _log_int(rng, 8, 24),
            "problems": rng.randint(2, 24), "precision": precision, "tol": 1e-8 if precision == "fp64" else 1e-10}


# ------------------------------------------------------------------ inputs
def _cuda(a):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda")


def _mesh(dim, side, seed):
    make = fv.Mesh.square if dim == 2 else fv.Mesh.cube
    return make(side, JITTER[dim], seed, on_device=True)


def _fields(m, dim, side, seed, sigma=None):
    """Face diffusivity, face flux (3D) and cell source of the generators' workloads."""
    sigma = SIGMA[dim] if sigma is None else sigma
    if dim == 2:
        kf, _, sc = m.fields(seed, 1.0, sigma, source_const=1.0)
        return kf, None, sc
    kappa0 = float(np.linalg.norm(VELOCITY)) / side / 3.0
    return m.fields(seed, kappa0, sigma, velocity=VELOCITY, source_uniform=True)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(n, seed):
    return torch.randn(n, dtype=torch.float64, device="cuda", generator=_generator(seed))


def _expression(s, previous=None):
    e = -fv.laplacian(s.get("scheme") or fv.Orthogonal(), s["kappa"])
    if s["flux"] is not None:
        e = fv.convection(fv.Upwind(s["flux"]), s["flux"]) + e
    if previous is not None:
        e = fv.time(fv.Euler(previous, s["dt"])) + e
    return e - fv.source(s["source"])


def _problem(case, seed):
    """One mesh with its fields resident on the GPU, and Dirichlet 0 on the boundary."""
    dim, side = case["dim"], case["side"]
    m = _mesh(dim, side, seed)
    kf, fl, sc = _fields(m, dim, side, seed)
    zero = torch.zeros(m.n_boundary_faces, dtype=torch.float64, device="cuda")
    return {"mesh": m, "kappa": _cuda(kf), "flux": None if fl is None else _cuda(fl), "source": _cuda(sc),
            "bc": (zero, zero.clone()), "dt": DT[dim]}


def _bump(m):
    """A smooth initial field: a Gaussian in the middle of the domain."""
    d2 = ((m.cell_center - 0.5) ** 2).sum(axis=1)
    return _cuda(np.exp(-d2 / 0.02))


def _factor(A, case):
    if case["precond"] == "diag":
        return fv.DiagonalPreconditioner.from_matrix(A)
    cls = fv.IncompleteCholesky if case["precond"] == "ic" else fv.IncompleteLowerUpper
    return cls.from_matrix(A, 0, ordering="boxes" if case["order"] == "boxes" else None)


def _krylov(case):
    return fv.conjugate_gradient if case["dim"] == 2 else fv.bi_conjugate_gradient_stab


def _sides(case):
    """Problem sizes of a batch: from a quarter of the largest side up to it."""
    k, n = case["problems"], case["side"]
    return [max(4, int(round(n * 4.0 ** (-i / max(1, k - 1))))) for i in range(k)]


def _batch_problem(case, seed):
    dim = case["dim"]
    sides = _sides(case)
    meshes = [_mesh(dim, n, seed * 1000 + k) for k, n in enumerate(sides)]
    fields = [_fields(m, dim, n, seed * 1000 + k, sigma=(0.5 + 0.75 * ((k * 0.37) % 1.0)) if dim == 2 else None)
              for k, (m, n) in enumerate(zip(meshes, sides))]
    mb = MeshBatch(meshes)
    zero = torch.zeros(mb.n_boundary_faces, dtype=torch.float64, device="cuda")
    return {"mesh": mb, "kappa": _cuda(mb.face_field([f[0] for f in fields])),
            "flux": None if dim == 2 else _cuda(mb.face_field([f[1] for f in fields])),
            "source": _cuda(mb.cell_field([f[2] for f in fields])), "bc": (zero, zero.clone()), "dt": DT[dim]}


def prepare(case, seed):
    op = case["op"]
    if op == "vector":
        n = case["n"]
        s = {"u": fv.DistributedVector(_randn(n, seed)), "v": fv.DistributedVector(_randn(n, seed + 1)),
             "w": fv.DistributedVector.from_size(n)}
        return dict(s, case=case)
    s = _batch_problem(case, seed) if op == "batch" else _problem(case, seed)
    s["case"] = case
    m = s["mesh"]
    n = m.n_cells
    if op in ("spmv", "assemble", "corrected"):
        s["u"] = fv.DistributedVector(_randn(n, seed))
        s["y"] = fv.DistributedVector.from_size(n)
    if op == "corrected":
        s["field"] = fv.DistributedVector(_bump(m) + 0.1 * _randn(n, seed + 2))
        s["g"] = fv.DistributedVector.from_size(n * m.dim)
        s["scheme"] = None
    if op == "steady":
        m.device()
        return s
    s["previous"] = fv.DistributedVector(_bump(m)) if op == "step" else None
    if op == "step":
        s["x"] = fv.DistributedVector.from_size(n)
    s["A"], s["b"] = fv.assemble(_expression(s, s["previous"].data if op == "step" else None), s["bc"], m)
    if op == "factor":
        s["r"] = fv.DistributedVector(_randn(n, seed))
        s["z"] = fv.DistributedVector.from_size(n)
    if op in ("factor", "step"):
        if case["order"] == "permuted":
            s["S"] = fv.PermutedSystem(s["A"], case["precond"])
        else:
            s["P"] = _factor(s["A"], case)
    if op == "batch":
        cls = fv.IncompleteCholesky if case["dim"] == 2 else fv.IncompleteLowerUpper
        s["P"] = cls.from_matrix(s["A"], 0, ordering="boxes", offsets=m.cell_offsets)
        s["B"] = BatchCG(s["A"], m.cell_offsets)
        s["x"] = fv.DistributedVector.from_size(n)
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    case = s["case"]
    op = case["op"]
    if op == "vector":
        u, v, w = s["u"], s["v"], s["w"]
        w.set(u)
        w += v
        w *= 0.5
        return {"w": w.data, "dot": w.dot(v), "sum": w.sum()}
    m = s["mesh"]
    if op == "spmv":
        s["A"].imul(s["y"], s["u"])
        return s["y"].data
    if op == "assemble":
        _, b = fv.assemble(_expression(s), s["bc"], m, lhs=s["A"])
        s["A"].imul(s["y"], s["u"])
        return {"b": b.data, "Au": s["y"].data}
    if op == "corrected":
        fv.compute_gradients(s["g"], s["field"], s["bc"], m)
        s["scheme"] = fv.Corrected(s["g"], 1.0)
        _, b = fv.assemble(_expression(s), s["bc"], m, lhs=s["A"])
        s["A"].imul(s["y"], s["u"])
        return {"g": s["g"].data, "b": b.data, "Au": s["y"].data}
    if op == "factor":
        if case["order"] == "permuted":
            s["S"].refresh()
            s["S"].P.precondition(s["z"], s["r"])
        else:
            s["P"].refactor()
            s["P"].precondition(s["z"], s["r"])
        return s["z"].data
    if op == "steady":
        A, b = fv.assemble(_expression(s), s["bc"], m)
        P = _factor(A, case)
        x = fv.DistributedVector.from_size(m.n_cells)
        _krylov(case)(x, A, b, P, None, fv.LinearSolverOptions(case["tol"], case["tol"], 10000))
        return {"b": b.data, "x": x.data}
    if op == "step":
        _, b = fv.assemble(_expression(s, s["previous"].data), s["bc"], m, lhs=s["A"])
        x = s["x"]
        x.set(s["previous"])
        options = fv.LinearSolverOptions(case["tol"], case["tol"], 10000)
        if case["order"] == "permuted":
            s["S"].refresh()
            s["S"].solve(x, b, options)
        else:
            s["P"].refactor()
            _krylov(case)(x, s["A"], b, s["P"], None, options)
        return {"b": b.data, "x": x.data}
    s["B"].solve(s["P"], s["b"], s["x"], precision=case["precision"], relative_tolerance=case["tol"],
                 absolute_tolerance=case["tol"], max_iterations=10000, outer_tolerance=case["tol"],
                 solver="cg" if case["dim"] == 2 else "bicgstab")
    return s["x"].data


# ------------------------------------------------------------------ work
def _counts(dim, side):
    """(cells, faces, boundary faces, CSR entries) of a generated mesh."""
    if dim == 2:
        n, fi, fb = 2 * side * side, 3 * side * side - 2 * side, 4 * side
    else:
        n, fi, fb = 6 * side ** 3, 12 * side ** 3 - 6 * side ** 2, 12 * side ** 2
    return n, fi + fb, fb, n + 2 * fi


def work(case):
    """Bytes and operations of one pass: every input once, every output once
    per kernel-independent stage; an iteration's passes over the matrix, the
    factors and the Krylov vectors, with the iteration counts these problems
    need (about 2.5 per side for CG + IC(0), 1.5 for BiCGStab + ILU(0), tens
    for a time step)."""
    op = case["op"]
    if op == "vector":
        return {"bytes": 8.0 * 5 * case["n"], "flops": 5.0 * case["n"]}
    total = {"bytes": 0.0, "flops": 0.0}
    sides = _sides(case) if op == "batch" else [case["side"]]
    for side in sides:
        n, f, fb, nnz = _counts(case["dim"], side)
        spmv = 12.0 * nnz + 20.0 * n
        asm = 32.0 * f + 16.0 * fb + 16.0 * n + 8.0 * nnz + 8.0 * n + (8.0 * f if case["dim"] == 3 else 0.0)
        apply = 12.0 * nnz + 40.0 * n
        factor = 20.0 * nnz
        it = apply + spmv + 88.0 * n if case["dim"] == 2 else 2.0 * (apply + spmv) + 120.0 * n
        flops_it = (4.0 * nnz + 12.0 * n) * (1 if case["dim"] == 2 else 2)
        b, fl = 0.0, 0.0
        if op == "spmv":
            b, fl = spmv, 2.0 * nnz
        elif op == "assemble":
            b, fl = asm + spmv, 10.0 * f + 2.0 * nnz
        elif op == "corrected":
            d = case["dim"]
            b = asm + spmv + 2.0 * 8.0 * n * d + 16.0 * d * f + 32.0 * 5 * n
            fl = 60.0 * f + 2.0 * nnz
        elif op == "factor":
            b, fl = factor + apply, 6.0 * nnz
        else:
            steps = (2.5 if case["dim"] == 2 else 1.5) * side if op != "step" else (40 if case["dim"] == 2 else 10)
            if op == "batch" and case["precision"] == "mixed":
                it *= 0.6
            b = (asm + factor if op != "batch" else 0.0) + it * steps
            fl = flops_it * steps
        total["bytes"] += b
        total["flops"] += fl
    return total


# ------------------------------------------------------------------ 64-bit values
class _Operator:
    """The assembled system by faces, in plain torch (64 bits)."""

    def __init__(self, s, previous=None, gradients=None):
        m = s["mesh"]
        d = m.dim
        self.n = m.n_cells
        own = _cuda(m.face_owner.astype(np.int64))
        nb = _cuda(m.face_neighbor.astype(np.int64))
        inner = nb >= 0
        cc = _cuda(np.asarray(m.cell_center).reshape(-1, d))
        fc = _cuda(np.asarray(m.face_center).reshape(-1, d))
        area = _cuda(m.face_area)
        vol = _cuda(m.cell_volume)
        other = torch.where(inner.unsqueeze(1), cc[nb.clamp(min=0)], fc)
        dv = other - cc[own]
        corr = None
        if gradients is None:
            t = 1.0 / dv.square().sum(1).sqrt()
        else:
            nv = _cuda(np.asarray(m.face_normal).reshape(-1, d))
            t = 1.0 / (nv * dv).sum(1)
            v = nv - t.unsqueeze(1) * dv
            w = ((fc - cc[own]) * nv).sum(1) * t
            g = gradients
            gi = g[own] * (1.0 - w).unsqueeze(1) + g[nb.clamp(min=0)] * w.unsqueeze(1)
            ge = torch.where(inner.unsqueeze(1), gi, g[own])
            corr = s["kappa"] * (ge * v).sum(1) * area  # -1 (laplacian's sign) times -(kappa explicit)
        li = s["kappa"] * t
        lj = -li
        if s["flux"] is not None:
            li = li + s["flux"].clamp(min=0.0)
            lj = lj + s["flux"].clamp(max=0.0)
        li, lj = li * area, lj * area
        o, q = own[inner], nb[inner]
        self.o, self.q, self.ai, self.aj = o, q, -li[inner], lj[inner]
        diag = torch.zeros(self.n, dtype=torch.float64, device="cuda")
        rhs = s["source"] * vol
        if previous is not None:
            diag += vol / s["dt"]
            rhs = rhs + previous / s["dt"] * vol
        diag.index_add_(0, own, li)
        diag.index_add_(0, q, -lj[inner])
        fb0 = m.n_faces - m.n_boundary_faces
        bi, be = s["bc"]
        diag.index_add_(0, own[fb0:], lj[fb0:] * bi)
        rhs = rhs.index_add(0, own[fb0:], -lj[fb0:] * be)
        if corr is not None:
            rhs = rhs.index_add(0, own, corr)
            rhs = rhs.index_add(0, q, -corr[inner])
        self.diag, self.rhs = diag, rhs

    def __call__(self, x):
        y = self.diag * x
        y.index_add_(0, self.o, self.aj * x[self.q])
        y.index_add_(0, self.q, self.ai * x[self.o])
        return y

    def solve(self, symmetric, limit):
        """Jacobi-preconditioned Krylov solve to the last bits, restarted from the true residual; None if it stalls."""
        x = torch.zeros_like(self.rhs)
        goal = 2e-15 * float(self.rhs.norm())
        best = float("inf")
        for _ in range(6):
            r = self.rhs - self(x)
            now = float(r.norm())
            if now <= goal or now > 0.5 * best:
                break
            best = now
            x = x + (self._cg(r, limit) if symmetric else self._bicgstab(r, limit))
        return x if float((self.rhs - self(x)).norm()) <= 1e-12 * float(self.rhs.norm()) else None

    def _cg(self, b, limit):
        x, r = torch.zeros_like(b), b.clone()
        z = r / self.diag
        p, rz = z.clone(), r.dot(z)
        end = 1e-13 * float(b.norm())
        for k in range(limit):
            ap = self(p)
            alpha = rz / p.dot(ap)
            x += alpha * p
            r -= alpha * ap
            if k % 25 == 24 and float(r.norm()) <= end:
                break
            z = r / self.diag
            new = r.dot(z)
            p = z + (new / rz) * p
            rz = new
        return x

    def _bicgstab(self, b, limit):
        x, r, h = torch.zeros_like(b), b.clone(), b.clone()
        p, rho = r.clone(), h.dot(r)
        end = 1e-13 * float(b.norm())
        best, at = x.clone(), float("inf")
        for k in range(limit):
            y = p / self.diag
            v = self(y)
            alpha = rho / h.dot(v)
            q = r - alpha * v
            z = q / self.diag
            t = self(z)
            omega = t.dot(q) / t.dot(t)
            x = x + alpha * y + omega * z
            r = q - omega * t
            if k % 5 == 4:
                now = float(r.norm())
                if not np.isfinite(now):
                    break
                if now < at:
                    best, at = x, now
                if now <= end:
                    break
            new = h.dot(r)
            p = r + (new / rho) * (alpha / omega) * (p - omega * v)
            rho = new
        return best


def _gradients64(s, field):
    """Least-squares cell gradients with the boundary values as neighbours."""
    m = s["mesh"]
    d = m.dim
    own = _cuda(m.face_owner.astype(np.int64))
    nb = _cuda(m.face_neighbor.astype(np.int64))
    inner = nb >= 0
    cc = _cuda(np.asarray(m.cell_center).reshape(-1, d))
    fc = _cuda(np.asarray(m.face_center).reshape(-1, d))
    G = torch.zeros(m.n_cells, d, d, dtype=torch.float64, device="cuda")
    R = torch.zeros(m.n_cells, d, dtype=torch.float64, device="cuda")
    fb0 = m.n_faces - m.n_boundary_faces
    bi, be = s["bc"]
    value = field[nb.clamp(min=0)].clone()
    value[fb0:] = bi * field[own[fb0:]] + be
    dv = torch.where(inner.unsqueeze(1), cc[nb.clamp(min=0)], fc) - cc[own]
    G.index_add_(0, own, dv.unsqueeze(2) * dv.unsqueeze(1))
    R.index_add_(0, own, dv * (value - field[own]).unsqueeze(1))
    o, q, e = own[inner], nb[inner], -dv[inner]
    G.index_add_(0, q, e.unsqueeze(2) * e.unsqueeze(1))
    R.index_add_(0, q, e * (field[o] - field[q]).unsqueeze(1))
    return torch.linalg.solve(G, R)


def exact(case, seed):
    op = case["op"]
    if op == "vector":
        u, v = _randn(case["n"], seed), _randn(case["n"], seed + 1)
        w = (u + v) * 0.5
        return {"w": w, "dot": float(w.dot(v)), "sum": float(w.sum())}
    if op == "factor":
        return None  # a sequential factorisation: no plain 64-bit form within reach
    s = _batch_problem(case, seed) if op == "batch" else _problem(case, seed)
    m = s["mesh"]
    n = m.n_cells
    symmetric = case["dim"] == 2
    if op == "corrected":
        field = _bump(m) + 0.1 * _randn(n, seed + 2)
        g = _gradients64(s, field)
        op64 = _Operator(s, gradients=g)
        return {"g": g.reshape(-1), "b": op64.rhs, "Au": op64(_randn(n, seed))}
    if op == "batch":
        return _Operator(s).solve(symmetric, 4000)
    op64 = _Operator(s, previous=_bump(m) if op == "step" else None)
    if op == "spmv":
        return op64(_randn(n, seed))
    if op == "assemble":
        return {"b": op64.rhs, "Au": op64(_randn(n, seed))}
    return {"b": op64.rhs, "x": op64.solve(symmetric, 20000 if symmetric else 1500)}
