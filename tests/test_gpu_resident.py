"""Resident sweeps (one cluster, the vector in shared memory) against the
level-chunk kernels of the same factor, asked for explicitly: the same bits,
at sizes around the step width, the cluster sizes and the record sizes, on
repeated applies and after a refactorisation, in FP64 (preconditioner apply)
and FP32 (mixed batch solve), with rows without any dependency and with
non-finite right-hand sides."""
import numpy as np
import pytest

from cases import convdiff_3d, diffusion_2d, equation

pytestmark = pytest.mark.gpu


def _pair(fv, cls, A, **kw):
    P, Q = cls.from_matrix(A, 0, **kw), cls.from_matrix(A, 0, **kw)
    Q.schedule(1)
    return P, Q


def _same_apply(fv, P, Q, n, seed=0):
    rng = np.random.default_rng(seed)
    z, y = fv.DistributedVector.from_size(n), fv.DistributedVector.from_size(n)
    for k in range(3):
        r = rng.standard_normal(n)
        if k == 2 and n > 3:
            r[n // 2], r[n // 3], r[0] = np.inf, np.nan, -0.0
        P.precondition(z, fv.DistributedVector(r))
        Q.precondition(y, fv.DistributedVector(r))
        a, b = z.numpy(), y.numpy()
        assert np.array_equal(a, b, equal_nan=True)
        assert np.array_equal(np.signbit(a[a == 0]), np.signbit(b[b == 0]))


@pytest.mark.parametrize("dim,side", [(2, 1), (2, 3), (2, 31), (2, 33), (2, 95), (2, 141), (3, 1), (3, 2), (3, 7),
                                      (3, 13), (3, 21), (3, 31)])
def test_resident_equals_level_chunks(fv, dim, side):
    case = diffusion_2d(fv, side, seed=61) if dim == 2 else convdiff_3d(fv, side, seed=62)
    cls = fv.IncompleteCholesky if dim == 2 else fv.IncompleteLowerUpper
    A, _ = fv.assemble(equation(fv, case), (case["bndi"], case["bnde"]), case["mesh"])
    n = case["mesh"].n_cells
    B = A.permuted(fv.order_boxes(A)[0])
    for M, kw in ((A, {}), (A, {"ordering": "boxes"}), (B, {})):
        P, Q = _pair(fv, cls, M, **kw)
        _same_apply(fv, P, Q, n)
    case["kappa"] = case["kappa"] * 1.7  # new values, the plan kept
    fv.assemble(equation(fv, case), (case["bndi"], case["bnde"]), case["mesh"], lhs=A)
    P, Q = _pair(fv, cls, A)
    case["kappa"] = case["kappa"] * 0.3
    fv.assemble(equation(fv, case), (case["bndi"], case["bnde"]), case["mesh"], lhs=A)
    P.refactor()
    Q.refactor()
    _same_apply(fv, P, Q, n, 1)


def _grid7(m):
    """7-point operator on an m^3 grid: rows of up to 7 entries, no mesh behind it."""
    i = np.arange(m ** 3)
    x, y, z = i % m, (i // m) % m, i // (m * m)
    rows, cols, vals = [i], [i], [np.full(m ** 3, 6.5)]
    for ok, off in ((x > 0, -1), (x < m - 1, 1), (y > 0, -m), (y < m - 1, m), (z > 0, -m * m), (z < m - 1, m * m)):
        rows.append(i[ok])
        cols.append(i[ok] + off)
        vals.append(np.full(ok.sum(), -1.0) + 0.01 * np.sin(i[ok] + off + i[ok]))
    r, c, v = np.concatenate(rows), np.concatenate(cols), np.concatenate(vals)
    o = np.lexsort((c, r))
    ptr = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=m ** 3))])
    return ptr, c[o], v[o], (x + y + z) % 2


@pytest.mark.parametrize("m", [2, 9, 24])
@pytest.mark.parametrize("kind", ["ic", "ilu"])
def test_resident_without_a_mesh_and_long_rows(fv, m, kind):
    ptr, cols, vals, colour = _grid7(m)
    A = fv.DistributedMatrix.from_csr(ptr, cols, vals)
    cls = fv.IncompleteCholesky if kind == "ic" else fv.IncompleteLowerUpper
    red_black = np.argsort(colour, kind="stable").astype(np.int32)  # 6 entries on one side of a row
    shuffled = np.random.default_rng(5).permutation(m ** 3).astype(np.int32)
    for kw in ({}, {"ordering": red_black}, {"ordering": shuffled}):
        P, Q = _pair(fv, cls, A, **kw)
        _same_apply(fv, P, Q, m ** 3)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("sides,ordering", [((3, 9, 5), None), ((3, 9, 5), "boxes"), ((2, 1, 2, 3, 1), "boxes"),
                                            (tuple(range(2, 20)), "boxes"), ((21, 4), "boxes")])
def test_resident_in_a_batch(fv, precision, sides, ordering):
    """Problems that converge at different iterations, on one cluster or several:
    converged rows are skipped the same way; again after new values."""
    from fvb200.batch import BatchCG, MeshBatch
    meshes = [fv.Mesh.cube(s, 0.15, 70 + s) for s in sides]
    f = [m.fields(70, 0.1, 0.5, velocity=(1.0, 0.5, 0.25), source_uniform=True) for m in meshes]
    mb = MeshBatch(meshes)
    kf, fl, sc = (mb.face_field([q[0] for q in f]), mb.face_field([q[1] for q in f]), mb.cell_field([q[2] for q in f]))
    bc = (np.zeros(mb.n_boundary_faces), np.zeros(mb.n_boundary_faces))
    A = None
    P = []
    for scale in (1.0, 2.5):
        eq = fv.convection(fv.Upwind(fl), fl) - fv.laplacian(fv.Orthogonal(), kf * scale) - fv.source(sc)
        A, b = fv.assemble(eq, bc, mb, lhs=A)
        out = []
        for k, explicit in enumerate((False, True)):
            if len(P) < 2:
                P.append(fv.IncompleteLowerUpper.from_matrix(A, 0, ordering=ordering,
                                                             offsets=mb.cell_offsets if ordering else None))
                if explicit:
                    P[k].schedule(1)
            else:
                P[k].refactor()
            x = fv.DistributedVector.from_size(mb.n_cells)
            info = BatchCG(A, mb.cell_offsets, 256).solve(P[k], b, x, precision=precision, solver="bicgstab")
            out.append((x.numpy(), info["iterations"].tolist()))
        assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]


@pytest.mark.parametrize("dim,side,ordering", [(2, 2, None), (2, 22, None), (2, 23, "boxes"), (2, 130, None),
                                               (2, 190, "boxes"), (3, 2, None), (3, 7, "boxes"), (3, 20, None)])
def test_resident_solve_equals_kernels(fv, dim, side, ordering):
    """Whole iterations in one cluster against the iteration's kernels (an explicit
    schedule takes them): the same bits, the same history, at row counts around
    the reduction blocks (1,024 rows), the cluster sizes and the limits, with the
    iteration limit reached in the middle and past the iterations of one launch."""
    case = diffusion_2d(fv, side, seed=63) if dim == 2 else convdiff_3d(fv, side, seed=64)
    cls = fv.IncompleteCholesky if dim == 2 else fv.IncompleteLowerUpper
    solve = fv.conjugate_gradient if dim == 2 else fv.bi_conjugate_gradient_stab
    A, b = fv.assemble(equation(fv, case), (case["bndi"], case["bnde"]), case["mesh"])
    P = cls.from_matrix(A, 0, ordering=ordering)
    Q = cls.from_matrix(A, 0, ordering=ordering)
    Q.schedule(1)
    n = case["mesh"].n_cells
    x0 = np.random.default_rng(9).standard_normal(n) * 1e-3
    for tol, limit in ((1e-8, 2000), (0.0, 7), (1e-300, 300)):
        got = []
        for M in (P, Q):
            x = fv.DistributedVector(x0)
            info = solve(x, A, b, M, None, fv.LinearSolverOptions(tol, tol, limit))
            got.append((x.numpy(), np.array(info.history), info.iterations, info.restarts, info.status,
                        info.initial_residual, info.final_residual))
        assert np.array_equal(got[0][0], got[1][0], equal_nan=True)
        assert np.array_equal(got[0][1], got[1][1], equal_nan=True)
        assert np.array_equal(got[0][2:], got[1][2:], equal_nan=True)


@pytest.mark.parametrize("side", [128, 181, 362, 392])
def test_resident_where_shared_memory_fills(fv, side):
    """Long natural orders whose rows and eight sets' buffers fit, fit on twice the
    CTAs, fit the largest cluster, or leave four sets: the same bits."""
    case = diffusion_2d(fv, side, seed=65)
    A, _ = fv.assemble(equation(fv, case), (case["bndi"], case["bnde"]), case["mesh"])
    P, Q = _pair(fv, fv.IncompleteCholesky, A)
    _same_apply(fv, P, Q, case["mesh"].n_cells)


@pytest.mark.parametrize("side", [200, 201])
def test_resident_up_to_its_rows_in_level_order(fv, side):
    """80,000 rows sorted by level and just above: the cluster's sweeps, then
    consecutive rows on all SMs; the same bits."""
    case = diffusion_2d(fv, side, seed=66)
    A, _ = fv.assemble(equation(fv, case), (case["bndi"], case["bnde"]), case["mesh"])
    P, Q = _pair(fv, fv.IncompleteCholesky, A.permuted(fv.order_boxes(A)[0]))
    _same_apply(fv, P, Q, case["mesh"].n_cells)
