"""The plans of the resident sweeps where shared memory, rows per level or levels
are at the ends of what they take: the same bits as the level-chunk kernels of
the same factor, and the plans that are expected."""
import numpy as np
import pytest

from cases import convdiff_3d, diffusion_2d, equation
from test_gpu_resident import _pair, _same_apply

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,side,fits", [(2, 128, True), (2, 134, True), (2, 150, True), (2, 181, True),
                                           (2, 392, True), (3, 26, True), (3, 35, False), (3, 37, False)])
def test_natural_orders_between_the_sizes_that_fit_at_once(fv, dim, side, fits):
    """Wide steps' buffers and the rows of a CTA together: twice the CTAs, or half
    the thread sets (3D beyond 200,000 rows: rows and halo alone leave no room)."""
    case = diffusion_2d(fv, side, seed=65) if dim == 2 else convdiff_3d(fv, side, seed=65)
    A, _ = fv.assemble(equation(fv, case), (case["bndi"], case["bnde"]), case["mesh"])
    P, Q = _pair(fv, fv.IncompleteCholesky if dim == 2 else fv.IncompleteLowerUpper, A)
    assert P.resident() == fits
    _same_apply(fv, P, Q, case["mesh"].n_cells)


def _channel(nx, ny):
    """5-point operator on nx x ny points, no mesh behind it: about nx rows per level."""
    n = nx * ny
    i = np.arange(n)
    x, y = i % nx, i // nx
    rows, cols, vals = [i], [i], [4.5 + 0.1 * np.sin(i)]
    for ok, off in ((x > 0, -1), (x < nx - 1, 1), (y > 0, -nx), (y < ny - 1, nx)):
        rows.append(i[ok])
        cols.append(i[ok] + off)
        vals.append(-1.0 + 0.01 * np.sin(i[ok] + (i[ok] + off)))
    r, c, v = np.concatenate(rows), np.concatenate(cols), np.concatenate(vals)
    o = np.lexsort((c, r))
    return np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]), c[o], v[o]


@pytest.mark.parametrize("nx,n,fits", [(1, 5000, True), (1, 40_000, False), (2, 20_000, True), (4, 100_000, False),
                                       (7, 60_000, True), (16, 100_000, True), (33, 50_000, True), (64, 300_000, True), (65, 30_000, True),
                                       (100, 300_000, True),
                                       (127, 40_000, True), (129, 40_000, True)])
def test_narrow_levels(fv, nx, n, fits):
    """Few rows per level: bands of levels, without a record's step for every row;
    where idle slots would be most of a large plan, there is none."""
    import torch
    A = fv.DistributedMatrix.from_csr(*_channel(nx, n // nx))
    rows = A.nrows()
    fv.IncompleteCholesky.from_matrix(A, 0).close()  # the symbolic analysis stays with A
    fv.release_kept_memory()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    P = fv.IncompleteCholesky.from_matrix(A, 0)
    torch.cuda.synchronize()
    taken = free - torch.cuda.mem_get_info()[0]
    assert P.resident() == fits
    assert taken <= 128 << 20 or taken <= 800 * rows  # 5 slots of 64 bytes, twice; factor and vectors
    Q = fv.IncompleteCholesky.from_matrix(A, 0)
    Q.schedule(1)
    _same_apply(fv, P, Q, rows)
    P.refactor()
    Q.refactor()
    _same_apply(fv, P, Q, rows, 1)


@pytest.mark.parametrize("dim,side,block,fits", [(2, 100, 1, True), (2, 150, 1, False), (2, 150, 512, True),
                                                 (3, 14, 1, True), (3, 22, 1, False)])
def test_orders_without_locality(fv, dim, side, block, fits):
    """Rows, or blocks of them, in random order: swept by level chunks where most values would be handed over."""
    case = diffusion_2d(fv, side, seed=69) if dim == 2 else convdiff_3d(fv, side, seed=69)
    A, _ = fv.assemble(equation(fv, case), (case["bndi"], case["bnde"]), case["mesh"])
    n = case["mesh"].n_cells
    parts = np.array_split(np.arange(n, dtype=np.int32), n // block)
    order = np.random.default_rng(8).permutation(len(parts))
    perm = np.concatenate([parts[k] for k in order])
    P, Q = _pair(fv, fv.IncompleteCholesky if dim == 2 else fv.IncompleteLowerUpper, A, ordering=perm)
    assert P.resident() == fits
    _same_apply(fv, P, Q, n)


@pytest.mark.parametrize("dim,side,ordering", [(2, 142, None), (2, 193, None), (2, 194, None), (2, 193, "boxes"),
                                               (3, 22, None), (3, 22, "boxes"), (3, 23, None)])
def test_whole_iterations_up_to_their_rows(fv, dim, side, ordering):
    """75,000 rows of CG and 65,000 of BiCGStab, just below and above: the kernels' bits and history."""
    case = diffusion_2d(fv, side, seed=71) if dim == 2 else convdiff_3d(fv, side, seed=71)
    solve = fv.conjugate_gradient if dim == 2 else fv.bi_conjugate_gradient_stab
    A, b = fv.assemble(equation(fv, case), (case["bndi"], case["bnde"]), case["mesh"])
    P, Q = _pair(fv, fv.IncompleteCholesky if dim == 2 else fv.IncompleteLowerUpper, A, ordering=ordering)
    for tol, limit in ((0.0, 7), (1e-6, 300)):
        got = []
        for M in (P, Q):
            x = fv.DistributedVector.from_size(A.nrows())
            info = solve(x, A, b, M, None, fv.LinearSolverOptions(tol, tol, limit))
            got.append((x.numpy(), np.array(info.history), info.iterations, info.status))
        assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
        assert got[0][2:] == got[1][2:]
