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
