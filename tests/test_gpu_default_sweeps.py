"""The library's own choice of sweeps: queried, given up for an explicit schedule,
taken up again, and among the tuner's candidates."""
import pytest

from cases import diffusion_2d, equation
from test_gpu_resident import _pair, _same_apply

pytestmark = pytest.mark.gpu


def test_the_default_sweeps_can_be_asked_for_again(fv):
    """An explicit schedule takes the other kernels; the default comes back with the same bits."""
    from fvb200.batch import autotune_schedule
    case = diffusion_2d(fv, 96, seed=67)
    A, b = fv.assemble(equation(fv, case), (case["bndi"], case["bnde"]), case["mesh"])
    n = case["mesh"].n_cells
    for M, schedule in ((A, 1), (A.permuted(fv.order_boxes(A)[0]), 4)):
        P, Q = _pair(fv, fv.IncompleteCholesky, M)
        assert P.resident() and not Q.resident()
        _same_apply(fv, P, Q, n)
        P.refactor()
        Q.refactor()
        Q.default_schedule()
        assert Q.resident() and Q.schedule()[0] == P.schedule()[0] == schedule
        P.schedule(3)
        assert not P.resident()
        _same_apply(fv, P, Q, n)
    P, Q = _pair(fv, fv.IncompleteCholesky, A)
    x = fv.DistributedVector.from_size(n)
    best, times = autotune_schedule(Q, b, x)  # 192 levels: several times faster in one cluster
    assert best == "default" and times["default"] < min(times[1], times[3]) and Q.resident()
    large = diffusion_2d(fv, 420, seed=68)  # more rows than a cluster takes: as ever
    A, b = fv.assemble(equation(fv, large), (large["bndi"], large["bnde"]), large["mesh"])
    P = fv.IncompleteCholesky.from_matrix(A, 0)
    best, times = autotune_schedule(P, b, fv.DistributedVector.from_size(A.nrows()))
    assert not P.resident() and best in (1, 3) and set(times) == {1, 3} and P.schedule()[0] == best
