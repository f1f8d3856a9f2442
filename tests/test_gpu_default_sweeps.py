"""The library's own choice of sweeps: queried, given up for an explicit schedule,
taken up again, and among the tuner's candidates."""
import numpy as np
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


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_a_batch_says_when_each_problem_has_its_cluster(fv, precision):
    from fvb200.batch import BatchCG, MeshBatch
    meshes = [fv.Mesh.square(s, 0.2, 70 + s) for s in (9, 14)]
    f = [m.fields(70, 1.0, 0.5, source_const=1.0) for m in meshes]
    mb = MeshBatch(meshes)
    zero = np.zeros(mb.n_boundary_faces)
    eq = -fv.laplacian(fv.Orthogonal(), mb.face_field([q[0] for q in f])) - fv.source(mb.cell_field([q[2] for q in f]))
    A, b = fv.assemble(eq, (zero, zero), mb)
    x = fv.DistributedVector.from_size(mb.n_cells)
    for ordering, clusters in (("boxes", True), (None, False)):
        P = fv.IncompleteCholesky.from_matrix(A, 0, ordering=ordering, offsets=mb.cell_offsets if ordering else None)
        assert not P.resident(batch=True)
        BatchCG(A, mb.cell_offsets, 256).solve(P, b, x, precision=precision)
        assert P.resident(batch=True) == clusters
        P.schedule(1)
        assert not P.resident(batch=True) and not P.resident()
