"""Freed device blocks of matrices and preconditioners are handed out again
only when the device has finished with them: objects built and dropped in turn
on several host threads and streams give the bits of the same work alone."""
import threading

import numpy as np
import pytest

from cases import convdiff_3d, diffusion_2d, equation

pytestmark = pytest.mark.gpu


def _once(fv, case, stream=None):
    cls = fv.IncompleteCholesky if case["c_conv"] == 0.0 else fv.IncompleteLowerUpper
    solve = fv.conjugate_gradient if case["c_conv"] == 0.0 else fv.bi_conjugate_gradient_stab
    A, b = fv.assemble(equation(fv, case), (case["bndi"], case["bnde"]), case["mesh"], stream=stream)
    P = cls.from_matrix(A, 0, stream=stream)
    x = fv.DistributedVector.from_size(case["mesh"].n_cells)
    solve(x, A, b, P, None, fv.LinearSolverOptions(1e-8, 1e-8, 500), stream=stream)
    return x


def test_blocks_reused_across_threads_and_streams(fv):
    import torch
    sizes = [(2, 40), (3, 12), (2, 120), (3, 22)]
    cases = [diffusion_2d(fv, s, seed=80 + s) if d == 2 else convdiff_3d(fv, s, seed=80 + s) for d, s in sizes]
    alone = [_once(fv, c).numpy() for c in cases]
    bad = []

    def work(k):
        st = torch.cuda.Stream()
        with torch.cuda.stream(st):
            for r in range(6):
                i = (k + r) % len(cases)
                x = _once(fv, cases[i], stream=st)
                st.synchronize()
                if not np.array_equal(x.numpy(), alone[i]):
                    bad.append((k, r, i))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


@pytest.mark.parametrize("n", [6, 12])
def test_kept_blocks_are_not_taken_while_a_solve_is_captured(fv, n):
    """Box tiles allocate at their first apply, which a solve captures: blocks kept
    from an earlier object must not be handed out there, in part or in whole."""
    case = convdiff_3d(fv, n, seed=6)
    A, b = fv.assemble(equation(fv, case), (case["bndi"], case["bnde"]), case["mesh"])
    opts = fv.LinearSolverOptions(1e-10, 1e-10, 2000)
    got = []
    for req in (1, 2, 2, 2):
        P = fv.IncompleteLowerUpper.from_matrix(A, 0)
        P.schedule(req)
        for _ in range(2):
            x = fv.DistributedVector.from_size(A.nrows())
            fv.bi_conjugate_gradient_stab(x, A, b, P, None, opts)
            got.append(x.numpy())
        P.close()
    for x in got[1:]:
        assert np.array_equal(x, got[0])
