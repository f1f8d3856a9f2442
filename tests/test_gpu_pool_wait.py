"""Blocks of a matrix that is dropped with work queued on them: the next matrix
gets them only when that work is done, on whatever stream it runs, and dropping
one does not disturb a stream capture on another host thread."""
import threading

import numpy as np
import pytest

from cases import convdiff_3d, equation

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [6, 20])
def test_dropped_with_work_queued(fv, side):
    import torch
    case = convdiff_3d(fv, side, seed=91)
    n = case["mesh"].n_cells
    x = fv.DistributedVector(np.random.default_rng(3).standard_normal(n))
    bc = (case["bndi"], case["bnde"])
    kappa = case["kappa"]

    def build(scale, stream):
        case["kappa"] = kappa * scale
        return fv.assemble(equation(fv, case), bc, case["mesh"], stream=stream)[0]

    streams = [torch.cuda.Stream(), torch.cuda.Stream()]  # non-blocking
    want = []
    for scale in (1.0, 3.0):
        y = fv.DistributedVector.from_size(n)
        build(scale, None).imul(y, x)
        want.append(y.numpy())
    assert not np.array_equal(*want)
    for _ in range(3):
        y = [fv.DistributedVector.from_size(n) for _ in range(2)]
        A = build(1.0, streams[0])
        torch.cuda.synchronize()
        with torch.cuda.stream(streams[0]):
            torch.cuda._sleep(20_000_000)  # some 10 ms
        A.imul(y[0], x, stream=streams[0])
        A.close()
        with torch.cuda.stream(streams[1]):
            B = build(3.0, streams[1])
            B.imul(y[1], x, stream=streams[1])
        torch.cuda.synchronize()
        assert np.array_equal(y[0].numpy(), want[0]) and np.array_equal(y[1].numpy(), want[1])


def test_dropped_while_another_thread_captures(fv):
    import torch
    case = convdiff_3d(fv, 6, seed=92)
    A, _ = fv.assemble(equation(fv, case), (case["bndi"], case["bnde"]), case["mesh"])
    P = fv.IncompleteLowerUpper.from_matrix(A, 0)
    v = torch.zeros(1000, device="cuda")
    g = torch.cuda.CUDAGraph()

    def drop():
        P.close()
        A.close()

    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        v += 1.0
        t = threading.Thread(target=drop)
        t.start()
        t.join()
    g.replay()
    torch.cuda.synchronize()
    assert float(v.sum()) == 1000.0
