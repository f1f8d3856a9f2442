"""dot / sum in one kernel: block sums in block order, as numpy adds them in the
same shape, bit for bit, at sizes around the blocks and the largest grid, on
several host threads at once."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BLOCK, MOST = 256, 592


def _shaped(v):
    """The kernel's order of additions over the products v."""
    blocks = max(1, min((len(v) + BLOCK - 1) // BLOCK, MOST))
    threads = blocks * BLOCK
    acc = np.zeros(threads)
    for s in range(0, len(v), threads):
        part = v[s:s + threads]
        acc[:len(part)] += part
    lanes = acc.reshape(-1, 32)
    for o in (16, 8, 4, 2, 1):  # lane l adds lane l + o
        lanes = lanes.copy()
        lanes[:, :o] += lanes[:, o:2 * o]
    warps = lanes[:, 0].reshape(blocks, BLOCK // 32)
    total = 0.0
    for b in range(blocks):
        t = 0.0
        for w in warps[b]:
            t += w
        total += t
    return total


@pytest.mark.parametrize("n", [1, 32, 255, 256, 257, 511 * 256, 592 * 256 - 1, 592 * 256 + 1, 700_001])
def test_reductions_in_their_order(fv, n):
    rng = np.random.default_rng(n)
    a, b = rng.standard_normal(n), rng.standard_normal(n)
    x, y = fv.DistributedVector(a), fv.DistributedVector(b)
    assert x.dot(y) == _shaped(a * b)
    assert x.sum() == _shaped(a)


def test_reductions_on_threads(fv):
    import torch
    rng = np.random.default_rng(2)
    xs = [fv.DistributedVector(rng.standard_normal(n)) for n in (1000, 40_000, 300_001, 77)]
    want = [(x.dot(x), x.sum()) for x in xs]
    bad = []

    def work(k):
        st = torch.cuda.Stream()
        for r in range(200):
            i = (k + r) % len(xs)
            if (xs[i].dot(xs[i], stream=st), xs[i].sum(stream=st)) != want[i]:
                bad.append((k, r))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
