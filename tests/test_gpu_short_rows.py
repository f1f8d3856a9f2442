"""IC(0) / ILU(0) of short rows (at most 6 entries, values as readiness) and the
level analysis against the oracle, bit for bit, on patterns whose rows do and do
not hold mutually adjacent neighbours, of 3 to 7 entries, at row counts around
a chunk of 32 rows, in natural and permuted order, again after new values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pattern(n, name):
    """Symmetric neighbour offsets per row."""
    edges = set()
    for i in range(n):
        for d in {"tri": (1,), "penta": (1, 2), "wide": (1, 2), "far": (7, 40), "seven": (1, 2, 3)}[name]:
            if i + d < n:
                edges.add((i, i + d))
        if name == "wide" and i % 2 == 0 and i + 35 < n:
            edges.add((i, i + 35))
    return sorted(edges)


def _matrix(n, name, seed, symmetric):
    rng = np.random.default_rng(seed)
    rows, cols, vals = list(range(n)), list(range(n)), list(8.0 + rng.random(n))
    for a, b in _pattern(n, name):
        u = -rng.random() - 0.1
        rows += [a, b]
        cols += [b, a]
        vals += [u, u if symmetric else -rng.random() * 1e-5 if (a + b) % 5 == 0 else -rng.random() - 0.1]
    r, c, v = np.array(rows), np.array(cols), np.array(vals)
    o = np.lexsort((c, r))
    ptr = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]).astype(np.int32)
    return ptr, c[o].astype(np.int32), v[o]


@pytest.mark.parametrize("kind", ["ic", "ilu"])
@pytest.mark.parametrize("name", ["tri", "penta", "wide", "far", "seven"])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 1000])
def test_short_rows_against_the_oracle(fv, orc, kind, name, n):
    cls = fv.IncompleteCholesky if kind == "ic" else fv.IncompleteLowerUpper
    ptr, cols, vals = _matrix(n, name, 3, kind == "ic")
    A = fv.DistributedMatrix.from_csr(ptr, cols, vals)
    perm = np.random.default_rng(4).permutation(n).astype(np.int32)
    r = np.random.default_rng(5).standard_normal(n)
    for ordering in (None, perm):
        P = cls.from_matrix(A, 0, ordering=ordering)
        bp, bc, bv = (ptr, cols, vals) if ordering is None else orc.permute(ptr, cols, vals, perm)
        o = orc.Precond(kind, bp, bc, bv)
        for _ in range(2):
            gp, gc, gv, gd = P.factors()
            op, oc, ov, _, od = o.export()
            assert np.array_equal(gp, op) and np.array_equal(gc, oc) and np.array_equal(gv, ov) and gd == od
            P.refactor()
        fl, bl, nf, nb = P.levels()
        of, onf = orc.levels(bp, bc)
        ob, onb = orc.levels(bp, bc, upper=True)
        assert np.array_equal(fl, of) and np.array_equal(bl, ob) and (nf, nb) == (onf, onb)
        z = fv.DistributedVector.from_size(n)
        P.precondition(z, fv.DistributedVector(r))
        expected = o.apply(r) if ordering is None else orc.Precond.reordered(kind, ptr, cols, vals, perm).apply(r)
        assert np.array_equal(z.numpy(), expected)
