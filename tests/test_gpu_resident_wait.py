"""The resident sweeps' wait for their record copies: a copy that never counts as
landed ends in one bounded wait (20 ms here) and one for the copies in flight,
over however many groups and sweeps, with the error word set and NaN for a
result; an error that is raised already ends it at once."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TIMEOUT, SINGULAR, LIMIT_MS = 1, 2, 20.0


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    from fvb200.build import CSRC, INCLUDE, NVCC_FLAGS, _nvcc
    out = tmp_path_factory.mktemp("wait") / "resident_wait.so"
    src = Path(__file__).resolve().parent / "resident_wait.cu"
    subprocess.run([_nvcc(), *NVCC_FLAGS, "-shared", "-I", str(INCLUDE), "-I", str(CSRC), "-include", "vector",
                    "-include", "cstring", str(src), "-o", str(out)], check=True)
    L = C.CDLL(str(out))
    L.run.restype = C.c_float

    def call(levels, never, raised):
        n = levels * 32
        rng = np.random.default_rng(levels)
        r, d, z, err = rng.standard_normal(n), rng.standard_normal(n), np.zeros(n), C.c_int(-1)
        p = [v.ctypes.data_as(C.c_void_p) for v in (r, d, z)]
        ms = L.run(levels, never, raised, *p, C.byref(err))
        return ms, z, d * (d * (d * (d * r))), err.value
    return call


@pytest.mark.parametrize("levels", [1, 4, 5, 20, 64, 250])
def test_copies_that_land(run, levels):
    for raised in (0, SINGULAR):
        ms, z, want, err = run(levels, 0, raised)
        assert ms >= 0 and err == raised and np.array_equal(z, want)


@pytest.mark.parametrize("levels", [1, 5, 64, 250])
def test_copies_that_never_land(run, levels):
    ms, z, _, err = run(levels, 1, 0)
    assert err == TIMEOUT and np.isnan(z).all()
    assert LIMIT_MS <= ms < 3 * LIMIT_MS
    ms, z, _, err = run(levels, 1, SINGULAR)
    assert err == SINGULAR and np.isnan(z).all()
    assert 0 <= ms < 2 * LIMIT_MS
