"""Memory that outlives a call -- the blocks of matrices and preconditioners,
the workspace of the reductions -- against a fake CUDA runtime (fake_cuda.cpp),
where a context can be replaced, memory can run out and queued work can be seen."""
import ctypes as C
import subprocess
import threading
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "finite-volumes-rs_b200" / "csrc"
MB = 1 << 20


@pytest.fixture(scope="module")
def lib_path(tmp_path_factory):
    from fvb200.build import INCLUDE, _nvcc
    d = tmp_path_factory.mktemp("fake")
    objs = []
    for src in (CSRC / "fv_pool.cu", CSRC / "fv_vector.cu"):
        objs.append(str(d / (src.stem + ".o")))
        subprocess.run([_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O1", "--extended-lambda",
                        "-Xcompiler", "-fPIC", "-I", str(INCLUDE), "-I", str(CSRC), "-c", str(src), "-o", objs[-1]],
                       check=True)
    out = d / "libfake.so"
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic,--no-undefined", "-I",
                    "/usr/local/cuda/include", str(ROOT / "tests" / "fake_cuda.cpp"), *objs, "-o", str(out)], check=True)
    return out


MALLOCS, FREES, BAD = range(3)


@pytest.fixture
def cu(lib_path, tmp_path):
    """The library of its own: nothing kept from another test."""
    own = tmp_path / "lib.so"
    own.write_bytes(lib_path.read_bytes())
    L = C.CDLL(str(own))
    L.pool_alloc.restype = C.c_void_p
    L.pool_alloc.argtypes = [C.c_size_t]
    L.pool_free.argtypes = [C.c_void_p]
    L.fake_use.argtypes = L.fake_busy.argtypes = [C.c_void_p]
    L.fake_count.restype = C.c_longlong
    L.fake_used.restype = L.fake_capacity.restype = C.c_size_t
    L.fake_capacity.argtypes = [C.c_size_t]
    L.fv_vec_sum.argtypes = [C.c_int64, C.c_void_p, C.c_void_p, C.POINTER(C.c_double)]
    L.fake_reset()
    return L


def _sum(L, n):
    out = C.c_double(-1.0)
    assert L.fv_vec_sum(n, C.c_void_p(16), None, C.byref(out)) == 0
    return out.value


@pytest.mark.parametrize("device", [0, 1])
def test_reductions_after_a_context_was_replaced(cu, device):
    """The partials and the pinned result belong to their device's context."""
    assert _sum(cu, 1000) == 1000.0
    cu.fake_device(device)
    assert _sum(cu, 1001) == 1001.0
    cu.fake_device(0)
    cu.fake_replace_context()
    cu.fake_device(device)
    assert _sum(cu, 1002) == 1002.0
    cu.fake_device(0)
    assert _sum(cu, 1003) == 1003.0
    assert cu.fake_count(BAD) == 0


@pytest.mark.parametrize("ids", [True, False])
def test_reductions_on_short_lived_threads_take_no_more_memory(cu, ids):
    cu.fake_no_context_ids(not ids)
    for device in (0, 1):
        cu.fake_device(device)
        assert _sum(cu, 5) == 5.0
    used = []
    for k in range(4):
        def work():
            for device in (0, 1):
                cu.fake_device(device)
                assert _sum(cu, 7 + k) == 7.0 + k
        t = threading.Thread(target=work)
        t.start()
        t.join()
        used.append([])
        for device in (0, 1):
            cu.fake_device(device)
            used[-1].append(cu.fake_used())
    assert used[0] == used[3] and cu.fake_count(BAD) == 0


def test_kept_blocks_serve_a_thread_without_a_context(cu):
    """A host thread's first call: no context is current on it yet, the kept blocks are still the device's."""
    cu.pool_free(cu.pool_alloc(8 * MB))
    got = []
    t = threading.Thread(target=lambda: got.append(cu.pool_alloc(8 * MB)))
    t.start()
    t.join()
    assert cu.fake_used() == 8 * MB  # the kept block, not a second one
    cu.pool_free(got[0])
    assert cu.pool_alloc(8 * MB) == got[0] and cu.fake_used() == 8 * MB
    assert cu.fake_count(BAD) == 0


def test_nothing_is_kept_when_contexts_are_unknown(cu):
    cu.fake_no_context_ids(1)
    for _ in range(3):
        cu.pool_free(cu.pool_alloc(MB))
    assert cu.fake_used() == 0 and cu.fake_count(BAD) == 0


def test_addresses_of_a_replaced_context(cu):
    """What was live or kept in a context that is gone says nothing about the same
    addresses in the next one."""
    first = cu.pool_alloc(MB)
    cu.pool_free(cu.pool_alloc(2 * MB))
    cu.fake_replace_context()
    large = cu.pool_alloc(100 * MB)
    assert large == first
    cu.pool_free(large)  # not a block of 1 MB to be kept
    assert cu.fake_used() == 0
    p = cu.pool_alloc(2 * MB)
    assert cu.fake_used() == 2 * MB
    cu.pool_free(p)
    assert cu.fake_count(BAD) == 0


@pytest.mark.parametrize("mb", [30, 100])
def test_kept_blocks_are_given_back_when_memory_runs_out(cu, mb):
    cu.fake_capacity(120 * MB)
    blocks = [cu.pool_alloc(10 * MB) for _ in range(10)]
    for p in blocks:
        cu.pool_free(p)
    assert cu.fake_used() == 100 * MB
    assert cu.pool_alloc(mb * MB)
    assert cu.fake_used() == mb * MB and cu.fake_count(BAD) == 0
    assert not cu.pool_alloc(121 * MB)


@pytest.mark.parametrize("allocator", ["device_alloc", "stream_alloc"])
def test_the_other_allocations_get_kept_blocks_back_too(cu, allocator):
    """Meshes, batches and distributed systems (device_alloc), the solvers' and the
    factorisation's workspaces (stream_alloc)."""
    cu.fake_capacity(120 * MB)
    for p in [cu.pool_alloc(10 * MB) for _ in range(10)]:
        cu.pool_free(p)
    f = getattr(cu, allocator)
    f.restype, f.argtypes = C.c_void_p, [C.c_size_t]
    assert f(90 * MB)
    assert cu.fake_used() == 90 * MB and cu.fake_count(BAD) == 0
    assert not f(31 * MB)

def test_release_kept_memory(cu):
    cu.pool_free(cu.pool_alloc(10 * MB))
    assert cu.fv_release_kept_memory() == 0
    assert cu.fake_used() == 0 and cu.fake_count(BAD) == 0


def test_the_oldest_kept_blocks_make_room(cu):
    """A large system that is gone leaves full shelves; what is in use now is kept all the same."""
    for p in [cu.pool_alloc(60 * MB) for _ in range(8)]:
        cu.pool_free(p)
    small = [cu.pool_alloc(10 * MB) for _ in range(4)]
    for p in small:
        cu.pool_free(p)
    before = cu.fake_count(MALLOCS)
    for _ in range(3):
        again = [cu.pool_alloc(10 * MB) for _ in range(4)]
        assert sorted(again) == sorted(small)
        for p in again:
            cu.pool_free(p)
    fences = 3 * 4  # fv_blocks_free may allocate to wait for the device
    assert cu.fake_count(MALLOCS) - before <= fences
    assert cu.fake_used() <= 512 * MB and cu.fake_count(BAD) == 0


def test_a_block_is_handed_out_again_only_when_its_work_is_done(cu):
    p = cu.pool_alloc(MB)
    cu.fake_use(p)
    cu.pool_free(p)
    assert cu.pool_alloc(MB) == p and not cu.fake_busy(p)
    before = cu.fake_count(MALLOCS), cu.fake_count(FREES)
    cu.pool_free(None)  # an object without blocks waits for nothing
    assert (cu.fake_count(MALLOCS), cu.fake_count(FREES)) == before and cu.fake_count(BAD) == 0


def test_flags_of_a_replaced_context(cu):
    cu.fake_pinned.restype = C.c_size_t
    for _ in range(3):
        assert cu.flag_is_there(1)
    assert cu.fake_pinned() == 1
    cu.fake_replace_context()
    assert cu.flag_is_there(1)
    assert cu.flag_is_there(0) and cu.fake_pinned() == 0  # taken again, then freed: work was in flight
    assert cu.fake_count(BAD) == 0
