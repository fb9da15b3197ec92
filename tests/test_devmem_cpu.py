"""The library's store of device blocks (csrc/devmem.cu) against a counting stand-in for the CUDA
allocator: what is kept is counted and bounded also when another thread ends the last plan, or a
failed allocation empties the store, while a block is on its way in. The other thread's action is
played from inside the wait for the device, where the store's lock is open."""
import ctypes
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MIB = 1 << 20

HARNESS = r"""
#include "devmem.cu"
#include <cstdlib>
#include <map>
static std::map<void*, size_t> g_live;
static size_t g_bytes = 0;
static int g_allocs = 0, g_fail = 0, g_in_wait = 0;   // g_in_wait: what another thread does meanwhile
extern "C" cudaError_t cudaMalloc(void** p, size_t n) {
    if (g_fail > 0) { --g_fail; return cudaErrorMemoryAllocation; }
    *p = std::malloc(1);
    g_live[*p] = n;
    g_bytes += n;
    ++g_allocs;
    return cudaSuccess;
}
extern "C" cudaError_t cudaFree(void* p) {
    if (!g_live.count(p)) std::abort();
    g_bytes -= g_live[p];
    g_live.erase(p);
    std::free(p);
    return cudaSuccess;
}
extern "C" cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }
extern "C" const char* cudaGetErrorString(cudaError_t) { return "error"; }
extern "C" cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
extern "C" cudaError_t cudaDeviceSynchronize() {
    const int what = g_in_wait;
    g_in_wait = 0;
    if (what >= 1) hfmm::dev_plan_count(-1);   // the last plan ends
    if (what >= 2) hfmm::dev_plan_count(1);    // and another begins
    if (what == 3) {                           // or an allocation fails once
        g_fail = 1;
        size_t cap;
        int dev;
        hfmm::dev_free(hfmm::dev_alloc(3 << 20, &cap, &dev), cap, dev, true);
    }
    return cudaSuccess;
}
extern "C" void plans(int n) { hfmm::dev_plan_count(n); }
extern "C" size_t live() { return g_bytes; }
extern "C" int allocs() { return g_allocs; }
extern "C" void in_wait(int what) { g_in_wait = what; }
extern "C" void* take(size_t n, size_t* cap) {
    int dev;
    return hfmm::dev_alloc(n, cap, &dev);
}
// cap of a DevBuf of `first` bytes after a second alloc of `second` bytes
extern "C" size_t resized(size_t first, size_t second) {
    hfmm::KeepBlocks keep;
    hfmm::DevBuf<char> b;
    b.alloc(first);
    b.alloc(second);
    return b.cap;
}
// bytes of a buffer of between `least` and `most`, the device full `times` times (0: refused)
extern "C" size_t between(size_t least, size_t most, int times) {
    hfmm::DevBuf<char> b;
    g_fail = 2 * times;   // dev_alloc tries again once the store is empty
    try {
        b.alloc_between(least, most);
    } catch (const hfmm::Error&) {
        g_fail = 0;
        return 0;
    }
    return b.n;
}
extern "C" void give(void* p, size_t cap, int scope) {   // scope: 1 inside a KeepBlocks, 2 an idle one
    if (scope) {
        hfmm::KeepBlocks keep(scope == 2);
        hfmm::dev_free(p, cap, 0, false);
    } else {
        hfmm::dev_free(p, cap, 0, false);
    }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cuda = next((d for d in (os.environ.get("CUDA_HOME"), "/usr/local/cuda") if d and os.path.isdir(d)), None)
    if shutil.which("g++") is None or cuda is None:
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("devmem")
    (d / "harness.cpp").write_text(HARNESS)
    out = str(d / "harness.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", os.path.join(ROOT, "hfmm_b200", "csrc"),
                    "-I", os.path.join(cuda, "include"), str(d / "harness.cpp"), "-o", out], check=True)
    so = ctypes.CDLL(out)
    so.take.restype = ctypes.c_void_p
    so.take.argtypes = [ctypes.c_size_t, ctypes.POINTER(ctypes.c_size_t)]
    so.give.argtypes = [ctypes.c_void_p, ctypes.c_size_t, ctypes.c_int]
    so.live.restype = so.resized.restype = so.between.restype = ctypes.c_size_t
    so.between.argtypes = [ctypes.c_size_t, ctypes.c_size_t, ctypes.c_int]
    so.resized.argtypes = [ctypes.c_size_t, ctypes.c_size_t]
    return so


def _take(so, n):
    cap = ctypes.c_size_t()
    return so.take(n, ctypes.byref(cap)), cap.value


@pytest.mark.parametrize("what", [1, 2, 3])
def test_bound_holds_across_threads(lib, what):
    lib.plans(1)
    for _ in range(300):
        p, cap = _take(lib, 1 * MIB)
        lib.in_wait(what)
        lib.give(p, cap, 1)
        if what == 1:
            assert lib.live() == 0   # no plan: nothing is kept
            lib.plans(1)
    blocks = [_take(lib, 4 * MIB) for _ in range(64)]
    for p, cap in blocks:
        lib.give(p, cap, 1)
    assert 100 * MIB < lib.live() <= 128 * MIB
    n = lib.allocs()
    again = [_take(lib, 4 * MIB) for _ in range(20)]   # served from what is kept
    assert lib.allocs() == n
    for p, cap in again:
        lib.give(p, cap, 1)
    lib.plans(-1)
    assert lib.live() == 0


def test_idle_scope_keeps_without_a_wait(lib):
    lib.plans(1)
    p, cap = _take(lib, MIB)
    lib.in_wait(1)   # would end the plan, and with it the block, if the device were waited for
    lib.give(p, cap, 2)
    assert lib.live() == cap
    lib.in_wait(0)
    lib.plans(-1)
    assert lib.live() == 0


def test_outside_a_scope_nothing_is_kept(lib):
    lib.plans(1)
    p, cap = _take(lib, MIB)
    lib.in_wait(1)   # would end the plan if the device were waited for
    lib.give(p, cap, 0)
    assert lib.live() == 0
    lib.in_wait(0)
    lib.plans(-1)


@pytest.mark.parametrize("n", [1, 513, MIB - 1, 31 * MIB + 5, 32 * MIB + 1, 33 * MIB + 7, 3 << 30, (5 << 30) + 12345])
def test_block_sizes(lib, n):
    """A block that may be kept is rounded up by an eighth (512 bytes) at most, a larger one not
    at all, so that a plan near the device's memory takes what its buffers hold."""
    lib.plans(1)
    p, cap = _take(lib, n)
    before = lib.live()
    assert n <= cap <= (n + max(n // 8, 512) if n <= 32 * MIB else n) and before >= cap
    lib.give(p, cap, 0)
    lib.plans(-1)
    assert lib.live() == 0


@pytest.mark.parametrize("second", [100 * MIB, 99 * MIB, 81 * MIB, 79 * MIB, 26 * MIB, MIB, 101 * MIB])
def test_resized_buffer(lib, second):
    """A buffer asked for less keeps its block only while that is at most a quarter larger."""
    lib.plans(1)
    cap = lib.resized(100 * MIB, second)
    assert second <= cap <= second + second // 4 + 512
    lib.plans(-1)
    assert lib.live() == 0


@pytest.mark.parametrize("times,n", [(0, 2048 * MIB), (1, 1024 * MIB), (3, 256 * MIB), (4, 200 * MIB), (5, 0)])
def test_as_much_as_fits(lib, times, n):
    lib.plans(1)
    assert lib.between(200 * MIB, 2048 * MIB, times) == n and lib.between(7, 7, 0) == 7
    lib.plans(-1)
    assert lib.live() == 0
