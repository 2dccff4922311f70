"""The host side of the read-back (rtm_copy.cu) against a stand-in for the CUDA runtime in which device
memory is host memory and allocations can be made to fail: no GPU is used."""
import ctypes as C
import os
import shutil
import subprocess
import threading

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "gubingluo_b200", "csrc")

FAKE = r"""
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <mutex>
#include <set>
#include <string>

// what the test sets and reads
extern "C" {
int alloc_left = -1, streams_left = -1;   // successes left (-1: no limit)
int allocs = 0, stale = 0, live = 0;                        // calls that succeeded; uses of a lost handle
unsigned long long context = 1;                             // a reset makes a new one
}
namespace rtm {
int fail(int rc, const std::string &) { return rc; }
bool host_team() { return true; }
int copy_out(void *, const void *, size_t, size_t, size_t, bool);
}

namespace {
std::recursive_mutex mu;
thread_local int device = 0;
thread_local cudaStream_t launch_stream;
std::set<void *> handles;   // live streams and page-locked blocks
void *make(size_t n)
{
    std::lock_guard<std::recursive_mutex> l(mu);
    void *p = std::malloc(n);
    handles.insert(p);
    return p;
}
bool known(void *p)
{
    std::lock_guard<std::recursive_mutex> l(mu);
    if (!handles.count(p)) stale++;
    return handles.count(p) != 0;
}
bool spend(int &left)
{
    std::lock_guard<std::recursive_mutex> l(mu);
    if (left == 0) return false;
    if (left > 0) left--;
    return true;
}
CUresult ctx_get_id(CUcontext, unsigned long long *id)
{
    *id = context;
    return CUDA_SUCCESS;
}
}

extern "C" {
int copy(void *dst, const void *src, size_t pitch, size_t row, size_t rows, int narrow)
{
    return rtm::copy_out(dst, src, pitch, row, rows, narrow != 0);
}
void use_device(int d) { device = d; }
void reset_device()   // everything made so far is gone (the memory itself is kept, so that a stale use is seen)
{
    std::lock_guard<std::recursive_mutex> l(mu);
    handles.clear();
    context++;
}

cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { device = d; return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned)
{
    if (!spend(alloc_left)) return cudaErrorMemoryAllocation;
    *p = make(n);
    std::lock_guard<std::recursive_mutex> l(mu);
    allocs++;
    live++;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p)
{
    if (!known(p)) return cudaErrorInvalidValue;
    std::lock_guard<std::recursive_mutex> l(mu);
    handles.erase(p);
    live--;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned)
{
    if (!spend(streams_left)) return cudaErrorMemoryAllocation;
    *s = (cudaStream_t)make(1);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s)
{
    if (!known(s)) return cudaErrorContextIsDestroyed;
    std::lock_guard<std::recursive_mutex> l(mu);
    handles.erase(s);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return known(s) ? cudaSuccess : cudaErrorContextIsDestroyed; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st)
{
    if (!known(st) || !known(d)) return cudaErrorContextIsDestroyed;
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2D(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, cudaMemcpyKind)
{
    if (w > dp || w > sp) return cudaErrorInvalidValue;
    for (size_t i = 0; i < h; i++) std::memcpy((char *)d + i * dp, (const char *)s + i * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, cudaMemcpyKind k, cudaStream_t st)
{
    return known(st) && known(d) ? cudaMemcpy2D(d, dp, s, sp, w, h, k) : cudaErrorContextIsDestroyed;
}
cudaError_t cudaLaunchKernel(const void *, dim3, dim3, void **args, size_t, cudaStream_t st)   // the narrowing kernel
{
    float *d = *(float **)args[1];
    if (!known(st) || !known(d)) return cudaErrorContextIsDestroyed;
    const double *s = *(const double **)args[0];
    for (int i = 0; i < *(int *)args[2]; i++) d[i] = (float)s[i];
    return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPoint(const char *, void **f, unsigned long long, cudaDriverEntryPointQueryResult *q)
{
    *f = (void *)ctx_get_id;
    if (q) *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
// what compiled kernels call
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, cudaStream_t st) { launch_stream = st; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *m, void *st)
{
    *g = *b = dim3(1);
    *m = 0;
    *(cudaStream_t *)st = launch_stream;
    return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {}
}
"""


@pytest.fixture(scope="module")
def build(tmp_path_factory):
    if not shutil.which("nvcc"):
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("readback")
    (d / "fake.cpp").write_text(FAKE)
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(shutil.which("nvcc")))), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-I" + cuda, "-c", str(d / "fake.cpp"), "-o", str(d / "fake.o")],
                   check=True)
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O1", "-Xcompiler", "-fPIC",
                    "-Xcompiler", "-fopenmp", "-I" + os.path.join(ROOT, "include"), "-I" + CSRC, "-c",
                    os.path.join(CSRC, "rtm_copy.cu"), "-o", str(d / "copy.o")], check=True)
    so = str(d / "libreadback.so")
    subprocess.run(["g++", "-shared", "-fopenmp", "-Wl,-Bsymbolic", "-o", so, str(d / "fake.o"), str(d / "copy.o")], check=True)
    return so


@pytest.fixture
def rb(build, tmp_path):
    """A fresh copy of the library for each test (its pool is process state)."""
    so = str(tmp_path / "libreadback.so")
    shutil.copy(build, so)
    L = C.CDLL(so)
    L.copy.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_size_t, C.c_size_t, C.c_int]
    return L


def _var(L, name):
    return C.c_int.in_dll(L, name)


def _copies(L, seed=0):
    """Contiguous, narrowed and pitched copies of several chunks of 1 MB (the last one partial), and one of
    rows longer than a chunk."""
    rng = np.random.default_rng(seed)
    a = rng.standard_normal(1_300_001).astype(np.float32)
    got = np.zeros_like(a)
    assert L.copy(got.ctypes.data, a.ctypes.data, a.nbytes, a.nbytes, 1, 0) == 0
    assert np.array_equal(got, a)
    w = rng.standard_normal(700_003)
    n = np.zeros(w.size, np.float32)
    assert L.copy(n.ctypes.data, w.ctypes.data, n.nbytes, n.nbytes, 1, 1) == 0
    assert np.array_equal(n, w.astype(np.float32))
    for rows, width, pitch in ((1201, 501, 512), (3, 300_000, 300_032)):
        f = rng.standard_normal((rows, pitch)).astype(np.float32)
        g = np.zeros((rows, width), np.float32)
        assert L.copy(g.ctypes.data, f.ctypes.data, 4 * pitch, 4 * width, rows, 0) == 0
        assert np.array_equal(g, f[:, :width])


# no page-locked memory at all, for one lane, for three; the same for streams
@pytest.mark.parametrize("what", ["alloc_left", "streams_left"])
@pytest.mark.parametrize("left", [0, 1, 3])
def test_copies_without_page_locked_memory_or_streams(rb, what, left):
    _var(rb, what).value = left
    for seed in range(3):
        _copies(rb, seed)
    assert _var(rb, "stale").value == 0


def test_each_device_keeps_its_own_lanes(rb):
    for d in (0, 1, 2, 0, 1, 2):
        rb.use_device(d)
        _copies(rb, d)
    assert _var(rb, "allocs").value == _var(rb, "live").value <= 3 * 4   # none was freed again


def test_copies_of_several_threads_leave_at_most_four_lanes(rb):
    errors = []

    def work(k):
        try:
            for _ in range(4):
                _copies(rb, k)
        except BaseException as e:   # (a thread's failure must reach the test)
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert _var(rb, "live").value <= 4 and _var(rb, "stale").value == 0


def test_lanes_lost_in_a_device_reset_are_not_used_again(rb):
    _copies(rb)
    rb.reset_device()
    _copies(rb, 1)
    assert _var(rb, "stale").value == 0
