"""Kept workspaces of the gather resampling (rtm_interp.cu) beside other shapes and callers."""
import os
import shutil
import subprocess
import threading

import numpy as np
import pytest


def _survey(G, nx, nt):
    return G.SurveyConfig(nx=nx, nz=60, nt=nt, dx=10.0, dz=10.0, dt=float(np.float32(1e-3)), npml=12, fdom=25.0,
                          layout=2, spx0=100.0, spz0=20.0, dspx=10.0, mode=1, mute=0)


def _models(nx):
    return np.full((60, nx), 2000, np.float32), np.full((60, nx), 2000, np.float32)


def _record(nt0, nx0, seed):
    return np.random.default_rng(seed).standard_normal((nt0, nx0)).astype(np.float32)


# a session's kept plan of the longest transforms, then a shorter shape's plan (alone, and another
# session's), then the kept one again: transforms of 8192, 4096 and 1024 points against 128
@pytest.mark.gpu
@pytest.mark.parametrize("nt0", [4096, 1500, 500])
def test_a_kept_plan_survives_a_shorter_one(rtmlib, nt0):
    G = rtmlib
    nx0, nx = 61, 121
    v, rho = _models(nx)
    obs, short = _record(nt0, nx0, nt0), _record(60, 10, 1)
    with G.Session(_survey(G, nx, nt0), G.RunOptions(), [1], v, rho) as ss:
        ss.set_gather_raw(0, obs, 1e-3)
        want = ss.gather(0)
        assert np.abs(want).max() > 0
        G.interp_gather(short, 19, 60, 1e-3, 1e-3)
        ss.set_gather_raw(0, obs, 1e-3)
        assert np.array_equal(ss.gather(0), want)
        vs, rs = _models(19)
        with G.Session(_survey(G, 19, 60), G.RunOptions(), [1], vs, rs) as other:
            other.set_gather_raw(0, short, 1e-3)
            ss.set_gather_raw(0, obs, 1e-3)
        assert np.array_equal(ss.gather(0), want)


@pytest.mark.gpu
def test_plans_of_two_lengths_in_two_threads(rtmlib):
    G = rtmlib
    shapes = [(1500, 41, 81), (60, 10, 19)]
    want = [G.interp_gather(_record(nt0, nx0, nt0), nx, nt0, 1e-3, 1e-3) for nt0, nx0, nx in shapes]
    errors = []

    def work(k):
        nt0, nx0, nx = shapes[k]
        obs = _record(nt0, nx0, nt0)
        try:
            for _ in range(40):
                assert np.array_equal(G.interp_gather(obs, nx, nt0, 1e-3, 1e-3), want[k])
        except Exception as e:   # (a thread's failure must reach the test)
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


# calls of the library's own C++ entry to the resampling, which Python does not reach: argv[1] names
# the check, and the result of a fresh plan is what every other call must give
OWN_ENTRY = r"""
#include <cuda_runtime.h>
#include <dlfcn.h>

#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "rtm_internal.h"

static int fail_next = 0;
extern "C" cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v)   // before the runtime's
{
    typedef cudaError_t (*Fn)(const void *, cudaFuncAttribute, int);
    if (fail_next) {
        fail_next--;
        return cudaErrorInvalidValue;
    }
    return ((Fn)dlsym(RTLD_NEXT, "cudaFuncSetAttribute"))(f, a, v);
}

int main(int, char **argv)
{
    const std::string what = argv[1];
    const int nx0 = 41, nt0 = 1500, nx = 81, nt = 1500;
    const float dt = 1e-3f;
    const size_t n = (size_t)nt * nx;
    std::vector<float> in((size_t)nx0 * nt0), want(n), got(n);
    for (size_t i = 0; i < in.size(); i++) in[i] = (float)((i * 2654435761u >> 8) % 1000) / 1000.0f - 0.5f;
    cudaStream_t st;
    if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking)) return 2;
    float *out;
    if (cudaMalloc(&out, 4 * n)) return 2;
    rtm::InterpPlan fresh, p;
    const auto run = [&](rtm::InterpPlan &q, float *to) {
        return rtm::interp_gather_device(q, in.data(), nx0, nt0, to, nx, nt, dt, dt, 0, st, nullptr);
    };
    const auto read = [&](std::vector<float> &v, const float *from) {
        return cudaMemcpyAsync(v.data(), from, 4 * n, cudaMemcpyDeviceToHost, st) == cudaSuccess &&
               cudaStreamSynchronize(st) == cudaSuccess;
    };
    if (run(fresh, out) || !read(want, out)) return 2;
    const float *from = out;
    if (what == "own result") {   // a plan made for a caller's buffer, then asked for one of its own
        if (run(p, out)) return 3;
        if (run(p, nullptr)) return 4;
        from = p.d_out;
        if (!from) return 5;
    } else if (what == "interrupted") {   // a plan that failed half way, then asked again
        fail_next = 1;
        if (!run(p, out)) return 3;
        if (run(p, out)) return 4;
    }
    if (!read(got, from)) return 6;
    p.release();
    fresh.release();
    std::puts(std::memcmp(got.data(), want.data(), 4 * n) ? "different" : "same");
    return 0;
}
"""


@pytest.fixture(scope="module")
def own_entry(rtmlib, tmp_path_factory):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    lib = os.path.join(root, "gubingluo_b200")
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc")))
    d = tmp_path_factory.mktemp("own_entry")
    (d / "own.cpp").write_text(OWN_ENTRY)
    subprocess.run(["g++", "-std=c++17", "-O1", "-rdynamic", "-I" + os.path.join(root, "include"),
                    "-I" + os.path.join(lib, "csrc"), "-I" + cuda + "/include", "-o", str(d / "own"), str(d / "own.cpp"),
                    os.path.join(lib, "librtm_b200.so"), "-L" + cuda + "/lib64", "-lcudart", "-ldl",
                    "-Wl,-rpath," + lib, "-Wl,-rpath," + cuda + "/lib64"], check=True)
    return str(d / "own")


@pytest.mark.gpu
def test_a_plan_without_room_for_the_result_is_not_asked_for_it(own_entry):
    r = subprocess.run([own_entry, "own result"], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "same", (r.returncode, r.stderr)


@pytest.mark.gpu
def test_a_plan_that_failed_half_way_is_made_again(own_entry):
    r = subprocess.run([own_entry, "interrupted"], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "same", (r.returncode, r.stderr)


# a result of 200 GB: refused with the code for memory, and the next call is as if nothing had been
@pytest.mark.gpu
def test_a_result_beyond_the_device_memory_is_refused(rtmlib):
    import ctypes as C

    G = rtmlib
    obs = _record(10, 25, 0)
    want = G.interp_gather(obs, 49, 20, 1e-3, 2e-3)
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    out = np.zeros(25, np.float32)   # (never written: the call fails before)
    rc = G.lib().rtm_interp_gather(p(obs), 25, 10, p(out), 25, 2_000_000_000, 1e-3, 2e-3, 0, 0)
    assert rc == -4 and b"alloc" in G.lib().rtm_last_error()
    assert np.array_equal(G.interp_gather(obs, 49, 20, 1e-3, 2e-3), want)


# odd and even counts of traces in and out (two share a transform in time), a pair whose traces differ by
# 1e5 in size, and lengths in x whose power of two (16 to 8192 points) takes every order of passes
@pytest.mark.gpu
@pytest.mark.parametrize("nx0,nt0,lx", [(2, 9, 2), (3, 40, 2), (4, 41, 3), (5, 8, 4), (17, 30, 3), (33, 60, 5),
                                        (65, 130, 2), (129, 20, 3), (250, 30, 4), (512, 21, 4), (1300, 12, 3), (2, 10, 300),
                                        (3, 12, 64)])
@pytest.mark.parametrize("mirror", [0, 1])
def test_pairs_of_traces_and_every_order_of_passes(rtmlib, nx0, nt0, lx, mirror):
    from test_fk import _fk

    obs = _record(nt0, nx0, nx0 * lx) * np.where(np.arange(nx0) % 4 == 1, 1e-5, 1.0).astype(np.float32)
    nx = lx * (nx0 - 1) + 1
    got = rtmlib.interp_gather(obs, nx, nt0, 1e-3, 1e-3, mirror)
    want = _fk(obs, nx, lx, mirror)
    # as test_fk: float32 rounding of the result and of max|Z|
    assert np.linalg.norm(got - want) < 1e-6 * np.linalg.norm(want)
