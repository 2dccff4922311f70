"""The shared-divisor quotient of the other imaging conditions (rtm_div.cuh) rounds as the division does: its
host form against IEEE division, bit for bit."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HOST = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#define __device__
#define __host__
#define __forceinline__ inline
static float __frcp_rn(float x) { return 1.0f / x; }
static float __fmul_rn(float a, float b) { return a * b; }
static float __fdiv_rn(float a, float b) { return a / b; }
static float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
static float __int_as_float(int i) { float f; std::memcpy(&f, &i, 4); return f; }
using std::fabs;
static float fabsf_(float x) { return std::fabs(x); }
#define fabsf fabsf_
#include "rtm_div.cuh"

static uint64_t s = 88172645463325252ull;
static uint32_t next() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return (uint32_t)(s >> 16); }
int main()
{
    long bad = 0;
    const float fixed[] = {1.0f, 2.5f, 5.0f, 7.5f, 10.0f, 12.5f, 25.0f, 3.3f, 1e-3f, 0.1f, 1e3f, 1e-10f, 1e10f,
                           0.99999994f, 1.0000001f, 1.9999999f, 9.9e-11f, 1.1e10f, 1e-15f, 1e15f, 1e-40f, 3e38f};
    const int nf = sizeof(fixed) / sizeof(*fixed);
    for (int k = 0; k < nf + 60; k++) {
        // the fixed ones, then drawn ones over the range of grid spacings
        const float b = k < nf ? fixed[k] : std::exp2((float)(next() % 2000) / 100.0f - 10.0f) * (1.0f + (next() % 4096) / 8192.0f);
        const float rb = __frcp_rn(b);
        const bool takes = div_by_takes(b);   // (the kernel divides by the others)
        for (int i = 0; i < 200000; i++) {
            // every exponent and the special values, and the edges of the quick range
            float a = __int_as_float((int)next());
            if (i % 16 == 0) a = __int_as_float(0x15f79688 + (int)(next() % 64) - 32);   // about 1e-25
            if (i % 16 == 1) a = __int_as_float(0x69045951 + (int)(next() % 64) - 32);   // about 1e25
            if (i == 2) a = 0.0f;
            if (i == 3) a = -0.0f;
            if (i == 4) a = INFINITY;
            if (i == 5) a = NAN;
            const float q = takes ? div_by(a, b, rb) : a / b, w = a / b;
            if (std::memcmp(&q, &w, 4) && !(q != q && w != w)) {
                if (!bad++) std::printf("%a / %a = %a, not %a\n", a, b, w, q);
            }
        }
    }
    std::printf("%ld wrong\n", bad);
    return bad != 0;
}
"""


def test_quotients_by_a_shared_divisor_are_correctly_rounded(tmp_path):
    (tmp_path / "host.cpp").write_text(HOST)
    exe = str(tmp_path / "host")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I" + os.path.join(ROOT, "gubingluo_b200", "csrc"),
                    "-o", exe, str(tmp_path / "host.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout


# a grid spacing that the shared-divisor quotient does not take (the kernel's other instance), in a model
# scaled with it, against the oracle: the energy norm holds all four quotients
@pytest.mark.gpu
@pytest.mark.parametrize("accum", [0, 1])
def test_energy_norm_at_a_far_grid_spacing(rtmlib, oracle, accum):
    G = rtmlib
    nx, nz, h = 61, 41, 1.5e10
    rng = np.random.default_rng(1)
    v = (1e9 * (2700 + 9 * np.arange(nz)[:, None] + 225 * rng.random((nz, nx)))).astype(np.float32)
    rho = np.full((nz, nx), 2000, np.float32)
    s = G.SurveyConfig(nx=nx, nz=nz, nt=130, dx=h, dz=h, dt=float(np.float32(1e-3)), npml=20, fdom=25.0, layout=2,
                       spx0=0.0, spz0=2 * h, dspx=0.0, mode=0, mute=0, amp=1.0e4, alp=1.0 / h)
    got = G.migrate(s, G.RunOptions(extra_images=1, accum_fp64=accum), [1], v, rho)
    want = oracle.rtm_model({k: getattr(s, k) for k in s.__dataclass_fields__}, [1], v, rho, extra=1)
    for k in ("image1", "image5s", "image5m"):   # the tolerance of test_gpu_parity
        a, b = got[k].astype(np.float64), want[k].astype(np.float64)
        assert np.linalg.norm(b) > 0 and np.linalg.norm(a - b) <= 1e-4 * np.linalg.norm(b), k
