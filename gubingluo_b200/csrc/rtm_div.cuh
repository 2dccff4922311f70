// rtm_div.cuh — quotients by a divisor that many cells share, correctly rounded.
#pragma once

// Divisors that div_by takes: nearer to 1 than its quotients' range, so that none leaves the normal numbers.
__host__ __device__ inline bool div_by_takes(float b) { return b >= 1.0e-10f && b <= 1.0e10f; }

// RN(a / b) given rb = RN(1 / b): two of Markstein's correction steps (exact residual by a fused
// multiply-add; a faithful quotient so corrected is the rounded one), in the range where no residual
// underflows; zero, which sends the library's division down its slow branch, is itself.
__device__ __forceinline__ float div_by(float a, float b, float rb)
{
    if (fabsf(a) >= 1.0e-25f && fabsf(a) < 1.0e25f) {
        float q = __fmul_rn(a, rb);
        q = __fmaf_rn(__fmaf_rn(-q, b, a), rb, q);
        return __fmaf_rn(__fmaf_rn(-q, b, a), rb, q);
    }
    return a == 0.0f ? a : __fdiv_rn(a, b);
}
