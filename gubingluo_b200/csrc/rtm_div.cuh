// rtm_div.cuh — quotients by a divisor that many cells share, correctly rounded.
#pragma once

// A divisor b > 0 with its reciprocal, and the smallest |a| that div_by takes without the library's division
// (infinity where b is too far from 1: the quotient could leave the range of normal numbers).
struct Divisor {
    float b, rb, lo;
};
__device__ __forceinline__ Divisor divisor(float b)
{
    return {b, __frcp_rn(b), b >= 1.0e-10f && b <= 1.0e10f ? 1.0e-25f : __int_as_float(0x7f800000)};
}

// RN(a / b): two of Markstein's correction steps (exact residual by a fused multiply-add; a faithful quotient
// so corrected is the rounded one), in the range where no residual underflows; zero, which sends the
// library's division down its slow branch, is itself.
__device__ __forceinline__ float div_by(float a, const Divisor &d)
{
    if (fabsf(a) >= d.lo && fabsf(a) < 1.0e25f) {
        float q = __fmul_rn(a, d.rb);
        q = __fmaf_rn(__fmaf_rn(-q, d.b, a), d.rb, q);
        return __fmaf_rn(__fmaf_rn(-q, d.b, a), d.rb, q);
    }
    return a == 0.0f ? a : __fdiv_rn(a, d.b);
}
