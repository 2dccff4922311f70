// rtm_fk.cuh — the F-K step of the gather resampling (reference GeneralFKinterp,
// Interp_function.cpp:53-244) on transforms of its own, in double precision.
//
// The reference transforms the gather zero-padded to [lx nx0][lx nt0] and works on the folded
// spectrum.  Its padded transform splits into lx x lx modulated transforms of the unpadded
// sizes: frequency lx q + r of the padded length is frequency q of the samples times
// exp(-2 pi i r n / (lx n0)).  So no padded array is formed, the unpadded transform K is the
// r = 0 part, the fold Z is the transform of every lx-th trace, and time frequencies above the
// Nyquist row are never computed (real input).
//
// Sizes are arbitrary (recorded shots rarely have a power of two), so each transform of length N
// is a chirp convolution (Bluestein's algorithm: nk = (n^2 + k^2 - (k-n)^2) / 2) by power-of-two
// transforms of length M >= 2 N - 1 in shared memory: radix-4 decimation in frequency forwards,
// the product with the chirp's spectrum in that digit-reversed order, and decimation in time
// back, so nothing is reordered.  Phases come from exact integers modulo the period and
// sincospi, once per plan; the errors stay at the 1e-15 of the double-precision library transforms.
// Two real traces share a time transform each way.
//
// Why not cuFFT here: a gather takes 0.2 ms, creating the four plans it needed 7.3 ms, which
// every stand-alone call and every new session paid (241 traces x 2000 samples, lx = 2: 7.3 ms a
// call -> 1.9 ms).
// What bounds the kernels: passes over the M points in shared memory at 16 warps per SM (registers), a
// third of that memory's rate.  So a pass takes two radix-4 levels, 16 points of a thread in registers,
// the middle one the last levels, the product with the spectrum and the first levels back, the first
// reads its input and the last writes its result: 6 passes at M = 8192 (one level a pass, one trace a
// transform and the phases worked out in place took 16).  A shot in a session with its upload, ms,
// cuFFT / one level a pass / now: 241 traces x 2000 samples, lx = 2, 0.35 / 0.39 / 0.25; x 4000 0.65 / 0.83 / 0.50;
// 400 x 4000, lx = 4, 1.43 / 2.23 / 1.25; 1024 x 4096, lx = 4, 3.7 / 5.9 / 2.9; 400 x 700, lx = 2, 0.19 / 0.30 / 0.19;
// cuFFT is ahead for few long traces, where a launch has fewer blocks than SMs: 60 x 4000 0.17 / - / 0.20.
#pragma once
#include <cuda_runtime.h>

namespace rtm {
namespace fk {

constexpr int kMaxN = 4096;   // longest transform: M = 8192 points, 144 KB of shared memory

__host__ __device__ inline int pow2_for(int n)   // M of a transform of length n
{
    int m = 16;
    while (m < 2 * n - 1) m *= 2;
    return m;
}
// The points are kept in shared memory with one slot of padding every 8 (M an odd power of two) or 16,
// the points that a thread takes in the middle pass, so that no pass has bank conflicts.
__host__ __device__ inline int pad_shift(int m)
{
    int k = 0;
    while (m >> k > 1) k++;
    return k & 1 ? 3 : 4;
}
inline size_t smem_bytes(int m) { return (size_t)(m + (m >> pad_shift(m))) * sizeof(double2); }
// Threads of a block: one group of 16 points each per pass, whole warps.
inline int threads(int m) { return m / 16 > 512 ? 512 : m / 16 < 32 ? 32 : m / 16; }

__device__ __forceinline__ double2 cmul(double2 a, double2 b)
{
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 conj2(double2 a) { return make_double2(a.x, -a.y); }
// exp(-i pi num / den), num reduced modulo the period 2 den first (exact)
__device__ __forceinline__ double2 unit(long long num, long long den)
{
    num %= 2 * den;
    double s, c;
    sincospi((double)num / (double)den, &s, &c);
    return make_double2(c, -s);
}

// Twiddles exp(-2 pi i k / mt), k < mt / 4; mt: the longest power of two in use.
__global__ void k_twiddles(double2 *tw, int mt)
{
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < mt / 4; k += gridDim.x * blockDim.x) tw[k] = unit(2LL * k, mt);
}

// Radix-4 butterflies of one level, decimation in frequency forwards and in time back; w: the
// level's twiddle of the butterfly.
__device__ __forceinline__ void fwd4(double2 &p0, double2 &p1, double2 &p2, double2 &p3, double2 w)
{
    const double2 s02 = cadd(p0, p2), d02 = csub(p0, p2), s13 = cadd(p1, p3), d13 = csub(p1, p3);
    const double2 w2 = cmul(w, w), w3 = cmul(w2, w);
    p0 = cadd(s02, s13);
    p1 = cmul(make_double2(d02.x + d13.y, d02.y - d13.x), w);   // d02 - i d13
    p2 = cmul(csub(s02, s13), w2);
    p3 = cmul(make_double2(d02.x - d13.y, d02.y + d13.x), w3);  // d02 + i d13
}
__device__ __forceinline__ void inv4(double2 &p0, double2 &p1, double2 &p2, double2 &p3, double2 w)
{
    const double2 w2 = cmul(w, w), w3 = cmul(w2, w);
    const double2 b0 = p0, b1 = cmul(p1, w), b2 = cmul(p2, w2), b3 = cmul(p3, w3);
    const double2 s02 = cadd(b0, b2), d02 = csub(b0, b2), s13 = cadd(b1, b3), d13 = csub(b1, b3);
    p0 = cadd(s02, s13);
    p1 = make_double2(d02.x - d13.y, d02.y + d13.x);   // d02 + i d13
    p2 = csub(s02, s13);
    p3 = make_double2(d02.x + d13.y, d02.y - d13.x);
}
// The same without a twiddle (level 4) and the radix-2 butterfly.
__device__ __forceinline__ void fwd4(double2 &p0, double2 &p1, double2 &p2, double2 &p3)
{
    const double2 s02 = cadd(p0, p2), d02 = csub(p0, p2), s13 = cadd(p1, p3), d13 = csub(p1, p3);
    p0 = cadd(s02, s13);
    p1 = make_double2(d02.x + d13.y, d02.y - d13.x);
    p2 = csub(s02, s13);
    p3 = make_double2(d02.x - d13.y, d02.y + d13.x);
}
__device__ __forceinline__ void inv4(double2 &p0, double2 &p1, double2 &p2, double2 &p3)
{
    const double2 s02 = cadd(p0, p2), d02 = csub(p0, p2), s13 = cadd(p1, p3), d13 = csub(p1, p3);
    p0 = cadd(s02, s13);
    p1 = make_double2(d02.x - d13.y, d02.y + d13.x);
    p2 = csub(s02, s13);
    p3 = make_double2(d02.x + d13.y, d02.y - d13.x);
}
__device__ __forceinline__ void both2(double2 &p0, double2 &p1)
{
    const double2 s = cadd(p0, p1), d = csub(p0, p1);
    p0 = s;
    p1 = d;
}

// A pass over the m points of a block: ld(i) of every point, butterflies, st(i, value).  pass16 takes the
// levels n and n / 4 together, 16 points of stride n / 16 in registers; pass4 the level n alone.
// FWD: frequency decimation (level n first); else time decimation (level n last).
template <bool FWD, typename Ld, typename St>
__device__ __forceinline__ void pass16(int m, int n, const double2 *__restrict__ tw, int mt, Ld ld, St st)
{
    const int h = n / 16, ts = mt / n;
    for (int g = threadIdx.x; g < m / 16; g += blockDim.x) {
        const int j = g & (h - 1), base = (g - j) * 16 + j;
        double2 v[4][4];   // point base + (4 q + s) h
#pragma unroll
        for (int k = 0; k < 16; k++) v[k / 4][k % 4] = ld(base + k * h);
        const double2 wq = FWD ? tw[4 * j * ts] : conj2(tw[4 * j * ts]);
        if (!FWD)
#pragma unroll
            for (int q = 0; q < 4; q++) inv4(v[q][0], v[q][1], v[q][2], v[q][3], wq);
#pragma unroll
        for (int s = 0; s < 4; s++) {
            const double2 w = tw[(j + s * h) * ts];
            if (FWD) fwd4(v[0][s], v[1][s], v[2][s], v[3][s], w);
            else inv4(v[0][s], v[1][s], v[2][s], v[3][s], conj2(w));
        }
        if (FWD)
#pragma unroll
            for (int q = 0; q < 4; q++) fwd4(v[q][0], v[q][1], v[q][2], v[q][3], wq);
#pragma unroll
        for (int k = 0; k < 16; k++) st(base + k * h, v[k / 4][k % 4]);
    }
}
template <bool FWD, typename Ld, typename St>
__device__ __forceinline__ void pass4(int m, int n, const double2 *__restrict__ tw, int mt, Ld ld, St st)
{
    const int h = n / 4, ts = mt / n;
    for (int g = threadIdx.x; g < m / 4; g += blockDim.x) {
        const int j = g & (h - 1), base = (g - j) * 4 + j;
        double2 v[4];
#pragma unroll
        for (int k = 0; k < 4; k++) v[k] = ld(base + k * h);
        const double2 w = FWD ? tw[j * ts] : conj2(tw[j * ts]);
        if (FWD) fwd4(v[0], v[1], v[2], v[3], w);
        else inv4(v[0], v[1], v[2], v[3], w);
#pragma unroll
        for (int k = 0; k < 4; k++) st(base + k * h, v[k]);
    }
}
// The last levels forwards (16 and 4, or 8 and 2), turn(i, value) on every point of the spectrum, in its
// digit-reversed order, and with BACK the same levels back.
template <bool BACK, typename Ld, typename Turn, typename St>
__device__ __forceinline__ void pass_turn(int m, bool odd, const double2 *__restrict__ tw, int mt, Ld ld, Turn turn, St st)
{
    if (odd) {
        const double2 w1 = tw[mt / 8];
        for (int g = threadIdx.x; g < m / 8; g += blockDim.x) {
            double2 v[8];
#pragma unroll
            for (int k = 0; k < 8; k++) v[k] = ld(8 * g + k);
            fwd4(v[0], v[2], v[4], v[6]);
            fwd4(v[1], v[3], v[5], v[7], w1);
#pragma unroll
            for (int k = 0; k < 8; k += 2) both2(v[k], v[k + 1]);
#pragma unroll
            for (int k = 0; k < 8; k++) v[k] = turn(8 * g + k, v[k]);
            if (!BACK) continue;
#pragma unroll
            for (int k = 0; k < 8; k += 2) both2(v[k], v[k + 1]);
            inv4(v[0], v[2], v[4], v[6]);
            inv4(v[1], v[3], v[5], v[7], conj2(w1));
#pragma unroll
            for (int k = 0; k < 8; k++) st(8 * g + k, v[k]);
        }
        return;
    }
    for (int g = threadIdx.x; g < m / 16; g += blockDim.x) {
        double2 v[16];
#pragma unroll
        for (int k = 0; k < 16; k++) v[k] = ld(16 * g + k);
        fwd4(v[0], v[4], v[8], v[12]);
#pragma unroll
        for (int j = 1; j < 4; j++) fwd4(v[j], v[j + 4], v[j + 8], v[j + 12], tw[j * (mt / 16)]);
#pragma unroll
        for (int k = 0; k < 16; k += 4) fwd4(v[k], v[k + 1], v[k + 2], v[k + 3]);
#pragma unroll
        for (int k = 0; k < 16; k++) v[k] = turn(16 * g + k, v[k]);
        if (!BACK) continue;
#pragma unroll
        for (int k = 0; k < 16; k += 4) inv4(v[k], v[k + 1], v[k + 2], v[k + 3]);
        inv4(v[0], v[4], v[8], v[12]);
#pragma unroll
        for (int j = 1; j < 4; j++) inv4(v[j], v[j + 4], v[j + 8], v[j + 12], conj2(tw[j * (mt / 16)]));
#pragma unroll
        for (int k = 0; k < 16; k++) st(16 * g + k, v[k]);
    }
}
// The block's transform of in(i), i < m, turned by turn in its spectrum and, with BACK, taken back (times
// m) into out(i, value).  x: shared memory.  The first pass reads in() and the last one writes out()
// themselves.
template <bool BACK, typename In, typename Turn, typename Out>
__device__ __forceinline__ void transform(double2 *x, int m, const double2 *__restrict__ tw, int mt, In in, Turn turn, Out out)
{
    const int sh = pad_shift(m), mid = sh == 3 ? 8 : 16;
    const auto ld = [&](int i) { return x[i + (i >> sh)]; };
    const auto st = [&](int i, double2 v) { x[i + (i >> sh)] = v; };
    int n = m;
    for (; n > mid; n /= n / 4 > mid ? 16 : 4) {
        if (n / 4 > mid) {
            if (n == m) pass16<true>(m, n, tw, mt, in, st);
            else pass16<true>(m, n, tw, mt, ld, st);
        } else {
            if (n == m) pass4<true>(m, n, tw, mt, in, st);
            else pass4<true>(m, n, tw, mt, ld, st);
        }
        __syncthreads();
    }
    if (m == mid) {
        pass_turn<BACK>(m, mid == 8, tw, mt, in, turn, out);
        return;
    }
    pass_turn<BACK>(m, mid == 8, tw, mt, ld, turn, st);
    if (!BACK) return;
    // the levels above the middle came in pairs but for the lowest of an odd number
    int levels = 0;
    for (n = mid; n < m; n *= 4) levels++;
    n = mid;
    if (levels & 1) {
        n *= 4;
        __syncthreads();
        if (n == m) pass4<false>(m, n, tw, mt, ld, out);
        else pass4<false>(m, n, tw, mt, ld, st);
    }
    while (n < m) {
        n *= 16;
        __syncthreads();
        if (n == m) pass16<false>(m, n, tw, mt, ld, out);
        else pass16<false>(m, n, tw, mt, ld, st);
    }
}

// Spectra of the chirps exp(+i pi n^2 / N), |n| < N, wrapped to M points, over M: block b for
// length len[b], into out[b].
struct ChirpArgs {
    int len[3];
    double2 *out[3];
};
__global__ void __launch_bounds__(512) k_chirps(ChirpArgs a, const double2 *tw, int mt)
{
    extern __shared__ double2 x[];
    const int n = a.len[blockIdx.x], m = pow2_for(n);
    const double f = 1.0 / m;
    double2 *o = a.out[blockIdx.x];
    transform<false>(
        x, m, tw, mt,
        [&](int i) {
            const int d = i < n ? i : m - i < n ? m - i : -1;
            return d < 0 ? make_double2(0.0, 0.0) : conj2(unit((long long)d * d, n));
        },
        [&](int i, double2 v) {
            o[i] = make_double2(v.x * f, v.y * f);
            return v;
        },
        [](int, double2) {});
}

// Phases of the transforms of a length: [parts][len], element i of part r the chirp exp(-i pi i^2 / len)
// times exp(-2 pi i r i / (parts len)).  Every transform of a plan reads them.
struct PhaseArgs {
    int len[3], parts[3];
    double2 *out[3];
};
__global__ void k_phases(PhaseArgs a)
{
    const int n = a.len[blockIdx.y], lx = a.parts[blockIdx.y], all = lx * n;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < all; e += gridDim.x * blockDim.x) {
        const int r = e / n, i = e % n;
        a.out[blockIdx.y][e] = unit(((long long)lx * i + 2 * r) * i, (long long)lx * n);
    }
}

// The block's transform of length n of in(i), i < n: out(k, X[k]) for k < kmax.  X[k] is frequency
// k + r / parts of the samples (r = 0: the plain transform); ph: the length's phases.
template <typename In, typename Out>
__device__ __forceinline__ void chirp_dft(double2 *x, int n, int r, const double2 *__restrict__ ph,
                                          const double2 *__restrict__ chirp, const double2 *__restrict__ tw, int mt,
                                          int kmax, In in, Out out)
{
    const double2 *__restrict__ phr = ph + (size_t)r * n;
    transform<true>(
        x, pow2_for(n), tw, mt, [&](int i) { return i < n ? cmul(in(i), phr[i]) : make_double2(0.0, 0.0); },
        [&](int i, double2 v) { return cmul(v, chirp[i]); },
        [&](int k, double2 v) {
            if (k < kmax) out(k, cmul(v, ph[k]));
        });
    __syncthreads();
}

struct FkArgs {
    const float *in;              // [nt0][nx0]
    int nx0, nt0, nx, lx, Nx, Nt, nf, nh;   // nh = Nt / 2 + 1 time frequencies of the padded gather
    int rows, mirror;             // rows written of the result
    double2 *A;                   // [Nt][(nx0 + 1) / 2]: time spectra of pairs of traces
    double2 *K, *S, *Z;           // [nf][nx0], [nf][Nx], [nf][nx0]
    double2 *G;                   // [nf][nx]: filtered, back in x
    unsigned *zmax;
    const double2 *ct, *cx, *cX;  // chirp spectra of lengths nt0, nx0, Nx
    const double2 *pt, *px, *pX;  // their phases, of lx, lx and 1 parts
    const double2 *tw;
    int mt;
    float *out;                   // [rows][nx]
};

// Time transforms: block (pair of traces, r), frequencies lx q + r of the padded length.  Two real
// traces are the real and imaginary parts of one transform; trace_at takes them apart.
__global__ void __launch_bounds__(512) k_fk_time(const FkArgs a)
{
    extern __shared__ double2 x[];
    const int pair = blockIdx.x, ix = 2 * pair, r = blockIdx.y, np = gridDim.x;
    const bool two = ix + 1 < a.nx0;
    chirp_dft(
        x, a.nt0, r, a.pt, a.ct, a.tw, a.mt, a.nt0,
        [&](int i) {
            const float *s = a.in + (size_t)i * a.nx0 + ix;
            return make_double2((double)s[0], two ? (double)s[1] : 0.0);
        },
        [&](int q, double2 v) { a.A[(size_t)(a.lx * q + r) * np + pair] = v; });
}
// Frequency kt of trace i: of the pair's transform X, (X(kt) + conj X(-kt)) / 2 or (X(kt) - conj X(-kt)) / 2i.
__device__ __forceinline__ double2 trace_at(const double2 *row, const double2 *mirrored, int i)
{
    const double2 u = row[i >> 1], w = mirrored[i >> 1];
    return i & 1 ? make_double2(0.5 * (u.y + w.y), 0.5 * (w.x - u.x)) : make_double2(0.5 * (u.x + w.x), 0.5 * (u.y - w.y));
}

// |z| as the reference's fftw_fabs: sqrtf of the float-rounded double re^2 + im^2.
__device__ __forceinline__ float cabs_f(double re, double im)
{
    return sqrtf(__double2float_rn(__dadd_rn(__dmul_rn(re, re), __dmul_rn(im, im))));
}

// Space transforms, one per block: first the folds Z of every time frequency kt (kept below nf) and the
// max |Z| over all of them (non-negative floats order like their bits); then the frequencies lx k + r of S for
// kt below nf; then K's rows, part 0 at every lx-th frequency, that are not below nf (those that are
// come with S).
__host__ __device__ inline int space_blocks(int nh, int nf, int lx) { return nh + nf * lx + nf - (nf + lx - 1) / lx; }
__global__ void __launch_bounds__(512) k_fk_space(const FkArgs a)
{
    extern __shared__ double2 x[];
    int kt = blockIdx.x, r = 0;
    const bool fold = kt < a.nh;
    if (!fold) {
        kt -= a.nh;
        if (kt < a.nf * a.lx) {
            r = kt % a.lx;
            kt /= a.lx;
        } else {
            kt = (kt - a.nf * a.lx + (a.nf + a.lx - 1) / a.lx) * a.lx;
        }
    }
    const int it = kt / a.lx;
    const bool isk = r == 0 && it * a.lx == kt && it < a.nf;
    const int np = (a.nx0 + 1) / 2;
    const double2 *row = a.A + (size_t)kt * np, *neg = a.A + (size_t)(kt ? a.Nt - kt : 0) * np;
    float mx = 0.0f;
    chirp_dft(
        x, a.nx0, r, a.px, a.cx, a.tw, a.mt, a.nx0,
        [&](int i) {
            const long long t = fold ? (long long)i * a.lx : i;
            return t < a.nx0 ? trace_at(row, neg, (int)t) : make_double2(0.0, 0.0);
        },
        [&](int k, double2 v) {
            if (fold) {
                mx = fmaxf(mx, cabs_f(v.x, v.y));
                if (kt < a.nf) a.Z[(size_t)kt * a.nx0 + k] = v;
                return;
            }
            if (kt < a.nf) a.S[(size_t)kt * a.Nx + a.lx * k + r] = v;
            if (isk) a.K[(size_t)it * a.nx0 + k] = v;
        });
    if (!fold) return;
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) atomicMax(a.zmax, __float_as_uint(mx));
}

// Filter of time frequency it: H = S / (Z + max|Z| 1e-5), |H| > lx^2 -> lx, times K; back in x
// (the conjugate of the transform of the conjugate), the first nx traces.
__global__ void __launch_bounds__(512) k_fk_filter(const FkArgs a)
{
    extern __shared__ double2 x[];
    const int it = blockIdx.x;
    const double2 *S = a.S + (size_t)it * a.Nx, *Z = a.Z + (size_t)it * a.nx0, *K = a.K + (size_t)it * a.nx0;
    const double eps = __dmul_rn((double)__uint_as_float(*a.zmax), 0.00001);
    chirp_dft(
        x, a.Nx, 0, a.pX, a.cX, a.tw, a.mt, a.nx,
        [&](int i) {
            const int ib = i % a.nx0;
            const double2 s = S[i], c = K[ib];
            double2 z = Z[ib];
            z.x = __dadd_rn(z.x, eps);
            const double den = __dadd_rn(__dmul_rn(z.x, z.x), __dmul_rn(z.y, z.y));
            double h0 = __ddiv_rn(__dadd_rn(__dmul_rn(s.x, z.x), __dmul_rn(s.y, z.y)), den);
            double h1 = __ddiv_rn(__dsub_rn(__dmul_rn(s.y, z.x), __dmul_rn(s.x, z.y)), den);
            if (cabs_f(h0, h1) > (float)(a.lx * a.lx)) {
                h0 = (double)(float)a.lx;
                h1 = 0.0;
            }
            return conj2(cmul(make_double2(h0, h1), c));
        },
        [&](int k, double2 v) { a.G[(size_t)it * a.nx + k] = conj2(v); });
}

// Back in time for a pair of traces: the first nf frequencies as they are, the rest the conjugate of
// frequency (nt0+1)/2 - (it-nf) (mirror 0, the reference's indexing, zero where that is past
// the last) or nt0 - it (mirror 1); the real part, which is the transform of the spectrum's Hermitian part
// (G(it) + conj G(-it)) / 2.  One trace's is taken back as the real part, the other's as the imaginary one.
__global__ void __launch_bounds__(512) k_fk_back(const FkArgs a)
{
    extern __shared__ double2 x[];
    const int ix = 2 * blockIdx.x;
    const bool two = ix + 1 < a.nx;
    const auto full = [&](int it, int trace) {
        if (it < a.nf) return a.G[(size_t)it * a.nx + trace];
        const int src = a.mirror ? a.nt0 - it : (a.nt0 + 1) / 2 - (it - a.nf);
        return src < a.nf ? conj2(a.G[(size_t)src * a.nx + trace]) : make_double2(0.0, 0.0);
    };
    const auto hermitian = [&](int it, int trace) {
        const double2 u = full(it, trace), w = full(it ? a.nt0 - it : 0, trace);
        return make_double2(0.5 * (u.x + w.x), 0.5 * (u.y - w.y));
    };
    chirp_dft(
        x, a.nt0, 0, a.pt, a.ct, a.tw, a.mt, a.rows,
        [&](int it) {   // (conjugated, as the transform back needs, and so is its result)
            const double2 u = hermitian(it, ix), w = two ? hermitian(it, ix + 1) : make_double2(0.0, 0.0);
            return make_double2(u.x - w.y, -(u.y + w.x));
        },
        [&](int it, double2 v) {
            float *o = a.out + (size_t)it * a.nx + ix;
            o[0] = __double2float_rn(v.x);
            if (two) o[1] = __double2float_rn(-v.y);
        });
}

}  // namespace fk
}  // namespace rtm
