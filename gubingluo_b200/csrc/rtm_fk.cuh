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
// sincospi; the errors stay at the 1e-15 of the double-precision library transforms.
//
// Why not cuFFT here: a gather takes 0.2 ms, creating the four plans it needed 7.3 ms, which
// every stand-alone call and every new session paid (241 traces x 2000 samples, lx = 2: 7.3 ms a
// call -> 2.0 ms, of which 0.3 ms in these kernels; in a session 0.166 -> 0.161 ms a shot of 400
// samples).  What bounds the kernels: shared-memory passes over the
// M points (6 radix-4 stages each way at M = 4096); one block per transform, 1400 transforms.
#pragma once
#include <cuda_runtime.h>

namespace rtm {
namespace fk {

constexpr int kMaxN = 4096;   // longest transform: M = 8192 points, 160 KB of shared memory

__host__ __device__ inline int pow2_for(int n)   // M of a transform of length n
{
    int m = 16;
    while (m < 2 * n - 1) m *= 2;
    return m;
}
// Shared-memory slot of point i: one slot of padding every four, so that the stages of small
// stride are free of bank conflicts.
__device__ __forceinline__ int slot(int i) { return i + (i >> 2); }
inline size_t smem_bytes(int m) { return (size_t)(m + m / 4) * sizeof(double2); }

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

// x (in shared memory, by slot) -> its transform in digit-reversed order; all threads of the
// block, which are synchronised before and after.
__device__ __forceinline__ void fft_fwd(double2 *x, int m, const double2 *__restrict__ tw, int mt)
{
    int n = m;
    for (; n >= 4; n /= 4) {
        const int h = n / 4, ts = mt / n;
        for (int b = threadIdx.x; b < m / 4; b += blockDim.x) {
            const int j = b & (h - 1), i = (b - j) * 4 + j;
            double2 *p0 = &x[slot(i)], *p1 = &x[slot(i + h)], *p2 = &x[slot(i + 2 * h)], *p3 = &x[slot(i + 3 * h)];
            const double2 s02 = cadd(*p0, *p2), d02 = csub(*p0, *p2), s13 = cadd(*p1, *p3), d13 = csub(*p1, *p3);
            const double2 w = tw[j * ts], w2 = cmul(w, w), w3 = cmul(w2, w);
            *p0 = cadd(s02, s13);
            *p1 = cmul(make_double2(d02.x + d13.y, d02.y - d13.x), w);   // d02 - i d13
            *p2 = cmul(csub(s02, s13), w2);
            *p3 = cmul(make_double2(d02.x - d13.y, d02.y + d13.x), w3);  // d02 + i d13
        }
        __syncthreads();
    }
    if (n == 2) {
        for (int b = threadIdx.x; b < m / 2; b += blockDim.x) {
            double2 *p0 = &x[slot(2 * b)], *p1 = &x[slot(2 * b + 1)];
            const double2 s = cadd(*p0, *p1), d = csub(*p0, *p1);
            *p0 = s;
            *p1 = d;
        }
        __syncthreads();
    }
}
// The way back (times m).
__device__ __forceinline__ void fft_inv(double2 *x, int m, const double2 *__restrict__ tw, int mt)
{
    int n = 4;
    if (__popc(m - 1) & 1) {   // odd power of two: a radix-2 stage first
        for (int b = threadIdx.x; b < m / 2; b += blockDim.x) {
            double2 *p0 = &x[slot(2 * b)], *p1 = &x[slot(2 * b + 1)];
            const double2 s = cadd(*p0, *p1), d = csub(*p0, *p1);
            *p0 = s;
            *p1 = d;
        }
        __syncthreads();
        n = 8;
    }
    for (; n <= m; n *= 4) {
        const int h = n / 4, ts = mt / n;
        for (int b = threadIdx.x; b < m / 4; b += blockDim.x) {
            const int j = b & (h - 1), i = (b - j) * 4 + j;
            double2 *p0 = &x[slot(i)], *p1 = &x[slot(i + h)], *p2 = &x[slot(i + 2 * h)], *p3 = &x[slot(i + 3 * h)];
            const double2 w = conj2(tw[j * ts]), w2 = cmul(w, w), w3 = cmul(w2, w);
            const double2 b0 = *p0, b1 = cmul(*p1, w), b2 = cmul(*p2, w2), b3 = cmul(*p3, w3);
            const double2 s02 = cadd(b0, b2), d02 = csub(b0, b2), s13 = cadd(b1, b3), d13 = csub(b1, b3);
            *p0 = cadd(s02, s13);
            *p1 = make_double2(d02.x - d13.y, d02.y + d13.x);   // d02 + i d13
            *p2 = csub(s02, s13);
            *p3 = make_double2(d02.x + d13.y, d02.y - d13.x);
        }
        __syncthreads();
    }
}

// Spectra of the chirps exp(+i pi n^2 / N), |n| < N, wrapped to M points, over M: block b for
// length len[b], into out[b].
struct ChirpArgs {
    int len[3];
    double2 *out[3];
};
__global__ void k_chirps(ChirpArgs a, const double2 *tw, int mt)
{
    extern __shared__ double2 x[];
    const int n = a.len[blockIdx.x], m = pow2_for(n);
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
        const int d = i < n ? i : m - i < n ? m - i : -1;
        x[slot(i)] = d < 0 ? make_double2(0.0, 0.0) : conj2(unit((long long)d * d, n));
    }
    __syncthreads();
    fft_fwd(x, m, tw, mt);
    const double f = 1.0 / m;
    for (int i = threadIdx.x; i < m; i += blockDim.x) a.out[blockIdx.x][i] = make_double2(x[slot(i)].x * f, x[slot(i)].y * f);
}

// The block's transform of length n of in(i), i < n: out(k, X[k]) for k < kmax.  X[k] is frequency
// k + r / lx of the samples (r = 0: the plain transform).
template <typename In, typename Out>
__device__ __forceinline__ void chirp_dft(double2 *x, int n, int r, int lx, const double2 *__restrict__ chirp,
                                          const double2 *__restrict__ tw, int mt, int kmax, In in, Out out)
{
    const int m = pow2_for(n);
    for (int i = threadIdx.x; i < m; i += blockDim.x)
        x[slot(i)] = i < n ? cmul(in(i), unit(((long long)lx * i + 2 * r) * i, (long long)lx * n)) : make_double2(0.0, 0.0);
    __syncthreads();
    fft_fwd(x, m, tw, mt);
    for (int i = threadIdx.x; i < m; i += blockDim.x) x[slot(i)] = cmul(x[slot(i)], chirp[i]);
    __syncthreads();
    fft_inv(x, m, tw, mt);
    for (int k = threadIdx.x; k < kmax; k += blockDim.x) out(k, cmul(x[slot(k)], unit((long long)k * k, n)));
    __syncthreads();
}

struct FkArgs {
    const float *in;              // [nt0][nx0]
    int nx0, nt0, nx, lx, Nx, Nt, nf, nh;   // nh = Nt / 2 + 1 time frequencies of the padded gather
    int rows, mirror;             // rows written of the result
    double2 *A;                   // [nh][nx0]: time spectra of the traces
    double2 *K, *S, *Z;           // [nf][nx0], [nf][Nx], [nf][nx0]
    double2 *G;                   // [nf][nx]: filtered, back in x
    unsigned *zmax;
    const double2 *ct, *cx, *cX;  // chirp spectra of lengths nt0, nx0, Nx
    const double2 *tw;
    int mt;
    float *out;                   // [rows][nx]
};

// Time transforms: block (ix, r), frequencies lx q + r of the padded length up to its Nyquist row.
__global__ void k_fk_time(const FkArgs a)
{
    extern __shared__ double2 x[];
    const int ix = blockIdx.x, r = blockIdx.y;
    chirp_dft(
        x, a.nt0, r, a.lx, a.ct, a.tw, a.mt, (a.nh - r + a.lx - 1) / a.lx,
        [&](int i) { return make_double2((double)a.in[(size_t)i * a.nx0 + ix], 0.0); },
        [&](int q, double2 v) { a.A[(size_t)(a.lx * q + r) * a.nx0 + ix] = v; });
}

// |z| as the reference's fftw_fabs: sqrtf of the float-rounded double re^2 + im^2.
__device__ __forceinline__ float cabs_f(double re, double im)
{
    return sqrtf(__double2float_rn(__dadd_rn(__dmul_rn(re, re), __dmul_rn(im, im))));
}

// Space transforms of time frequency kt: S (all lx parts) and the fold Z below nf, K at every
// lx-th frequency, and max |Z| over all of them (non-negative floats order like their bits).
__global__ void k_fk_space(const FkArgs a)
{
    extern __shared__ double2 x[];
    const int kt = blockIdx.x;
    const double2 *row = a.A + (size_t)kt * a.nx0;
    float mx = 0.0f;
    chirp_dft(
        x, a.nx0, 0, 1, a.cx, a.tw, a.mt, a.nx0,
        [&](int i) { return (long long)i * a.lx < a.nx0 ? row[i * a.lx] : make_double2(0.0, 0.0); },
        [&](int k, double2 v) {
            mx = fmaxf(mx, cabs_f(v.x, v.y));
            if (kt < a.nf) a.Z[(size_t)kt * a.nx0 + k] = v;
        });
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) atomicMax(a.zmax, __float_as_uint(mx));
    const int it = kt / a.lx;
    const bool isk = it * a.lx == kt && it < a.nf;
    for (int r = 0; r < a.lx; r++) {
        if (kt >= a.nf && !(r == 0 && isk)) break;
        chirp_dft(
            x, a.nx0, r, a.lx, a.cx, a.tw, a.mt, a.nx0, [&](int i) { return row[i]; },
            [&](int k, double2 v) {
                if (kt < a.nf) a.S[(size_t)kt * a.Nx + a.lx * k + r] = v;
                if (r == 0 && isk) a.K[(size_t)it * a.nx0 + k] = v;
            });
    }
}

// Filter of time frequency it: H = S / (Z + max|Z| 1e-5), |H| > lx^2 -> lx, times K; back in x
// (the conjugate of the transform of the conjugate), the first nx traces.
__global__ void k_fk_filter(const FkArgs a)
{
    extern __shared__ double2 x[];
    const int it = blockIdx.x;
    const double2 *S = a.S + (size_t)it * a.Nx, *Z = a.Z + (size_t)it * a.nx0, *K = a.K + (size_t)it * a.nx0;
    const double eps = __dmul_rn((double)__uint_as_float(*a.zmax), 0.00001);
    chirp_dft(
        x, a.Nx, 0, 1, a.cX, a.tw, a.mt, a.nx,
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

// Back in time for trace ix: the first nf frequencies as they are, the rest the conjugate of
// frequency (nt0+1)/2 - (it-nf) (mirror 0, the reference's indexing, zero where that is past
// the last) or nt0 - it (mirror 1); the real part.
__global__ void k_fk_back(const FkArgs a)
{
    extern __shared__ double2 x[];
    const int ix = blockIdx.x;
    chirp_dft(
        x, a.nt0, 0, 1, a.ct, a.tw, a.mt, a.rows,
        [&](int it) {   // (conjugated, as the transform back needs)
            if (it < a.nf) return conj2(a.G[(size_t)it * a.nx + ix]);
            const int src = a.mirror ? a.nt0 - it : (a.nt0 + 1) / 2 - (it - a.nf);
            return src < a.nf ? a.G[(size_t)src * a.nx + ix] : make_double2(0.0, 0.0);
        },
        [&](int it, double2 v) { a.out[(size_t)it * a.nx + ix] = __double2float_rn(v.x); });
}

}  // namespace fk
}  // namespace rtm
