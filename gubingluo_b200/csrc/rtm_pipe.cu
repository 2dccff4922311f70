// rtm_pipe.cu — the time-step kernels in their pipelined form (sm_100a): persistent blocks, a
// producer warp that keeps two tiles in flight, consumer warps with four columns by U rows per
// thread.
//
// A launch covers a list of tiles (128 columns by BZ rows).  Each resident block takes the
// tile of its index and then tiles from a device counter.  Its producer warp fills the block's stages
// ahead of the consumers: the halo boxes and the per-cell operands (1/rho, vx, vz or kappa, p)
// by the tensor memory accelerator, a copy of the shot's descriptor, and an L2 prefetch of the
// operands that only some tiles need (split PML fields, imaging accumulators).  A full and an
// empty mbarrier per stage connect the two sides, so consumer warps never wait for each other.
//
//   * A thread owns columns x0+4g .. x0+4g+3 and U adjacent rows.  The x-derivatives of four
//     columns read seven 16-byte words of the staged row; the z-derivatives of 4 x U cells walk
//     outwards from the centre rows, one new row above and below per tap, so U+19 16-byte loads
//     serve them all with 2U rows live.
//   * Tap sums, damping and updates run in packed fp32 pairs (two columns per instruction, each
//     lane rounded as the scalar operation), in the order i = 1 .. 10 of every other form: the
//     results are the same bits.
//   * The host marks in each tile what its cells need (TileRef.interior): interior tiles take
//     the update alone; the others test only for what they hold, update whole 16-byte words and
//     select per column; the strips of the source pass are saved by the tiles that hold their
//     cells, so a source-pass step is two launches.
//   * One launch may carry tiles of two kinds (a pressure kind and a velocity kind) that do
//     not depend on each other, so a backward step is two launches: {reconstruction pressure,
//     receiver velocity} and {receiver pressure with imaging, next step's reconstruction
//     velocity}.
//   * Launches use programmatic dependent launch: a kernel's blocks are set up while the kernel
//     before it drains, and wait for its completion before they read any field; the first tile's
//     copies of what no kernel of the pass writes (1/rho or kappa, damping factors) start before
//     that wait.
//
// What bounds it: 64 shots of 1801x451, us a launch at 1965 MHz (one tile per block before; each field
// read and written once at 6.46 TB/s): receiver velocity 192 (248; 191), forward velocity with its strips
// 210 (251 + 28; 193), receiver pressure and imaging 317 (347; 302): the memory's rate at that clock.
// Forward pressure 252 (281; 187): latency of shared-memory reads and instructions.  Reconstruction 171
// and 140 (191, 176; 144, 120): the tiles with strips.  A long run is power-capped to 1690-1890 MHz, and
// there the first three read 0.88-0.94 of the memory's rate and gain 10% from 16% more clock: the SMs'
// side (shared-memory reads and their latency) bounds them as much as the memory.  One shot of 401x201: 4.6 us a launch (7 launches of 7 us a
// step before, 4 now): one tile's chain of copy, sums and stores.
//
// Reference kernels these replace: see rtm_stencil.cu.
#include <atomic>
#include <type_traits>

#include "rtm_launch.h"
#include "rtm_vec.cuh"

#ifndef RTM_PIPE_BZ
#error "compiled once per tile height: -DRTM_PIPE_BZ=8, 12, 16, 32, 64"
#endif
#define RTM_MIN2(a, b) ((a) < (b) ? (a) : (b))

namespace {

// ---- packed pairs -----------------------------------------------------------------------
__device__ __forceinline__ float2 lo2(const float4 &v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4 &v) { return make_float2(v.z, v.w); }
__device__ __forceinline__ float2 both(float c) { return make_float2(c, c); }
// a - b as a multiply-add by -1 (an exact product, one rounding).  The assembler contracts a
// packed multiplication into a packed addition or subtraction that follows it, although both
// ask for their own rounding, and takes a multiply-add by +1 for an addition, but not one by
// -1: every sum below is written as the difference of a negated product.
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, both(-1.f), a); }


// Four adjacent columns as two pairs.
struct P4 {
    float2 a, b;
};
__device__ __forceinline__ P4 p4(const float4 &v) { return {lo2(v), hi2(v)}; }
__device__ __forceinline__ float4 q4(const P4 &v) { return make_float4(v.a.x, v.a.y, v.b.x, v.b.y); }
__device__ __forceinline__ P4 mul(const P4 &u, const P4 &v) { return {__fmul2_rn(u.a, v.a), __fmul2_rn(u.b, v.b)}; }
__device__ __forceinline__ P4 mul(const P4 &u, float c) { return {__fmul2_rn(u.a, both(c)), __fmul2_rn(u.b, both(c))}; }
__device__ __forceinline__ P4 sub(const P4 &u, const P4 &v) { return {sub2(u.a, v.a), sub2(u.b, v.b)}; }
// damp() of rtm_stencil_common.cuh on four columns
__device__ __forceinline__ P4 damp(const P4 &f, const P4 &d, const P4 &c1, const P4 &ic2)
{
    return mul(sub(mul(c1, f), d), ic2);
}
// Column j takes a when its bit is set in m, else b.
__device__ __forceinline__ float4 pick(unsigned m, const float4 &a, const float4 &b)
{
    return make_float4(m & 1 ? a.x : b.x, m & 2 ? a.y : b.y, m & 4 ? a.z : b.z, m & 8 ? a.w : b.w);
}
// Bits of the columns x .. x+3 that lie in [lo, hi).
__device__ __forceinline__ unsigned cols_in(int x, int lo, int hi)
{
    unsigned m = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) m |= (unsigned)(x + j >= lo && x + j < hi) << j;
    return m;
}
// A field word that the kernel before this one wrote (never through the read-only path: under
// programmatic dependent launch that kernel may still run when this one starts).
__device__ __forceinline__ float4 ldv4(const float *p)
{
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
    return v;
}

// x-derivative sums of four columns from one staged row (dx4 of rtm_vec.cuh).  Of a tap's two
// operands one pair is always misaligned in the 16-byte words, so the differences are taken as
// single instructions and only the multiply-adds as pairs.
template <int F, int G, typename C>
__device__ __forceinline__ P4 dx_sum(const float *rw, C coef)
{
    float a[28];
#pragma unroll
    for (int q = 0; q < 7; q++) {
        const float4 v = lds4(rw + 4 * q);
        a[4 * q] = v.x; a[4 * q + 1] = v.y; a[4 * q + 2] = v.z; a[4 * q + 3] = v.w;
    }
    float2 s[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
    for (int i = 1; i <= R; i++)
#pragma unroll
        for (int h = 0; h < 2; h++)
            s[h] = __ffma2_rn(coef(h, i - 1),
                              make_float2(__fsub_rn(a[F + 2 * h + i], a[G + 2 * h - i]),
                                          __fsub_rn(a[F + 2 * h + 1 + i], a[G + 2 * h + 1 - i])),
                              s[h]);
    return {s[0], s[1]};
}
// z-derivative sums of 4 columns x U rows; `col`: the columns' word in the group's first staged
// row.  Output row u takes rows u+9+i and u+10-i.
template <int U, int STRIDE, typename C>
__device__ __forceinline__ void dz_sum(const float *col, P4 (&s)[U], C coef)
{
    float4 up[U], dn[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
        s[u] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        up[u] = lds4(col + (u + 10) * STRIDE);
    }
#pragma unroll
    for (int u = 0; u < U; u++) dn[u] = u ? up[u - 1] : lds4(col + 9 * STRIDE);
#pragma unroll
    for (int i = 1; i <= R; i++) {
#pragma unroll
        for (int u = 0; u < U; u++) {
            s[u].a = __ffma2_rn(coef(u, 0, i - 1), sub2(lo2(up[u]), lo2(dn[u])), s[u].a);
            s[u].b = __ffma2_rn(coef(u, 1, i - 1), sub2(hi2(up[u]), hi2(dn[u])), s[u].b);
        }
        if (i == R) break;
#pragma unroll
        for (int u = 0; u + 1 < U; u++) up[u] = up[u + 1];
        up[U - 1] = lds4(col + (U - 1 + 10 + i) * STRIDE);
#pragma unroll
        for (int u = U - 1; u > 0; u--) dn[u] = dn[u - 1];
        dn[0] = lds4(col + (9 - i) * STRIDE);
    }
}

// ---- stages -----------------------------------------------------------------------------
__host__ __device__ constexpr int pad128(int bytes) { return (bytes + 127) / 128 * 128; }
// Stage of a velocity tile: p rows z0-9 .. z0+BZ+9 (columns x0-12 .. x0+139), then 1/rho, vx and
// vz of the tile.  Stage of a pressure tile: vx rows of the tile (columns x0-12 ..), vz rows
// z0-10 .. z0+BZ+8, then kappa and p of the tile.  Offsets in floats.
template <int BZ>
struct Stage {
    static constexpr int v_op = pad128((BZ + 19) * WW * 4) / 4, v_bytes = v_op * 4 + 3 * BZ * BX * 4;
    static constexpr int p_vz = BZ * WW, p_op = p_vz + (BZ + 19) * BX, p_bytes = (p_op + 2 * BZ * BX) * 4;
    static_assert(BZ * WW * 4 % 128 == 0, "every box starts on 128 bytes");
};
// A launch's shape.  PM, VM: pressure and velocity mode of its tiles (-1: none of that kind).
// Tiles of up to 16 rows stage what only some pressure tiles need as well: the split PML fields
// of band tiles; ps, g1 and illum of the receiver pass's tiles with interior cells (which then
// load their split fields, if any, directly, one row ahead).  Taller tiles have no room for it.
template <int BZ, int PM, int VM, typename ACC, bool THIN = false>
struct Pipe {
    static constexpr bool staged = BZ <= 16;
    static constexpr int row = BZ * BX * 4;   // bytes of one operand of a tile
    static constexpr int extra = !staged ? 0 : PM == 0 ? 2 * row : PM == 2 ? (1 + 2 * (int)sizeof(ACC) / 4) * row : 0;
    static constexpr int bytes = RTM_MAX2(PM >= 0 ? Stage<BZ>::p_bytes + extra : 0, VM >= 0 ? Stage<BZ>::v_bytes : 0);
    // blocks of n stages that fit an SM's shared memory (a block's own part: descriptors, barriers,
    // coefficients and the system's 1 KB)
    static constexpr int fit(int n) { return 228 * 1024 / (n * bytes + n * (1600 + 8 * BZ) + (PM == 3 && VM < 0 ? 1200 : 3700)); }
    // 8-row tiles: up to three blocks of four warps, or the thin shape (kThinTiles).  12- and 16-row
    // tiles: two blocks where two stages each fit, else one.  The rows a thread takes: fewer rows mean
    // more shared-memory reads per cell but twice the warps, and with eight consumer warps on an SM
    // the pressure kernels wait on instruction and read latency (issue slots 34% used, DRAM 46%):
    // 64 shots of 1801x451 (us, 12 rows with U = 3 / 2) forward pressure 306 / 276, receiver pressure
    // 320 / 328; a step of 16 shots 389 / 370.  Velocity at 16 rows reads the least per cell and is
    // at the memory's rate with U = 4: 203 / 221 (U = 4 / 2).
    static constexpr bool two = (BZ == 12 || BZ == 16) && fit(2) >= 2;
    static constexpr int U = THIN ? 1 : BZ == 16 ? (PM < 0 ? 4 : 2) : BZ <= 12 ? 2 : BZ == 64 ? 8 : 4;
    static constexpr int warps = BZ / U, threads = 32 * (warps + 1);   // consumers; and the producer warp
    static constexpr int blocks = THIN ? 2 : BZ == 8 ? (PM == 3 && VM < 0 ? fit(2) : RTM_MIN2(fit(2), 3)) : two ? 2 : 1;
    static constexpr int stages = BZ <= 16 && blocks > 1 ? 2 : fit(3) ? 3 : fit(2) ? 2 : 1;
};

// What the consumers of a stage read besides its boxes: the tile, its shot's descriptor and, for
// tiles that are not interior, the damping factors of the tile's columns and rows (c1 and 1/c2 of
// the tile's field kind; 1 outside the bands and where the field has no cell).
template <int BZ>
struct alignas(16) StageMeta {   // (every stage's factors are read as 16-byte words)
    float c1x[BX], ic2x[BX], c1z[BZ], ic2z[BZ];
    TileRef t;
    ShotDev S;
};

// Bytes that the barrier's phase waits for besides the producer's arrival.
__device__ __forceinline__ void mbar_expect_tx(unsigned long long *bar, unsigned bytes)
{
    asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// n floats of a 16-byte aligned block (n a multiple of 4).
__device__ __forceinline__ void bulk_copy(float *dst, const float *src, int n, unsigned long long *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(smem_u32(dst)),
                 "l"(src), "r"(n * 4), "r"(smem_u32(bar))
                 : "memory");
}
// One thread: the damping factors of a tile's columns and rows into the stage's descriptor (tiles of
// the full grid start at multiples of 128 columns and BZ rows, so every block is aligned and
// inside the padded arrays).
template <int BZ>
__device__ __forceinline__ void fill_damping(StageMeta<BZ> &m, int c1x, int ic2x, int c1z, int ic2z, unsigned long long *bar)
{
    const float *pml = m.S.pml;
    mbar_expect_tx(bar, 2 * (BX + BZ) * 4);
    bulk_copy(m.c1x, pml + c1x + m.t.x0, BX, bar);
    bulk_copy(m.ic2x, pml + ic2x + m.t.x0, BX, bar);
    bulk_copy(m.c1z, pml + c1z + m.t.z0, BZ, bar);
    bulk_copy(m.ic2z, pml + ic2z + m.t.z0, BZ, bar);
}
__device__ __forceinline__ const void *tmap(const char *maps, int which) { return maps + which * RTM_TMAP_BYTES; }
// One thread: the copies of a tile into a stage, in two parts: what no kernel of the pass writes (the
// bytes expected in all, 1/rho or kappa, damping factors), which the first tile's copies start with
// before the kernel in front has finished, and the fields, which come first in every later tile:
// a stage is idle until its largest boxes are on their way (64 shots of 1801x451: 1369 us a step
// with the constant part first, 1324 with the fields first, 1300 with the descriptor's words
// stored after the fields' copies too).
template <int BZ, int MODE>
__device__ __forceinline__ void fill_vel_const(StageMeta<BZ> &m, float *st, unsigned long long *bar)
{
    mbar_expect_tx(bar, ((BZ + 19) * WW + 3 * BZ * BX) * 4);
    tma_box(st + Stage<BZ>::v_op, tmap_of(m.S, MODE == 0 ? RTM_TMAP_IRF : MODE == 2 ? RTM_TMAP_IRB : RTM_TMAP_IRB_RECON),
            m.t.x0, m.t.z0, bar);
    if (MODE != 3 && !(m.t.interior & 1)) {
        const PmlOffsets o = pml_offsets(m.S.X, m.S.Z);
        fill_damping<BZ>(m, o.c1vx, o.ic2vx, o.c1vz, o.ic2vz, bar);
    }
}
template <int BZ, int MODE>
__device__ __forceinline__ void fill_vel(const char *maps, const TileRef &t, float *st, unsigned long long *bar)
{
    float *op = st + Stage<BZ>::v_op;
    tma_box(st, tmap(maps, MODE == 2 ? RTM_TMAP_B_P : MODE == 3 ? RTM_TMAP_A_P_RECON : RTM_TMAP_A_P), t.x0 - 12,
            t.z0 - 9, bar);
    tma_box(op + BZ * BX, tmap(maps, MODE == 0 ? RTM_TMAP_A_VX_OWN : MODE == 2 ? RTM_TMAP_B_VX_OWN : RTM_TMAP_A_VX_OWN_RECON),
            t.x0, t.z0, bar);
    tma_box(op + 2 * BZ * BX,
            tmap(maps, MODE == 0 ? RTM_TMAP_A_VZ_OWN : MODE == 2 ? RTM_TMAP_B_VZ_OWN : RTM_TMAP_A_VZ_OWN_RECON), t.x0, t.z0,
            bar);
}
// What a pressure tile stages besides its boxes: imaging operands, or split fields.
template <int BZ, int MODE>
__device__ __forceinline__ bool stages_img(const TileRef &t)
{
    return BZ <= 16 && MODE == 2 && (t.interior & (1 | RTM_TILE_IMG));
}
template <int BZ, int MODE>
__device__ __forceinline__ bool stages_band(const TileRef &t)
{
    return BZ <= 16 && MODE != 3 && (t.interior & RTM_TILE_BAND) && !stages_img<BZ, MODE>(t);
}
template <int BZ, int MODE, typename ACC>
__device__ __forceinline__ void fill_pres_const(StageMeta<BZ> &m, float *st, unsigned long long *bar)
{
    constexpr int row = BZ * BX * 4;
    mbar_expect_tx(bar, (BZ * WW + (BZ + 19) * BX) * 4 + 2 * row +
                            (stages_img<BZ, MODE>(m.t) ? (1 + 2 * (int)sizeof(ACC) / 4) * row
                             : stages_band<BZ, MODE>(m.t) ? 2 * row : 0));
    tma_box(st + Stage<BZ>::p_op, tmap_of(m.S, MODE == 0 ? RTM_TMAP_KF : MODE == 2 ? RTM_TMAP_KB : RTM_TMAP_KB_RECON),
            m.t.x0, m.t.z0, bar);
    if (MODE != 3 && !(m.t.interior & 1)) {
        const PmlOffsets o = pml_offsets(m.S.X, m.S.Z);
        fill_damping<BZ>(m, o.c1x, o.ic2x, o.c1z, o.ic2z, bar);
    }
}
template <int BZ, int MODE, typename ACC>
__device__ __forceinline__ void fill_pres(const char *maps, const TileRef &t, float *st, unsigned long long *bar)
{
    tma_box(st, tmap(maps, MODE == 2 ? RTM_TMAP_B_VX : MODE == 3 ? RTM_TMAP_A_VX_RECON : RTM_TMAP_A_VX), t.x0 - 12, t.z0,
            bar);
    tma_box(st + Stage<BZ>::p_vz, tmap(maps, MODE == 2 ? RTM_TMAP_B_VZ : MODE == 3 ? RTM_TMAP_A_VZ_RECON : RTM_TMAP_A_VZ),
            t.x0, t.z0 - 10, bar);
    float *op = st + Stage<BZ>::p_op;
    tma_box(op + BZ * BX, tmap(maps, MODE == 0 ? RTM_TMAP_A_P_OWN : MODE == 2 ? RTM_TMAP_B_P_OWN : RTM_TMAP_A_P_OWN_RECON),
            t.x0, t.z0, bar);
    float *ex = op + 2 * BZ * BX;
    if (stages_img<BZ, MODE>(t)) {   // ps, g1, illum (8-byte accumulators: two words per column)
        constexpr int w = (int)sizeof(ACC) / 4;
        tma_box(ex, tmap(maps, RTM_TMAP_A_P_OWN), t.x0, t.z0, bar);
        tma_box(ex + BZ * BX, tmap(maps, RTM_TMAP_G1), w * t.x0, t.z0, bar);
        tma_box(ex + (1 + w) * BZ * BX, tmap(maps, RTM_TMAP_ILLUM), w * t.x0, t.z0, bar);
    }
    if (stages_band<BZ, MODE>(t)) {
        tma_box(ex, tmap(maps, MODE == 0 ? RTM_TMAP_A_SX : RTM_TMAP_B_SX), t.x0, t.z0, bar);
        tma_box(ex + BZ * BX, tmap(maps, MODE == 0 ? RTM_TMAP_A_SZ : RTM_TMAP_B_SZ), t.x0, t.z0, bar);
    }
}

// The producer warp's L2 prefetch of rows [z0, z1) of a tile's columns of one field.
__device__ __forceinline__ void prefetch_tile(const void *field, int es, int z0, int z1, int x0, int pitch)
{
    const unsigned bytes = (unsigned)(min(RTM_BX, pitch - x0) * es);
    for (int z = z0 + (int)(threadIdx.x & 31); z < z1; z += 32)
        prefetch_l2((const char *)field + ((size_t)z * pitch + x0) * es, bytes);
}

// Coefficients of reduced orders, for two adjacent columns at a time: row (k, r) of the table in
// shared memory holds the ten taps of the pair of half-orders (r, r) for k = 0, (r, r+1) for
// k = 1 and (r, r-1) for k = 2, r = 1 .. 10 (adjacent columns differ by at most one).  Orders
// below 1 (the grid's edge, which the update leaves alone, and the row padding) read as 1.
constexpr int kPairs = 30 * R;
__device__ __forceinline__ const float2 *pair_row(const float2 *tab, int r0, int r1)
{
    r0 = max(r0, 1);
    r1 = max(r1, 1);
    return tab + ((r1 > r0 ? R : r1 < r0 ? 2 * R : 0) + r0 - 1) * R;
}
__device__ __forceinline__ float2 pair_entry(const float *coef, int i)
{
    const int k = i / (R * R), r = i / R % R, tap = i % R, r1 = min(max(k == 1 ? r + 1 : k == 2 ? r - 1 : r, 0), R - 1);
    return make_float2(coef[r * R + tap], coef[r1 * R + tap]);
}

// Destination of strip cell idx of the step being saved (fp32 strips, or the staging ring of
// the packed forms).
__device__ __forceinline__ float *strip_dst(const StepArgs &a, const ShotDev &S)
{
    return a.strip_prec == RTM_FP32 ? (float *)S.strips + (size_t)a.it * S.strip_len
                                    : S.strip_stage + (size_t)a.ring * S.strip_len;
}

// The columns of a word that lie in a strip (mask m): saved to d[0 .. 3], restored from i0 .. i0+3.
__device__ __forceinline__ void strip_put(float *d, unsigned m, const float (&v)[4])
{
#pragma unroll
    for (int j = 0; j < 4; j++)
        if (m >> j & 1) d[j] = v[j];
}
__device__ __forceinline__ void strip_get(float (&v)[4], const void *strips, size_t i0, unsigned m, int prec, float scale)
{
    if (prec == RTM_FP32) {
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (m >> j & 1) v[j] = ((const float *)strips + i0)[j];
        return;
    }
    const unsigned short *p = (const unsigned short *)strips + i0;
    unsigned short h[4] = {0, 0, 0, 0};
#pragma unroll
    for (int j = 0; j < 4; j++)
        if (m >> j & 1) h[j] = p[j];
#pragma unroll
    for (int j = 0; j < 4; j++)
        v[j] = (prec == RTM_FP16 ? __half2float(__ushort_as_half(h[j])) : __bfloat162float(__ushort_as_bfloat16(h[j]))) * scale;
}

// ---- velocity (later: the step whose saved strips the reconstruction restores) -----------
template <int BZ, int U, int MODE>
__device__ __forceinline__ void vel_compute(const StepArgs &a, const StageMeta<BZ> &m, const TileRef &t, const float *st,
                                            const float2 *s_tab, int later)
{
    const ShotDev &S = m.S;
    const int g = threadIdx.x & 31, r = threadIdx.x >> 5;
    const int x = t.x0 + 4 * g, zr = t.z0 + U * r;
    const int pitch = S.pitch;
    const WaveDev &W = MODE == 2 ? S.b : S.a;
    float *vxp = W.vx, *vzp = W.vz;
    const float *rowbase = st + (U * r + 9) * WW + 4 * g;    // staged p row of grid row zr, word of column x-12
    const float *colbase = st + (U * r) * WW + 4 * g + 12;   // the group's first staged row, word of column x
    const float *op = st + Stage<BZ>::v_op + (U * r) * BX + 4 * g;
    // (the reconstruction adds its increments: it subtracts their negatives)
    const float dtx = MODE == 3 ? -a.dtx : a.dtx, dtz = MODE == 3 ? -a.dtz : a.dtz;
    const auto cx = [&](int, int i) { return a.c2[i]; };
    const auto cz = [&](int, int, int i) { return a.c2[i]; };

    if (t.interior & 1) {   // every cell interior, full orders, no strip: the update alone
        P4 dz[U];
        dz_sum<U, WW>(colbase, dz, cz);
        unsigned id = (unsigned)zr * pitch + x;
#pragma unroll
        for (int u = 0; u < U; u++, id += pitch) {
            const P4 dx = dx_sum<12, 13>(rowbase + u * WW, cx);
            const P4 ir = p4(lds4(op + u * BX));
            const P4 ix = mul(mul(dx, dtx), ir), iz = mul(mul(dz[u], dtz), ir);
            const P4 ov = p4(lds4(op + (BZ + u) * BX)), ow = p4(lds4(op + (2 * BZ + u) * BX));
            st4(&vxp[id], q4(sub(ov, ix)));
            st4(&vzp[id], q4(sub(ow, iz)));
        }
        return;
    }

    const int X = S.X, Z = S.Z, npml = S.npml, F = t.interior;
    // (the reconstruction leaves every column outside [npml-R, X-npml+R) alone)
    if (x >= X || zr >= Z || (MODE == 3 && (x + 4 <= npml - R || x >= X - npml + R))) return;
    // columns whose vx, vz the update writes, and the strip columns of vx (the ten to the left of
    // the interior and the ten from X-npml-1 on)
    unsigned mvx = 15u, mvz = 15u, msl = 0u, msr = 0u;
    if (F & RTM_TILE_XBAND) {
        mvx = MODE == 3 ? cols_in(x, npml, X - npml - 1) : cols_in(x, 0, X - 1);
        mvz = MODE == 3 ? cols_in(x, npml, X - npml) : cols_in(x, 0, X);
        if (MODE == 3 || MODE == 0) {
            msl = cols_in(x, npml - R, npml);
            msr = cols_in(x, X - npml - 1, min(X - npml - 1 + R, X - 1));
        }
    }
    // groups of rows or tiles of columns that reach the outer ten cells take table coefficients:
    // vx order per column (cuda_norderx), vz order per row (cuda_norderz); the reconstruction
    // writes only cells at least npml >= R from the edge, where every order is full
    const auto order = [&](int i, int n) { return min(min(i + 1, n - 1 - i), R); };
    const bool edge_x = MODE != 3 && (U == 1 || (F & RTM_TILE_XEDGE));
    const bool edge_z = MODE != 3 && (U == 1 || (zr < R || zr + U > Z - R));
    const float2 *ex[2] = {s_tab, s_tab};
    if (edge_x) {
        ex[0] = pair_row(s_tab, order(x, X), order(x + 1, X));
        ex[1] = pair_row(s_tab, order(x + 2, X), order(x + 3, X));
    }
    P4 dz[U];
    if (!edge_z) dz_sum<U, WW>(colbase, dz, cz);
    else dz_sum<U, WW>(colbase, dz, [&](int u, int, int i) { return s_tab[(max(order(zr + u, Z), 1) - 1) * R + i]; });
    const int nxi = S.nxi, nzi = S.nzi;
    const bool save = MODE == 0 && a.save;
    // strip cells of column x in row zr: vx left and right of the interior (R apart per row), and vz
    // in row 0 of its strips
    const int sl = (zr - npml) * R + x - (npml - R), sr = (nzi + zr - npml) * R + x - (X - npml - 1);
    const int stb = 2 * R * nzi + x - npml;
    const unsigned mtb = MODE == 3 ? mvz : cols_in(x, npml, X - npml);
    float *strips = save ? strip_dst(a, S) : nullptr;
    const size_t s0 = (size_t)later * S.strip_len;
    float scx = 1.0f, scz = 1.0f;
    if (MODE == 3 && a.strip_prec) {
        scx = S.strip_scale[(size_t)later * 4 + 0];
        scz = S.strip_scale[(size_t)later * 4 + 1];
    }
    unsigned id = (unsigned)zr * pitch + x;
#pragma unroll
    for (int u = 0; u < U; u++, id += pitch) {
        const int z = zr + u;
        if (z >= Z) break;
        const bool zin = z >= npml && z < Z - npml;
        const int srow = MODE == 3 || save ? strip_row_tb(z, npml, Z - npml - 1, nxi) : -1;
        float rx[4], rz[4];   // restored: vx of a row of the interior, vz of a strip row
        if (MODE == 3 && zin) {   // read_d_vxpml, kernel.cu:1294-1320
            if (msl) strip_get(rx, S.strips, s0 + sl + u * R, msl, a.strip_prec, scx);
            if (msr) {
                float q[4];
                strip_get(q, S.strips, s0 + sr + u * R, msr, a.strip_prec, scx);
#pragma unroll
                for (int j = 0; j < 4; j++)
                    if (msr >> j & 1) rx[j] = q[j];
            }
        }
        if (MODE == 3 && srow >= 0 && mvz)   // read_d_vzpml, kernel.cu:1321-1347
            strip_get(rz, S.strips, s0 + stb + srow, mvz, a.strip_prec, scz);
        P4 dx;
        if (!edge_x) dx = dx_sum<12, 13>(rowbase + u * WW, cx);
        else dx = dx_sum<12, 13>(rowbase + u * WW, [&](int h, int i) { return ex[h][i]; });
        const P4 ir = p4(lds4(op + u * BX));
        const P4 ix = mul(mul(dx, dtx), ir), iz = mul(mul(dz[u], dtz), ir);
        const float4 ov = lds4(op + (BZ + u) * BX), ow = lds4(op + (2 * BZ + u) * BX);
        if (MODE == 3) {
            // kernel.cu:318-388 (+=) on the interior; strips of the step after elsewhere
            if (zin && (mvx | msl | msr)) {
                float4 n = pick(mvx, q4(sub(p4(ov), ix)), ov);
                if (msl | msr) n = pick(msl | msr, f4(rx), n);
                st4(&vxp[id], n);
            }
            if (z >= npml && z <= Z - npml - 2) {
                if (mvz) st4(&vzp[id], pick(mvz, q4(sub(p4(ow), iz)), ow));
            } else if (mvz && srow >= 0) {
                st4(&vzp[id], pick(mvz, f4(rz), ow));
            }
            continue;
        }
        // kernel.cu:430-500 (interior) and :542-713 (PML; with factors of 1 the damped update
        // rounds as the plain one)
        float4 nx;
        if (F & RTM_TILE_XBAND) nx = pick(mvx, q4(damp(p4(ov), ix, p4(lds4(&m.c1x[4 * g])), p4(lds4(&m.ic2x[4 * g])))), ov);
        else nx = q4(sub(p4(ov), ix));
        st4(&vxp[id], nx);
        if (z >= Z - 1) continue;
        float4 nz;
        if (z >= npml && z < Z - npml - 1) nz = q4(sub(p4(ow), iz));
        else {
            const float2 c1 = both(m.c1z[U * r + u]), ic2 = both(m.ic2z[U * r + u]);
            nz = q4(damp(p4(ow), iz, {c1, c1}, {ic2, ic2}));
        }
        if (F & RTM_TILE_XBAND) nz = pick(mvz, nz, ow);
        st4(&vzp[id], nz);
        if (save) {   // save_d_vxpml, save_d_vzpml (kernel.cu:1186-1240)
            const float vx[4] = {nx.x, nx.y, nx.z, nx.w}, vz[4] = {nz.x, nz.y, nz.z, nz.w};
            if (zin && msl) strip_put(strips + sl + u * R, msl, vx);
            if (zin && msr) strip_put(strips + sr + u * R, msr, vx);
            if (srow >= 0) strip_put(strips + stb + srow, mtb, vz);
        }
    }
}

// ---- pressure ---------------------------------------------------------------------------
template <int BZ, int U, int MODE, typename ACC>
__device__ __forceinline__ void pres_compute(const StepArgs &a, const StageMeta<BZ> &m, const TileRef &t, const float *st,
                                             const float2 *s_tab, int record)
{
    const ShotDev &S = m.S;
    const int g = threadIdx.x & 31, r = threadIdx.x >> 5;
    const int x = t.x0 + 4 * g, zr = t.z0 + U * r;
    const int pitch = S.pitch;
    const WaveDev &W = MODE == 2 ? S.b : S.a;
    float *pp = W.p;
    const float *psp = S.a.p;
    ACC *g1p = (ACC *)S.g1, *ilp = (ACC *)S.illum;
    const float *rowbase = st + (U * r) * WW + 4 * g;                       // vx row of grid row zr, word of column x-12
    const float *colbase = st + Stage<BZ>::p_vz + (U * r) * BX + 4 * g;     // the group's first staged vz row
    const float *op = st + Stage<BZ>::p_op + (U * r) * BX + 4 * g;
    // the increment dxs + dzs as dxs - (-dzs); the reconstruction's, which it adds, negated
    const float dtx = MODE == 3 ? -a.dtx : a.dtx, mdtz = MODE == 3 ? a.dtz : -a.dtz;
    const auto cx = [&](int, int i) { return a.c2[i]; };
    const auto cz = [&](int, int, int i) { return a.c2[i]; };
    const unsigned id0 = (unsigned)zr * pitch + x;

    constexpr bool staged = BZ <= 16;
    const float *ex = op + 2 * BZ * BX;   // the stage's further operands (fill_pres)
    constexpr int w = (int)sizeof(ACC) / 4;
    const ACC *g1s = (const ACC *)(st + Stage<BZ>::p_op + 3 * BZ * BX) + (U * r) * BX + 4 * g;
    const ACC *ils = (const ACC *)(st + Stage<BZ>::p_op + (3 + w) * BZ * BX) + (U * r) * BX + 4 * g;
    // imaging operands not staged: row 0's are loaded before the z-derivatives, row u+1's before
    // row u
    float4 ps[2];
    ACC og1[2][4], oil[2][4];
    const auto load_img = [&](int u) {
        ps[u & 1] = ldv4(&psp[id0 + u * pitch]);
        ld_acc4<ACC>(&g1p[id0 + u * pitch], og1[u & 1]);
        ld_acc4<ACC>(&ilp[id0 + u * pitch], oil[u & 1]);
    };
    const auto image = [&](int u, const float4 &pn) {   // kernel.cu:1401-1416
        const int k = u & 1;
        if (staged) {
            ps[k] = lds4(ex + u * BX);
            ld_acc4<ACC>(g1s + u * BX, og1[k]);
            ld_acc4<ACC>(ils + u * BX, oil[k]);
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            og1[k][j] = image_g1<ACC>(og1[k][j], comp(ps[k], j), comp(pn, j));
            oil[k][j] = image_il<ACC>(oil[k][j], comp(ps[k], j));
        }
        st_acc4<ACC>(&g1p[id0 + u * pitch], og1[k]);
        st_acc4<ACC>(&ilp[id0 + u * pitch], oil[k]);
    };

    if (t.interior & 1) {
        if (MODE == 2 && !staged) load_img(0);
        P4 dz[U];
        dz_sum<U, BX>(colbase, dz, cz);
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (MODE == 2 && !staged && u + 1 < U) load_img(u + 1);
            const P4 dx = dx_sum<11, 12>(rowbase + u * WW, cx);
            const P4 kk = p4(lds4(op + u * BX)), p0 = p4(lds4(op + (BZ + u) * BX));
            const P4 maz = mul(mul(dz[u], mdtz), kk);
            float4 pn;
            if (MODE == 0 && a.fuse) {   // p0 - fma(ax, kk, az) as p0 + fma(-ax, kk, -az)
                const P4 nax = mul(dx, -a.dtx);
                pn = q4({__fadd2_rn(p0.a, __ffma2_rn(nax.a, kk.a, maz.a)), __fadd2_rn(p0.b, __ffma2_rn(nax.b, kk.b, maz.b))});
            } else {
                pn = q4(sub(p0, sub(mul(mul(dx, dtx), kk), maz)));
            }
            st4(&pp[id0 + u * pitch], pn);
            if (MODE == 2) image(u, pn);
        }
        return;
    }

    const int X = S.X, Z = S.Z, npml = S.npml, F = t.interior;
    // (the reconstruction leaves every column outside [npml-R, X-npml+R) alone)
    if (x >= X || zr >= Z || (MODE == 3 && (x + 4 <= npml - R || x >= X - npml + R))) return;
    // image-interior columns, and the strip columns of p
    unsigned min_ = 15u, msl = 0u, msr = 0u;
    if (F & RTM_TILE_XBAND) {
        min_ = cols_in(x, npml, X - npml);
        if (MODE == 3 || MODE == 0) {
            msl = cols_in(x, npml - R, npml);
            msr = cols_in(x, X - npml, X - npml + R);
        }
    }
    // split fields (staged in band tiles, except the receiver pass's that hold image cells)
    const bool band_st = staged && (MODE == 0 || !(F & RTM_TILE_IMG));
    float4 s1[2], s2[2];
    float *sxp = W.sx, *szp = W.sz;
    const auto load = [&](int u) {
        const int z = zr + u, k = u & 1;
        const bool zin = z >= npml && z < Z - npml;
        if (z >= Z) return;
        if (MODE != 3 && (min_ != 15u || !zin)) {
            if (band_st) {
                s1[k] = lds4(ex + u * BX);
                s2[k] = lds4(ex + (BZ + u) * BX);
            } else {
                s1[k] = ldv4(&sxp[id0 + u * pitch]);
                s2[k] = ldv4(&szp[id0 + u * pitch]);
            }
        }
        if (MODE == 2 && !staged && zin && min_) load_img(u);
    };
    load(0);
    // local order of a cell (cuda_norder): the distance to the nearest edge in x or z, at most
    // R; 0 on the edge itself, which keeps its pressure
    const auto order = [&](int xj, int z) { return min(min(min(xj, X - 1 - xj), min(z, Z - 1 - z)), R); };
    const bool edge = MODE != 3 && (U == 1 || (F & RTM_TILE_XEDGE) || zr < R || zr + U > Z - R);
    const float2 *ec[U][2];   // edge groups: the coefficients of the row's two column pairs
    if (edge) {
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
            for (int h = 0; h < 2; h++)
                ec[u][h] = pair_row(s_tab, order(x + 2 * h, zr + u), order(x + 2 * h + 1, zr + u));
    }
    const auto ecoef = [&](int u, int h, int i) { return ec[u][h][i]; };
    P4 dz[U];
    if (!edge) dz_sum<U, BX>(colbase, dz, cz);
    else dz_sum<U, BX>(colbase, dz, ecoef);
    const int nxi = S.nxi, nzi = S.nzi;
    const bool save = MODE == 0 && a.save;
    // strip cells of column x in row zr: p left and right of the interior (R apart per row), and in
    // row 0 of the strips above and below it
    const int ps0 = 2 * R * (nzi + nxi), sl = ps0 + (zr - npml) * R + x - (npml - R),
              sr = ps0 + (nzi + zr - npml) * R + x - (X - npml), stb = ps0 + 2 * R * nzi + x - npml;
    float *strips = save ? strip_dst(a, S) : nullptr;
    const size_t s0 = (size_t)a.it * S.strip_len;
    float scx = 1.0f, scz = 1.0f;
    if (MODE == 3 && a.strip_prec) {
        scx = S.strip_scale[(size_t)a.it * 4 + 2];
        scz = S.strip_scale[(size_t)a.it * 4 + 3];
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        const int z = zr + u;
        if (z >= Z) break;
        const unsigned id = id0 + u * pitch;
        const int k = u & 1;
        if (u + 1 < U) load(u + 1);
        const bool zin = z >= npml && z < Z - npml;
        const int srow = (MODE == 3 || save) && !zin ? strip_row_tb(z, npml, Z - npml, nxi) : -1;
        unsigned ml = 0u;   // restored columns
        float rp[4];
        if (MODE == 3) {   // read_d_ppmllr, read_d_ppmltb (kernel.cu:1348-1400)
            ml = zin ? msl | msr : srow >= 0 ? min_ : 0u;
            if (zin && msl) strip_get(rp, S.strips, s0 + sl + u * R, msl, a.strip_prec, scx);
            if (zin && msr) {
                float q[4];
                strip_get(q, S.strips, s0 + sr + u * R, msr, a.strip_prec, scx);
#pragma unroll
                for (int j = 0; j < 4; j++)
                    if (msr >> j & 1) rp[j] = q[j];
            }
            if (srow >= 0 && min_) strip_get(rp, S.strips, s0 + stb + srow, min_, a.strip_prec, scz);
        }
        P4 dx;
        if (!edge) dx = dx_sum<11, 12>(rowbase + u * WW, cx);
        else dx = dx_sum<11, 12>(rowbase + u * WW, [&](int h, int i) { return ecoef(u, h, i); });
        const P4 kk = p4(lds4(op + u * BX));
        const float4 p0 = lds4(op + (BZ + u) * BX);
        const P4 dxs = mul(mul(dx, dtx), kk), mdzs = mul(mul(dz[u], mdtz), kk);
        const float4 inner = q4(sub(p4(p0), sub(dxs, mdzs)));
        float pn[4];
        bool wr = true;
        if (MODE == 3) {
            // reconstruction: kernel.cu:389-429, strips of step it, source subtracted
            const unsigned up = zin ? min_ : 0u;
            float4 n = pick(up, inner, p0);
            if (ml) n = pick(ml, f4(rp), n);
            pn[0] = n.x; pn[1] = n.y; pn[2] = n.z; pn[3] = n.w;
            wr = (up | ml) != 0;
        } else {
            // kernel.cu:501-541 (interior) and :714-1185 (split-field PML)
            const unsigned in = zin ? min_ : 0u;
            float4 n = inner;
            unsigned upd = 15u;   // cells that the update writes: not the grid's edge, nor the row padding
            if (edge || (F & RTM_TILE_XBAND)) {
                upd = 0u;
#pragma unroll
                for (int j = 0; j < 4; j++) upd |= (unsigned)(x + j < X && order(x + j, z) > 0) << j;
            }
            if (in != 15u) {
                const P4 n1 = damp(p4(s1[k]), dxs, p4(lds4(&m.c1x[4 * g])), p4(lds4(&m.ic2x[4 * g])));
                const float2 c1 = both(-m.c1z[U * r + u]), ic2 = both(-m.ic2z[U * r + u]);
                // (damp of -dzs with negated factors: c1 s - dzs as -((-c1) s - (-dzs)))
                const P4 n2 = damp(p4(s2[k]), mdzs, {c1, c1}, {ic2, ic2});
                const float4 e1 = q4(n1), e2 = q4(n2);
                const float4 e = make_float4(__fadd_rn(e1.x, e2.x), __fadd_rn(e1.y, e2.y), __fadd_rn(e1.z, e2.z),
                                             __fadd_rn(e1.w, e2.w));
                n = in ? pick(in, n, e) : e;
                const unsigned w = upd & ~in;
                st4(&sxp[id], w == 15u ? e1 : pick(w, e1, s1[k]));
                st4(&szp[id], w == 15u ? e2 : pick(w, e2, s2[k]));
            }
            if (upd != 15u) n = pick(upd, n, p0);
            pn[0] = n.x; pn[1] = n.y; pn[2] = n.z; pn[3] = n.w;
        }
        if (MODE != 2 && (F & RTM_TILE_SRC) && (unsigned)(z - S.sbz0) < (unsigned)S.sbnz) {   // kernel.cu:36-47
            const float wit = a.wavelet[a.it];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int xj = x + j;
                if ((unsigned)(xj - S.sbx0) < (unsigned)S.sbnx && (MODE != 3 || (xj >= npml - R && xj < X - npml + R))) {
                    const float v = S.src[(z - S.sbz0) * S.sbnx + (xj - S.sbx0)];
                    if (MODE == 3) pn[j] -= v * wit;
                    else pn[j] += v * wit;
                    wr = true;
                }
            }
        }
        if ((F & RTM_TILE_REC) && z == S.rz && (MODE == 2 || (MODE == 0 && record))) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int xr = x + j - S.rx0;
                if ((unsigned)xr < (unsigned)S.nrec) {
                    if (MODE == 0) ((float *)S.gather)[(size_t)a.it * S.nrec + xr] = pn[j];   // kernel.cu:48-71
                    else pn[j] = a.dt * gather_at(a, S, xr);                                   // kernel.cu:72-95
                }
            }
        }
        if (wr) st4(&pp[id], f4(pn));
        if (MODE == 2 && zin && min_) image(u, f4(pn));
        if (save) {   // save_d_ppmllr, save_d_ppmltb (kernel.cu:1241-1293)
            if (zin && msl) strip_put(strips + sl + u * R, msl, pn);
            if (zin && msr) strip_put(strips + sr + u * R, msr, pn);
            if (srow >= 0) strip_put(strips + stb + srow, min_, pn);
        }
    }
}

// ---- the kernel -------------------------------------------------------------------------
__device__ __forceinline__ void mbar_arrive(unsigned long long *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_init_n(unsigned long long *bar, unsigned n)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(n) : "memory");
}

template <int BZ, int PM, int VM, typename ACC, bool THIN>
__global__ void __launch_bounds__(Pipe<BZ, PM, VM, ACC, THIN>::threads, Pipe<BZ, PM, VM, ACC, THIN>::blocks)
    k_pipe(const StepArgs a, int ntiles, int record)
{
    using P = Pipe<BZ, PM, VM, ACC, THIN>;
    constexpr int ST = P::stages, U = P::U, SB = P::bytes, NC = P::warps;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(16) StageMeta<BZ> s_meta[ST];
    __shared__ __align__(8) unsigned long long s_full[ST], s_empty[ST];
    __shared__ float2 s_tab[kPairs];
    // what does not depend on the kernel before this one: barriers, coefficients, the tile list
    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; s++) {
            mbar_init_n(&s_full[s], 1);
            mbar_init_n(&s_empty[s], NC);
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (PM == 0 || PM == 2 || VM == 0 || VM == 2)
        for (int i = threadIdx.x; i < kPairs; i += blockDim.x) s_tab[i] = pair_entry(a.coef, i);
    const int n = a.counts ? a.counts[a.list] : ntiles;   // fixed-grid launches: the batch's own count
    const int step = (int)gridDim.x, lane = threadIdx.x & 31;
    const auto is_pres = [&](const TileRef &t) { return VM < 0 || (PM >= 0 && !(t.interior & RTM_TILE_VEL)); };
    pdl_launch_dependents();
    __syncthreads();

    if (threadIdx.x >= 32 * NC) {   // the producer warp
        // the tile being filled and the one after it: in launches of many tiles per block every
        // step-th tile; in shorter ones, where a block with slow tiles would hold up the launch,
        // claimed from the counter, one fill ahead of the loads that need it (one shot of 1801x451:
        // blocks end after 17 / 22 / 32 us, first / median / last, with a stride and 21.7 / 23.1 / 24.3
        // claimed; at 64 shots, 100 tiles a block, claiming costs 1-2%)
        const bool dynamic = n <= 16 * step;
        // long lists run backwards in every other launch: what the launch before touched last is
        // still in L2
        const bool back = !dynamic && a.qsel;
        constexpr int W = sizeof(ShotDev) / 4, WL = (W + 31) / 32;
        TileRef t{};
        unsigned w[WL] = {};   // the next tile's shot descriptor, one word per lane and round
        const auto load = [&](int i) {
            t = a.tiles[back ? n - 1 - i : i];
            const unsigned *src = (const unsigned *)&a.shots[t.shot];
#pragma unroll
            for (int k = 0; k < WL; k++) w[k] = lane + 32 * k < W ? src[lane + 32 * k] : 0u;
        };
        int i = blockIdx.x, ahead = i + step;
        // into stage s: the loaded tile's descriptor
        const auto begin = [&](int s) {
            StageMeta<BZ> &m = s_meta[s];
            unsigned *dst = (unsigned *)&m.S;
#pragma unroll
            for (int k = 0; k < WL; k++)
                if (lane + 32 * k < W) dst[lane + 32 * k] = w[k];
            if (lane == 0) m.t = t;
            __syncwarp();
        };
        if (i < n) {
            load(i);
            begin(0);
            if (lane == 0) {
                if (is_pres(t)) {
                    if constexpr (PM >= 0) fill_pres_const<BZ, PM, ACC>(s_meta[0], (float *)smem, &s_full[0]);
                } else {
                    if constexpr (VM >= 0) fill_vel_const<BZ, VM>(s_meta[0], (float *)smem, &s_full[0]);
                }
            }
        }
        pdl_wait();
        if (blockIdx.x == 0 && lane == 0) a.queue[a.qsel ^ 1] = 0u;   // (the launch before has finished with it)
        const auto claim = [&] { return lane == 0 ? step + (int)atomicAdd(&a.queue[a.qsel], 1u) : 0; };
        int s = 0;
        unsigned parity = 1;   // the first use of a stage waits for no one
        for (int k = 0;; k++) {   // k: stages filled so far
            constexpr int M = offsetof(ShotDev, tmaps) / 4;   // (the shot's tensor maps, from the loaded words)
            const unsigned m0 = __shfl_sync(0xffffffffu, w[M / 32], M % 32);
            const unsigned m1 = __shfl_sync(0xffffffffu, w[(M + 1) / 32], (M + 1) % 32);
            const char *maps = (const char *)((unsigned long long)m1 << 32 | m0);
            if (!tile_wait(&s_empty[s], a.err, parity)) {
                // the consumers are gone: leave when the copies in flight have landed (bounded)
                for (int q = 0; q < ST; q++)
                    if (const int fills = (k + ST - 1 - q) / ST) tile_wait(&s_full[q], a.err, (fills - 1) & 1);
                return;
            }
            if (i >= n) {   // no tile left: tell the consumers
                if (lane == 0) {
                    s_meta[s].t.shot = -1;
                    mbar_arrive(&s_full[s]);
                }
                return;
            }
            float *st = (float *)(smem + s * SB);
            if (is_pres(t)) {
                if constexpr (PM >= 0) {
                    if (lane == 0) fill_pres<BZ, PM, ACC>(maps, t, st, &s_full[s]);
                    if (k > 0) {
                        begin(s);
                        if (lane == 0) fill_pres_const<BZ, PM, ACC>(s_meta[s], st, &s_full[s]);
                    }
                    const ShotDev &S = s_meta[s].S;
                    if (a.prefetch && PM != 3) {
                        const WaveDev &W_ = PM == 2 ? S.b : S.a;
                        const int z1 = min(t.z0 + BZ, S.Z);
                        if ((t.interior & RTM_TILE_BAND) && (!P::staged || (PM == 2 && (t.interior & RTM_TILE_IMG)))) {
                            prefetch_tile(W_.sx, 4, t.z0, z1, t.x0, S.pitch);
                            prefetch_tile(W_.sz, 4, t.z0, z1, t.x0, S.pitch);
                        }
                        if (PM == 2 && !P::staged) {   // imaging operands of the interior rows
                            const int i0 = max(t.z0, S.npml), i1 = min(z1, S.Z - S.npml);
                            prefetch_tile(S.a.p, 4, i0, i1, t.x0, S.pitch);
                            prefetch_tile(S.g1, (int)sizeof(ACC), i0, i1, t.x0, S.pitch);
                            prefetch_tile(S.illum, (int)sizeof(ACC), i0, i1, t.x0, S.pitch);
                        }
                    }
                }
            } else {
                if constexpr (VM >= 0) {
                    if (lane == 0) fill_vel<BZ, VM>(maps, t, st, &s_full[s]);
                    if (k > 0) {
                        begin(s);
                        if (lane == 0) fill_vel_const<BZ, VM>(s_meta[s], st, &s_full[s]);
                    }
                }
            }
            if (k == 0 && dynamic) ahead = claim();
            if (lane == 0) mbar_arrive(&s_full[s]);
            i = __shfl_sync(0xffffffffu, ahead, 0);
            if (i < n) {
                ahead = dynamic ? claim() : i + step;
                load(i);
            }
            if (++s == ST) {
                s = 0;
                parity ^= 1;
            }
        }
    }

    int s = 0;
    unsigned parity = 0;
    pdl_wait();
    for (;;) {
        if (!tile_wait(&s_full[s], a.err, parity)) return;
        const TileRef t = s_meta[s].t;
        if (t.shot < 0) return;
        const float *st = (const float *)(smem + s * SB);
        if (is_pres(t)) {
            if constexpr (PM >= 0) pres_compute<BZ, U, PM, ACC>(a, s_meta[s], t, st, s_tab, record);
        } else {
            if constexpr (VM >= 0) vel_compute<BZ, U, VM>(a, s_meta[s], t, st, s_tab, PM == 2 ? a.it : a.it + 1);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&s_empty[s]);   // this warp has read the stage
        if (++s == ST) {
            s = 0;
            parity ^= 1;
        }
    }
}

// ---- host launchers ---------------------------------------------------------------------
template <int BZ, int PM, int VM, typename ACC, bool THIN>
void pipe_launch_v(const StepArgs &a, int ntiles, int record, cudaStream_t st)
{
    using P = Pipe<BZ, PM, VM, ACC, THIN>;
    // every launch of b blocks per SM takes a b-th of the SM's shared memory for each: a block of the
    // next launch, which starts when a block of this one ends, then fits the room that it leaves (with
    // each kernel's own size the rooms left over were too small for a third block, and a launch of
    // 8-row tiles ran in two waves: modelling 64 shots of 1801x451 724 us a step, 524 without the
    // early starts, 16 shots' migration 451 and, with equal rooms, 403)
    constexpr size_t used = (size_t)P::stages * P::bytes;
    constexpr size_t own = 1024 + P::stages * (sizeof(StageMeta<BZ>) + 16) + (PM == 3 && VM < 0 ? 0 : kPairs * sizeof(float2));
    constexpr size_t room = (228 * 1024 / P::blocks - own) / 128 * 128;
    constexpr size_t bytes = P::blocks > 1 && room > used ? room : used;
    // the shared-memory limit is an attribute of the instance on each device; the resident
    // blocks per device follow from it (looked up once per device)
    static std::atomic<int> slots[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return;   // the launch would report the error
    int cap = dev < 64 ? slots[dev].load(std::memory_order_acquire) : 0;
    if (!cap) {
        int sms = 0, per = 0;
        cudaFuncSetAttribute(k_pipe<BZ, PM, VM, ACC, THIN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_pipe<BZ, PM, VM, ACC, THIN>, P::threads, bytes);
        cap = sms * (per > 0 ? per : 1);
        if (dev < 64) slots[dev].store(cap, std::memory_order_release);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ntiles < cap ? ntiles : cap);
    cfg.blockDim = dim3(P::threads);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k_pipe<BZ, PM, VM, ACC, THIN>, a, ntiles, record);
}

// The 8-row tiles' launches of up to two tiles per SM take the thin shape (one row per thread, 8
// consumer warps): every tile is then resident at once and a launch lasts as long as one tile's
// chain of wait, sums and stores, which is shorter with half the rows per thread. A step of
// 401x201 (248 tiles per launch) 21.7 us with U = 2 and 19.0 us thin, 201x101 20.2 and 18.4 us;
// with more tiles than that the wide shape's fewer instructions and shared-memory reads per cell
// count: 1701x351 at any length 36.1 us wide and 39.8 thin, 12 shots of 481x331 104.6 and 118.6 us.
constexpr int kThinTiles = 296;
template <int BZ, int PM, int VM, typename ACC>
void pipe_launch_t(const StepArgs &a, int ntiles, int record, cudaStream_t st)
{
    if constexpr (BZ == 8)
        if (ntiles <= kThinTiles) return pipe_launch_v<BZ, PM, VM, ACC, true>(a, ntiles, record, st);
    pipe_launch_v<BZ, PM, VM, ACC, false>(a, ntiles, record, st);
}

}  // namespace

#define RTM_CAT_(a, b) a##b
#define RTM_CAT(a, b) RTM_CAT_(a, b)
void RTM_CAT(launch_pipe_, RTM_PIPE_BZ)(int pm, int vm, const StepArgs &a, int ntiles, int record, cudaStream_t st)
{
    constexpr int BZ = RTM_PIPE_BZ;
    if (pm < 0) {
        if (vm == 0) pipe_launch_t<BZ, -1, 0, float>(a, ntiles, record, st);
        else if (vm == 2) pipe_launch_t<BZ, -1, 2, float>(a, ntiles, record, st);
        else pipe_launch_t<BZ, -1, 3, float>(a, ntiles, record, st);
    } else if (pm == 0) {
        pipe_launch_t<BZ, 0, -1, float>(a, ntiles, record, st);
    } else if (pm == 3) {
        if (vm < 0) pipe_launch_t<BZ, 3, -1, float>(a, ntiles, record, st);
        else pipe_launch_t<BZ, 3, 2, float>(a, ntiles, record, st);
    } else if (vm < 0) {
        if (a.accum_fp64 == RTM_ACC_FP64) pipe_launch_t<BZ, 2, -1, double>(a, ntiles, record, st);
        else if (a.accum_fp64 == RTM_ACC_KAHAN) pipe_launch_t<BZ, 2, -1, KahanAcc>(a, ntiles, record, st);
        else pipe_launch_t<BZ, 2, -1, float>(a, ntiles, record, st);
    } else {
        if (a.accum_fp64 == RTM_ACC_FP64) pipe_launch_t<BZ, 2, 3, double>(a, ntiles, record, st);
        else if (a.accum_fp64 == RTM_ACC_KAHAN) pipe_launch_t<BZ, 2, 3, KahanAcc>(a, ntiles, record, st);
        else pipe_launch_t<BZ, 2, 3, float>(a, ntiles, record, st);
    }
}
