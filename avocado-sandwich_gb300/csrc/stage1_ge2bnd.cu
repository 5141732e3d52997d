// Stage 1: tile QR/LQ block-bidiagonalisation (GE2BND), FP64 and FP32 tiles.
//
// Reference: Blockbidiag! (KAbasedSVD/src/tiledalgos.jl:17-59) on the tile
// views of KAbasedSVD/src/TiledMatrix.jl:77-113, with the GEQRT / TSQRT tile
// kernels of KAbasedSVD/src/QRkernels.jl:3-129 and the reflector applies of
// QRkernels.jl:131-197.
//
// Each GE2BND step k is two half-steps, both written as "QR of a column panel
// plus left-apply to the trailing columns" on a view of the matrix:
//   QR half: view = A,   top tile row pr = k,   panel column tile pc = k
//   LQ half: view = A^T, top tile row pr = k+1, panel column tile pc = k
// (the reference runs the LQ half as QR kernels on adjoint views,
//  TiledMatrix.jl:85-88, 98-102).
//
// Panel kernel.  Role 0 runs GEQRT on the top tile; role p >= 1 runs TSQRT on
// [R; tile p], exactly the flat tree of the reference.  Reflectors of
// different roles that touch different rows commute, and step i of a TSQRT block
// reads row i of the block's diagonal block only, so role p runs its step i as soon
// as role p-1 has finished step i: the roles form a systolic pipeline over the row
// tiles whose critical path is one hand-off per tile plus the reflector steps of one
// tile, instead of #tiles * b reflector steps.  Within a block the 16 reflectors are
// generated one column at a time, and the block is applied to the rest of the tile
// in compact-WY form (16 reflectors).  A role hands block cb on in two parts: the
// rows of the 16 x 16 diagonal block one by one as its reflectors make them (all the
// next role's reflectors read), and the trailing top rows after its apply (which the
// next role reads only in its own apply).  Roles are handed out by an atomic ticket in
// launch order,
// so a role only ever waits on a role already running: no co-residency
// assumption, and every wait is bounded.  The panel computes in its tile type,
// except with the double-float trailing updates of FP64 tiles (AVS_PREC_FP64X2),
// where it computes in double-float too (FP64 storage).  In the lookahead of the
// tensor-core path (stage1_ge2bnd_tc) a role may also wait for its own tile,
// which the previous update's chain finishes on the other stream.
//
// Trailing update kernels: per column the serial order of the reference's
// Qtapply1_par! / Qtapply2_par! (TiledMatrix.jl:107-113) -- the GEQRT blocks, then row
// tile by row tile the TSQRT blocks, compact WY per 16 reflectors -- all columns in
// parallel.  update_kernel (tiles of 32 and 64, and FP64 tiles of 16): a CTA takes a
// ticket for a (tile group, column strip) and receives the strip of the top tile row
// from the CTA of the group before through global memory, block of 16 rows by block,
// behind counters.  update16_kernel (FP32 tiles of 16): a CTA per 16-column strip
// walks all tiles.  Tiles of 128 and 256: update_full_kernel (stage1_wy.cu).
//
// Householder vectors stay where the reference leaves them before it zeroes
// them (tiledalgos.jl:40,46,52,58); later stages read only the band, so the
// zeroing launches are not needed.
#include <algorithm>
#include <cmath>
#include <cstdio>

#include <type_traits>

#include "avs_common.cuh"
#include "df64.cuh"
#include "reflect.cuh"
#include "vec16.cuh"

namespace avs {
namespace {

constexpr int kIB = 16;    // reflectors per compact-WY block

struct PanelArgs {
    void *a;
    int64_t lda;
    int b;
    int pr, pc;      // top tile row, panel tile column (view coordinates)
    int P;           // number of roles (tiles in the panel)
    int first_role;  // 0, or 1 for a lone TSQRT
    void *tau;       // [P][b]
    void *tblk;      // [P][b/kIB][kIB*kIB]
    int *ticket;
    int *progress;   // [2P]: diagonal block handed on, trailing top rows handed on
    int *err;
    const int *ready;  // optional: role p's tile is final once ready[p] >= ready_need
    int ready_need;
    unsigned long long *mail;  // optional: rows of the diagonal blocks, role to role (tagged words)
    unsigned tag;              // this launch's tag, never 0
    const void *ref;  // optional: the b diagonal values of the call's first panel, at ref_ld, sRef per matrix
    int64_t ref_ld, sRef;
    int64_t sA, sTau, sTblk, sFlags, sMail;  // per-matrix strides (blockIdx.y = matrix)
};

struct UpdateArgs {
    void *a;
    int64_t lda;
    int64_t n;
    int b;
    int pr, pc, P;
    int first_role;  // 1: the top tile's own (GEQRT) blocks were applied earlier
    int nstrip;      // column strips
    int group;       // consecutive tiles per CTA
    const void *tblk;
    int fine;        // 1: a counter per block of a strip, 0: one per strip
    int *flags;      // [0] ticket, then the counters: tiles done with the block (the strip); zeroed
    int *err;
    int64_t sA, sTblk, sFlags;  // per-matrix strides (blockIdx.y = matrix)
};

// ---------------------------------------------------------------------------
// Panel arithmetic by compute type.  Sq: a sum of squares (compensated pairs
// (sum, error) for FP32 and double-float, merged without renormalising between
// levels; plain for FP64).  scalars: the reference's expressions
// (QRkernels.jl:27-31) in closed form: n1 = ||x||, nu = alpha + sign(alpha) n1,
// tau = 2 nu^2 / (s + nu^2) = |nu| / n1, tc = tau / nu = sign(nu) / n1,
// f = tau / nu^2 = 1 / (n1 |nu|), inv = 1 / nu, beta = -sign(alpha) n1 (the new
// diagonal); evaluated in double-float for FP32 tiles and rounded once, in FP64
// for FP64 tiles (reflect.cuh: hardware estimates and one residual each).  They are
// meaningless for a zero column; small: the squared norm is 0, or so small that f may
// overflow (or NaN); vanished: it is 0, a zero column for FP32 and double-float, an
// error for FP64 if alpha != 0.
template <typename CT>
struct PRefl {
    CT nu, tc, f, inv, beta, tau;
};

template <typename CT>
struct PAr;
constexpr float kSmallF = 0x1.02p-128f;  // n1 |nu| >= n1^2 above it: f below 2^128

struct PSqPair {
    using Sq = float2;
    static __device__ __forceinline__ Sq merge(Sq a, Sq b) {
        const df64 t = two_sum(a.x, b.x);
        return make_float2(t.hi, __fadd_rn(t.lo, __fadd_rn(a.y, b.y)));
    }
    static __device__ __forceinline__ Sq merge_xor(Sq a, int o) {
        return merge(a, make_float2(__shfl_xor_sync(0xffffffffu, a.x, o), __shfl_xor_sync(0xffffffffu, a.y, o)));
    }
};
template <>
struct PAr<float> : PSqPair, MacAr<float> {
    static __device__ __forceinline__ Sq sq(float x) {
        const float p = __fmul_rn(x, x);
        return make_float2(p, __fmaf_rn(x, x, -p));
    }
    // The two hardware estimates start as soon as their arguments are known to
    // FP32 and everything else is a residual of them: with r ~ 1/n1 and z ~ 1/|nu|,
    // n1 = x r (1 + g), 1/n1 = r (1 + g), 1/|nu| = z (1 + k); relative errors
    // below 2^-44 before the one rounding of each result.
    static constexpr bool kFp64 = false;
    static __device__ __forceinline__ bool small(Sq s, float alpha) { return !(fmaf(alpha, alpha, s.x) > kSmallF); }
    static __device__ __forceinline__ bool vanished(Sq s, float alpha) { return fmaf(alpha, alpha, s.x) <= 0.0f; }
    static __device__ __forceinline__ PRefl<float> scalars(Sq s, float alpha) {
        PRefl<float> o;
        const float xa = fmaf(alpha, alpha, s.x);  // n1^2 to FP32
        const float r = rsqrt_hw(xa);
        const df64 a2 = two_prod(alpha, alpha);
        const df64 x = two_sum(a2.hi, s.x);
        const float xl = __fadd_rn(x.lo, __fadd_rn(a2.lo, s.y));
        const float t = __fmul_rn(x.hi, r);
        const float tl = __fmaf_rn(xl, r, __fmaf_rn(x.hi, r, -t));
        const float aa = fabsf(alpha);
        const df64 u = two_sum(aa, t);
        const float z = rcp_hw(u.hi);
        const float e = __fmaf_rn(-tl, r, __fmaf_rn(-t, r, 1.0f));
        const float g = __fmul_rn(e, __fmaf_rn(0.375f, e, 0.5f));
        const float nl = __fmaf_rn(t, g, tl);   // n1 = t + nl
        const float ul = __fadd_rn(u.lo, nl);   // |nu| = u.hi + ul
        const float ez = __fmaf_rn(-ul, z, __fmaf_rn(-u.hi, z, 1.0f));
        const float k = __fmaf_rn(ez, ez, ez);
        const bool neg = alpha < 0.0f;
        const float nu = __fadd_rn(u.hi, ul), n1 = __fadd_rn(t, nl);
        const float rn = __fmaf_rn(r, g, r), inv = __fmaf_rn(z, k, z);
        const float p = __fmul_rn(u.hi, r);
        o.tau = __fadd_rn(p, __fmaf_rn(p, g, __fmaf_rn(ul, r, __fmaf_rn(u.hi, r, -p))));
        const float q = __fmul_rn(r, z);
        o.f = __fadd_rn(q, __fmaf_rn(q, __fadd_rn(g, k), __fmaf_rn(r, z, -q)));
        o.nu = neg ? -nu : nu;
        o.tc = neg ? -rn : rn;
        o.inv = neg ? -inv : inv;
        o.beta = neg ? n1 : -n1;
        return o;
    }
};
// FP64 tiles in double-float arithmetic (AVS_PREC_FP64X2)
template <>
struct PAr<dfx> : PSqPair, MacAr<dfx> {
    static __device__ __forceinline__ Sq sq(dfx v) {
        const df64 x = v.v;
        const float p = __fmul_rn(x.hi, x.hi);
        return make_float2(p, __fmaf_rn(2.0f * x.hi, x.lo, __fmaf_rn(x.hi, x.hi, -p)));
    }
    static constexpr bool kFp64 = false;
    static __device__ __forceinline__ bool small(Sq s, dfx al) {
        const Sq m = merge(s, sq(al));
        return !(__fadd_rn(m.x, m.y) > kSmallF);
    }
    static __device__ __forceinline__ bool vanished(Sq s, dfx al) {
        const Sq m = merge(s, sq(al));
        return __fadd_rn(m.x, m.y) <= 0.0f;
    }
    static __device__ __forceinline__ PRefl<dfx> scalars(Sq s, dfx al) {
        PRefl<dfx> r;
        const df64 alpha = al.v;
        const Sq m = merge(s, sq(al));
        const df64 x = fast_two_sum(m.x, m.y);
        df64 rn, n1;
        rsqrt_sqrt(x, rn, n1);
        const bool neg = df_lt0(alpha);
        const df64 u = df_add(neg ? df_neg(alpha) : alpha, n1);
        const df64 iu = rcp_est(u);
        r.nu = dfx(neg ? df_neg(u) : u);
        r.tau = dfx(df_mul(u, rn));
        r.tc = dfx(neg ? df_neg(rn) : rn);
        r.inv = dfx(neg ? df_neg(iu) : iu);
        r.f = dfx(df_mul(rn, iu));
        r.beta = dfx(neg ? n1 : df_neg(n1));
        return r;
    }
};
template <>
struct PAr<double> : MacAr<double> {
    using Sq = double;
    static __device__ __forceinline__ Sq sq(double x) { return x * x; }
    static __device__ __forceinline__ Sq merge(Sq a, Sq b) { return a + b; }
    static __device__ __forceinline__ Sq merge_xor(Sq a, int o) { return a + __shfl_xor_sync(0xffffffffu, a, o); }
    static constexpr bool kFp64 = true;
    static __device__ __forceinline__ bool small(Sq s, double alpha) {
        return (__double2hiint(fma(alpha, alpha, s)) & 0x7ff00000) == 0;  // below 2^-1022
    }
    static __device__ __forceinline__ bool vanished(Sq s, double alpha) { return fma(alpha, alpha, s) == 0.0; }
    static __device__ __forceinline__ PRefl<double> scalars(Sq s, double alpha) {
        PRefl<double> r;
        const double x = fma(alpha, alpha, s);
        double rn, n1;
        rsqrt_sqrt(x, rn, n1);
        const bool neg = alpha < 0.0;
        const double u = fabs(alpha) + n1;
        const double iu = rcp_est(u);
        r.nu = neg ? -u : u;
        r.tau = u * rn;
        r.tc = neg ? -rn : rn;
        r.inv = neg ? -iu : iu;
        r.f = rn * iu;
        r.beta = neg ? n1 : -n1;
        return r;
    }
};

// Warp shuffles and finiteness of the panel's compute types.
__device__ __forceinline__ float vshfl_xor(float v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
__device__ __forceinline__ double vshfl_xor(double v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
__device__ __forceinline__ dfx vshfl_xor(dfx v, int o) {
    return dfx(df64{__shfl_xor_sync(0xffffffffu, v.v.hi, o), __shfl_xor_sync(0xffffffffu, v.v.lo, o)});
}
__device__ __forceinline__ bool vfinite(float v) { return isfinite(v); }
__device__ __forceinline__ bool vfinite(double v) { return (__double2hiint(v) & 0x7ff00000) != 0x7ff00000; }
__device__ __forceinline__ bool vfinite(dfx v) { return isfinite(v.v.hi) && isfinite(v.v.lo); }

// Magnitudes in order, as integers: the bits of |v| (FP64: of its upper word), -1 for
// Inf and NaN; and whether a magnitude is nothing against another (below the unit
// roundoff of the type, and less).
__device__ __forceinline__ int mag_bits(float v) {
    const int m = __float_as_int(v) & 0x7fffffff;
    return m < 0x7f800000 ? m : -1;
}
__device__ __forceinline__ int mag_bits(double v) {
    const int m = __double2hiint(v) & 0x7fffffff;
    return m < 0x7ff00000 ? m : -1;
}
__device__ __forceinline__ int mag_bits(dfx v) { return mag_bits(v.v.hi); }
template <typename CT>
__device__ __forceinline__ bool negligible(int m, int big) {
    constexpr int k = std::is_same<CT, float>::value ? (30 << 23) : (std::is_same<CT, dfx>::value ? (56 << 23) : (60 << 20));
    return m >= 0 && m < big - k;
}

// two sums of squares at a 16-byte aligned address
template <typename Sq>
struct PSq2;
template <>
struct PSq2<float2> {
    static __device__ __forceinline__ void ld(const float2 *p, float2 &a, float2 &b) {
        const float4 x = *reinterpret_cast<const float4 *>(p);
        a = make_float2(x.x, x.y);
        b = make_float2(x.z, x.w);
    }
};
template <>
struct PSq2<double> {
    static __device__ __forceinline__ void ld(const double *p, double &a, double &b) {
        const double2 x = *reinterpret_cast<const double2 *>(p);
        a = x.x;
        b = x.y;
    }
};
// 16 consecutive values of CT at a 16-byte aligned address in shared memory.
template <typename CT>
__device__ __forceinline__ void ld16(const CT *p, CT (&v)[kIB]) {
#pragma unroll
    for (int q = 0; q < kIB; q += PVec<CT>::VN) PVec<CT>::ld(p + q, v + q);
}
template <typename CT>
__device__ __forceinline__ void st16(CT *p, const CT (&v)[kIB]) {
#pragma unroll
    for (int q = 0; q < kIB; q += PVec<CT>::VN) PVec<CT>::st(p + q, v + q);
}
// RPL rows of one column of the view (LAYOUT 0: contiguous, 16-byte aligned).
template <typename T, int LAYOUT, typename CT, int RPL>
__device__ __forceinline__ void load_col(const View<T, LAYOUT> &V, int64_t r, int64_t c, CT (&v)[RPL]) {
    if (LAYOUT == 0) {
#pragma unroll
        for (int q = 0; q < RPL; q += PVec<T>::VN) {
            T w[PVec<T>::VN];
            PVec<T>::ldcg(&V(r + q, c), w);
#pragma unroll
            for (int e = 0; e < PVec<T>::VN; ++e) v[q + e] = CT(w[e]);
        }
    } else {
#pragma unroll
        for (int q = 0; q < RPL; ++q) v[q] = CT(__ldcg(&V(r + q, c)));
    }
}
template <typename T, int LAYOUT, typename CT, int RPL>
__device__ __forceinline__ void store_col(const View<T, LAYOUT> &V, int64_t r, int64_t c, const CT (&v)[RPL]) {
    if (LAYOUT == 0) {
#pragma unroll
        for (int q = 0; q < RPL; q += PVec<T>::VN) {
            T w[PVec<T>::VN];
#pragma unroll
            for (int e = 0; e < PVec<T>::VN; ++e) w[e] = (T)v[q + e];
            PVec<T>::st(&V(r + q, c), w);
        }
    } else {
#pragma unroll
        for (int q = 0; q < RPL; ++q) V(r + q, c) = (T)v[q];
    }
}

__device__ __forceinline__ void bar_named(int id, int cnt) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(cnt) : "memory");
}

// One value with its tag, role to role through L2: a 64-bit word {32 bits, tag},
// two of them for an 8-byte type.  A word is written and read whole, so a value
// whose tags are this launch's is complete, with no flag and no fence beside it.
__device__ __forceinline__ void mail_put(unsigned long long *at, float v, unsigned tag) {
    const unsigned long long w = ((unsigned long long)tag << 32) | __float_as_uint(v);
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(at), "l"(w) : "memory");
}
__device__ __forceinline__ void mail_put2(unsigned long long *at, unsigned a, unsigned b, unsigned tag) {
    const unsigned long long t = (unsigned long long)tag << 32;
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(at), "l"(t | a), "l"(t | b) : "memory");
}
__device__ __forceinline__ void mail_put(unsigned long long *at, double v, unsigned tag) {
    mail_put2(at, (unsigned)__double2loint(v), (unsigned)__double2hiint(v), tag);
}
__device__ __forceinline__ void mail_put(unsigned long long *at, dfx v, unsigned tag) {
    mail_put2(at, __float_as_uint(v.v.hi), __float_as_uint(v.v.lo), tag);
}
__device__ __forceinline__ bool mail_get(const unsigned long long *at, float &v, unsigned tag) {
    unsigned long long w;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(at) : "memory");
    v = __uint_as_float((unsigned)w);
    return (unsigned)(w >> 32) == tag;
}
__device__ __forceinline__ bool mail_get2(const unsigned long long *at, unsigned &a, unsigned &b, unsigned tag) {
    unsigned long long x, y;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "l"(at) : "memory");
    a = (unsigned)x;
    b = (unsigned)y;
    return (unsigned)(x >> 32) == tag && (unsigned)(y >> 32) == tag;
}
__device__ __forceinline__ bool mail_get(const unsigned long long *at, double &v, unsigned tag) {
    unsigned a, b;
    const bool ok = mail_get2(at, a, b, tag);
    v = __hiloint2double((int)b, (int)a);
    return ok;
}
__device__ __forceinline__ bool mail_get(const unsigned long long *at, dfx &v, unsigned tag) {
    unsigned a, b;
    const bool ok = mail_get2(at, a, b, tag);
    v = dfx(df64{__uint_as_float(a), __uint_as_float(b)});
    return ok;
}
__device__ __forceinline__ int ld_shared_volatile(const int *p) { return *reinterpret_cast<const volatile int *>(p); }

// ---------------------------------------------------------------------------
// Panel kernel (roles, schedule and outputs as described at the top).
//
// What bounds it: latency.  The critical path is (P - 1) reflector loops of 16
// steps with a hand-off each, plus b/16 whole blocks (reflectors, Gram matrix,
// apply), all on one SM per role.  So:
//   * the block's 16 columns live in registers, a lane owning one column's rows
//     of its half of the warp's 32 rows: a step's dot products and updates are in
//     the lane (one shuffle joins the halves), against the reflector's column
//     broadcast through shared memory; the norm is one butterfly of compensated
//     pairs beside them.  (With a row per lane the 16 dot products took a warp
//     reduce-scatter of 423 cycles a step.)  Across warps one shared-memory pass
//     and one barrier of the b / 32 reflector warps, none for tiles 16 and 32;
//   * a TSQRT step changes one row of the diagonal block only: each new row goes to
//     the next role at once, as tagged words through L2 that the next role's fetch warp
//     polls and lays in shared memory ahead of its reflectors (about 1.5 k cycles from
//     role to role; with whole blocks behind a counter the hand-off cost the 16 steps
//     too, 9.5 k: stage 1 of FP32 n = 1296 tile 16 49.3 -> 17.7 ms, n = 2048 tile 64 17.2
//     -> 11.3, n = 4096 tile 128 39.1 -> 32.5, split BF16 n = 5760 tile 128 49.2 -> 36.1,
//     FP64 n = 1024 tile 64 28.2 -> 20.6).  Only the last role writes the rows to the
//     matrix;
//   * the block reflector is applied from the Gram matrix, not from T: with
//     G = Y^T Y and T^-1 = diag(1/tau) + striu(G), W = T^T Z is the forward
//     substitution w_l = tau_l (z_l - sum_{m<l} G_ml w_m), one thread per
//     column; 16 unit right-hand sides beside them give T (an output, for the
//     trailing update);
//   * the trailing columns of the tile stay in shared memory for the role's
//     whole life: all of them for tiles up to 128, the last 128 of an FP32 tile of
//     256 (its first ones, and those of an 8-byte tile of 256, are read from L2);
//     the next block's 16 columns go from the apply to the next block in
//     registers;
//   * Z = Y^T C is split over column pairs and row ranges so that all warps
//     work whatever the columns left; C -= Y W runs two rows per thread.
// Measured (GB300; stage 1 of one call, before: runtime tile size, columns in
// shared memory, a row per lane, explicit T): FP32 n = 1296 tile 16 195 -> 75 ms,
// n = 1024 tile 64 20.4 -> 14.1, n = 4096 tile 128 91.8 -> 63.8, split BF16 n =
// 5760 tile 128 96.8 -> 49.8, n = 16384 tile 256 344 -> 276; FP64 n = 1024 tile 64
// 78.0 -> 43.0, double-float n = 2048 tile 128 103 -> 66; then the row hand-off above.
// A block of 16
// reflectors: 9.5 k cycles (tile 16), 14.5 k (64), 17 k (128), 21 k (256), before
// about 48 k.
// Who fetches a block's top rows: a warp of its own, a warp that the reflectors leave
// idle, or the first reflector warp (whole blocks, no mailbox).
enum : int { kFetchNone, kFetchIdle, kFetchOwn };
template <typename CT, int B>
struct PanelCfg {
    static constexpr int NB = B / kIB;
    static constexpr int NWR = B >= 32 ? B / 32 : 1;  // reflector warps
    static constexpr int RPL = (B >= 32 ? 32 : B) / 2;  // rows per lane
    static constexpr int NT = B >= 128 ? 256 : (B == 64 ? 128 : (B == 32 ? 64 : 32));
    // tiles up to 64 have the registers for one more warp (a ninth one would leave the
    // others 168), 128 has idle ones; at 256 every warp has reflector rows
    static constexpr int FETCH = B <= 64 ? kFetchOwn : (B == 128 ? kFetchIdle : (sizeof(CT) == 4 ? kFetchOwn : kFetchNone));
    static constexpr int NTL = NT + (FETCH == kFetchOwn ? 32 : 0);  // threads launched
    static constexpr int NW = NT / 32;
    static constexpr bool F4 = sizeof(CT) == 4;
    static constexpr int YLD = F4 ? 20 : 18;      // row stride of Y and W (16-byte rows, conflict-free vectors)
    static constexpr int CLD = B + (F4 ? 4 : 2);  // resident trailing columns: [column][row]
    static constexpr int RESC = B <= 128 ? B - kIB : (F4 ? 128 : 0);  // resident columns, the last of the tile
    static constexpr int S0 = B - RESC;           // first resident column
    static constexpr int KSMAX = F4 ? 8 : 4;
    static constexpr int NR = B > kIB ? B - kIB : kIB;  // trailing columns at most
    static constexpr bool STREAM = NB > 1 && RESC < NR;
    // split of Z = Y^T C over nw warps: wcol warps of 64 columns, ks row ranges
    __host__ __device__ static constexpr int wcol(int nc) { return (nc + 63) / 64; }
    __host__ __device__ static constexpr int ks(int nc, int nw) {
        const int k = nc > 0 ? nw / wcol(nc) : 1;
        const int k2 = k >= 8 ? 8 : (k >= 4 ? 4 : (k >= 2 ? 2 : 1));
        return k2 < KSMAX ? k2 : KSMAX;
    }
    // streamed columns of the nrest trailing ones, and the warps of each part
    __host__ __device__ static constexpr int nstream(int nrest) {
        return nrest > RESC ? nrest - RESC : 0;
    }
    __host__ __device__ static constexpr int warps_r(int nrest) { return nstream(nrest) > 0 ? (RESC > 0 ? NW / 2 : 0) : NW; }
    __host__ __device__ static constexpr int zsize(int nrest) {  // columns x row ranges of the partial Z
        const int ns = nstream(nrest), nr = nrest - ns, wr = warps_r(nrest);
        return (nr > 0 ? nr * ks(nr, wr) : 0) + (ns > 0 ? ns * ks(ns, NW - wr) : 0);
    }
    static constexpr int zcols() {
        int m = 0;
        for (int r = kIB; r <= NR; r += kIB) m = zsize(r) > m ? zsize(r) : m;
        return m;
    }
    static constexpr size_t smem_bytes() {  // in the order of the kernel's carving
        return 16 * NWR + sizeof(CT) * (2 * NWR * kIB + 2 * NWR * 32 + 2 * kIB + kIB + 2 * kIB * (kIB + 4) + kIB * kIB +
                                       (F4 ? NW * kIB * kIB : 0) + (size_t)B * YLD +
                                       (NB > 1 ? (size_t)NR * YLD + (size_t)kIB * zcols() + (size_t)RESC * CLD : 0));
    }
};

// The fetch warp of a TSQRT role, block cb: top row i from the role ahead, as soon as
// that role has made it, into dst; `rows` counts the rows in place.  Four rows are
// polled at a time, so that the poll's round trip is paid once for them.  Without a
// mailbox the whole block comes from the matrix, once the role ahead (if one runs)
// counts it done.  False: gave up (the reflector warps stop waiting and the role ends
// at their barrier).
template <typename T, int LAYOUT, typename CT, int NB>
__device__ __forceinline__ bool fetch_top(const View<T, LAYOUT> &V, int64_t top0, int64_t col0, int cb, bool follow,
                                          const unsigned long long *box, unsigned tag, const int *progress, CT *dst,
                                          int *rows, int *fail, int *err) {
    constexpr int MW = sizeof(CT) / 4;
    const int lane = threadIdx.x & 31, jc = lane & (kIB - 1), rr = lane >> 4;
    const int c0 = cb * kIB;
    auto give_up = [&]() {
        if (lane == 0) {
            *reinterpret_cast<volatile int *>(fail) = 1;
            __threadfence_block();
            *reinterpret_cast<volatile int *>(rows) = kIB * NB;
        }
        return false;
    };
    if (follow && box) {
        const unsigned long long *src = box + (size_t)cb * kIB * kIB * MW;
        const long long t0 = clock64();
        int done = 0;
#pragma unroll 1
        for (long long it = 0; done < kIB; ++it) {
            const int r0 = done + rr, r1 = done + 2 + rr;
            CT v0 = CT(0), v1 = CT(0);
            bool ok0 = r0 < kIB, ok1 = r1 < kIB;
            if (ok0 && jc >= r0) ok0 = mail_get(src + (r0 * kIB + jc) * MW, v0, tag);
            if (ok1 && jc >= r1) ok1 = mail_get(src + (r1 * kIB + jc) * MW, v1, tag);
            const unsigned b0 = __ballot_sync(0xffffffffu, ok0), b1 = __ballot_sync(0xffffffffu, ok1);
            int got = 0;  // rows done, done + 1, ... that are all here
            if ((b0 & 0xffffu) == 0xffffu) {
                got = 1;
                if ((b0 >> 16) == 0xffffu) {
                    got = 2;
                    if ((b1 & 0xffffu) == 0xffffu) got = (b1 >> 16) == 0xffffu ? 4 : 3;
                }
            }
            if (rr < got) dst[r0 * (kIB + 4) + jc] = v0;
            if (2 + rr < got) dst[r1 * (kIB + 4) + jc] = v1;
            if (got > 0) {
                __threadfence_block();
                __syncwarp();
                done += got;
                if (lane == 0) *reinterpret_cast<volatile int *>(rows) = c0 + done;
            } else if ((it & 15) == 15) {  // another role's failure, the bounds: every 16 polls
                int stop = 0;
                if (lane == 0) {
                    stop = ld_acquire(err) != kDevOk;
                    if (!stop && (it > kSpinLimit || clock64() - t0 > 2 * kWaitNs)) {
                        atomicCAS(err, kDevOk, kDevTimeout);
                        stop = 1;
                    }
                }
                if (__shfl_sync(0xffffffffu, stop, 0)) return give_up();
                if (it > 64) __nanosleep(20);
            }
        }
    } else {
        int ok = 1;
        if (follow && lane == 0) ok = wait_geq(progress, cb + 1, err) ? 1 : 0;
        if (!__shfl_sync(0xffffffffu, ok, 0)) return give_up();
        constexpr int RU = kIB * kIB / 32;  // all loads in flight
        T v[RU];
#pragma unroll
        for (int u = 0; u < RU; ++u) {
            const int idx = lane + u * 32;
            const int l = LAYOUT == 0 ? idx % kIB : idx / kIB;
            const int j = LAYOUT == 0 ? idx / kIB : idx % kIB;
            v[u] = __ldcg(&V(top0 + c0 + l, col0 + c0 + j));
        }
#pragma unroll
        for (int u = 0; u < RU; ++u) {
            const int idx = lane + u * 32;
            const int l = LAYOUT == 0 ? idx % kIB : idx / kIB;
            const int j = LAYOUT == 0 ? idx / kIB : idx % kIB;
            dst[l * (kIB + 4) + j] = CT(v[u]);
        }
        __threadfence_block();
        __syncwarp();
        if (lane == 0) *reinterpret_cast<volatile int *>(rows) = c0 + kIB;
    }
    return true;
}
// The reflector warps' wait for `need` top rows; returns the rows in place.
__device__ __forceinline__ int wait_rows(const int *rows, int need, int *fail, int *err) {
    int have = ld_shared_volatile(rows);
    if (have < need) {
        const long long t0 = clock64();
        for (long long it = 0; (have = ld_shared_volatile(rows)) < need; ++it) {
            if ((it & 1023) == 1023 && clock64() - t0 > 4 * kWaitNs) {  // the fetch warp gives up before this
                *reinterpret_cast<volatile int *>(fail) = 1;
                atomicCAS(err, kDevOk, kDevTimeout);
                break;
            }
        }
    }
    __syncwarp();
    return have;
}

template <typename T, int LAYOUT, typename CT, int B>
__global__ void __launch_bounds__(PanelCfg<CT, B>::NTL) panel_kernel(PanelArgs args) {
    using Cfg = PanelCfg<CT, B>;
    using Ar = PAr<CT>;
    using Sq = typename Ar::Sq;
    using Mac = typename Ar::Mac;
    constexpr int NB = Cfg::NB, NWR = Cfg::NWR, NT = Cfg::NT, NW = Cfg::NW, YLD = Cfg::YLD, CLD = Cfg::CLD;
    constexpr int RPL = Cfg::RPL, RESC = Cfg::RESC, S0 = Cfg::S0;
    constexpr int TV = PVec<T>::VN, CV = PVec<CT>::VN;
    constexpr int MW = sizeof(CT) / 4;  // mailbox words per value
    static_assert(sizeof(Sq) == 8 && sizeof(CT) == sizeof(T), "panel types");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Sq *spart = reinterpret_cast<Sq *>(smem_raw);                 // [2][NWR]
    CT *part = reinterpret_cast<CT *>(spart + 2 * NWR);           // [2][16][NWR]
    CT *xs = part + 2 * NWR * kIB;                                // [2][NWR][32] the step's column
    CT *rowb = xs + 2 * NWR * 32;                                 // [2][16]
    CT *stau = rowb + 2 * kIB;                                    // [16]
    CT *Rbuf = stau + kIB;                                        // [2][16][20], block cb's top rows [l * 20 + j]
    CT *G = Rbuf + 2 * kIB * (kIB + 4);                              // [16][16], G[l * 16 + m] = y_l^T y_m
    CT *Gp = G + kIB * kIB;                                       // FP32: [NW][16][16]
    CT *Yr = Gp + (Cfg::F4 ? NW * kIB * kIB : 0);                 // [B][YLD]
    CT *Ws = Yr + (size_t)B * YLD;                                // [columns][YLD]
    CT *Zp = Ws + (NB > 1 ? (size_t)Cfg::NR * YLD : 0);           // [row range][16][columns], both parts
    CT *Cs = Zp + (NB > 1 ? (size_t)kIB * Cfg::zcols() : 0);      // [column - S0][CLD]

    __shared__ int s_role, s_ok, s_fail;
    __shared__ int s_rows, s_used;  // top rows fetched, blocks whose reflectors are done
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int64_t zb = blockIdx.y;
    int *progress = args.progress + zb * args.sFlags;
    if (tid == 0) {
        s_role = atomicAdd(args.ticket + zb * args.sFlags, 1) + args.first_role;
        s_fail = 0;
        s_rows = s_used = 0;
    }
    __syncthreads();
    const int p = s_role;
    if (p >= args.P) return;

    View<T, LAYOUT> V{reinterpret_cast<T *>(args.a) + zb * args.sA, args.lda};
    const int64_t row0 = (int64_t)(args.pr + p) * B;
    const int64_t top0 = (int64_t)args.pr * B;
    const int64_t col0 = (int64_t)args.pc * B;
    const bool geqrt = (p == 0);
    const bool follow = !geqrt && p > args.first_role;  // another role runs ahead
    T *tau_out = reinterpret_cast<T *>(args.tau) + zb * args.sTau + (size_t)p * B;
    T *tblk_out = reinterpret_cast<T *>(args.tblk) + zb * args.sTblk + (size_t)p * NB * kIB * kIB;

    if (args.ready) {  // the tile is still being written by the previous update's chain
        if (tid == 0) s_ok = wait_geq(args.ready + p, args.ready_need, args.err);
        __syncthreads();
        if (!s_ok) return;
    }
    int *full = progress + args.P;  // per role: block cb's trailing top rows are final

    const bool mail = Cfg::FETCH != kFetchNone && args.mail != nullptr;
    const bool last = p == args.P - 1;
    unsigned long long *box = mail ? args.mail + zb * args.sMail + (size_t)p * NB * kIB * kIB * MW : nullptr;
    const unsigned long long *from = mail && !geqrt ? box - (size_t)NB * kIB * kIB * MW : nullptr;
    if constexpr (Cfg::FETCH == kFetchOwn) {  // a warp of its own: a block ahead of the reflectors
        if (wid == NW) {
            if (geqrt) return;
            for (int cb = 0; cb < NB; ++cb) {
                const long long t0 = clock64();
                for (long long it = 0; ld_shared_volatile(&s_used) < cb - 1; ++it) {  // block cb - 2 still in use
                    if (ld_shared_volatile(&s_fail)) return;
                    if (it > kSpinLimit || clock64() - t0 > 8 * kWaitNs) {
                        if (lane == 0) {
                            atomicCAS(args.err, kDevOk, kDevTimeout);
                            *reinterpret_cast<volatile int *>(&s_fail) = 1;
                        }
                        return;
                    }
                    __nanosleep(64);
                }
                __syncwarp();
                if (!fetch_top<T, LAYOUT, CT, NB>(V, top0, col0, cb, follow, from, args.tag, progress + p - 1,
                                                  Rbuf + (cb & 1) * kIB * (kIB + 4), &s_rows, &s_fail, args.err))
                    return;
            }
            return;
        }
    }

    // my column of the block and my rows of it (reflector warps)
    const bool refl = wid < NWR;
    const int jc = lane & (kIB - 1), half = lane >> 4;
    const int rb = wid * 32 + half * RPL;
    CT col[RPL];
    int big = 0;  // the largest column so far
    if (refl) load_col<T, LAYOUT, CT, RPL>(V, row0 + rb, col0 + jc, col);
    if constexpr (RESC > 0 && NB > 1) {  // the trailing columns, kept until the role is done
        constexpr int U = 16;
        constexpr int NC = RESC, TOT = NC * B;
        for (int base = tid; base < TOT; base += NT * U) {
            T v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int idx = base + u * NT;
                const int tt = LAYOUT == 0 ? idx % B : idx / NC;
                const int j = LAYOUT == 0 ? idx / B : idx % NC;
                v[u] = idx < TOT ? __ldcg(&V(row0 + tt, col0 + S0 + j)) : T(0);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int idx = base + u * NT;
                const int tt = LAYOUT == 0 ? idx % B : idx / NC;
                const int j = LAYOUT == 0 ? idx / B : idx % NC;
                if (idx < TOT) Cs[(size_t)j * CLD + tt] = CT(v[u]);
            }
        }
    }

    for (int cb = 0; cb < NB; ++cb) {
        const int c0 = cb * kIB;
        const int jbase = c0 + kIB;
        const int nrest = B - jbase;
        const int ns = Cfg::nstream(nrest), nr = nrest - ns;  // columns jbase.. streamed, the last nr resident
        const int wr = Cfg::warps_r(nrest);
        const int KR = Cfg::ks(nr, wr), KST = Cfg::ks(ns, NW - wr);
        CT *ZpS = Zp + (size_t)kIB * KR * nr;  // the streamed part's partial Z

        if (refl) {
            const CT *Rts = Rbuf + (cb & 1) * kIB * (kIB + 4);  // this block's top rows (TSQRT)
            if constexpr (Cfg::FETCH == kFetchNone) {  // read by the reflector warps themselves
                if (!geqrt) {
                    if (wid == 0) fetch_top<T, LAYOUT, CT, NB>(V, top0, col0, cb, follow, nullptr, args.tag, progress + p - 1,
                                                     Rbuf + (cb & 1) * kIB * (kIB + 4), &s_rows, &s_fail, args.err);
                    bar_named(1, NWR * 32);
                }
            }
            // ---- the 16 reflectors of the block, one per step: a loop, not unrolled
            // (a step is some 200 instructions, and straight-line code that a single
            // warp runs once per block is bound by instruction fetch).  GEQRT: rows at
            // or above the pivot row do not take part (zeros in the broadcast column);
            // the pivot row is row i % RPL of the lanes of its segment.
            CT myinv = CT(0), mytau = CT(0);
            bool bad = false;  // a reflector that its type cannot hold
            // the largest column of this block up to the i-th (within a factor of two) and of
            // the blocks before it
            auto largest = [&](int i) {
                const int m = mag_bits(myinv);
                return max(big, __reduce_max_sync(0xffffffffu, jc < i && m > 0 ? 2 * mag_bits(CT(1)) - m : 0));
            };
            auto put_x = [&](int i) {  // column i's live rows for every lane of the warp
                if (jc == i) {
                    CT *dst = xs + ((i & 1) * NWR + wid) * 32 + half * RPL;
                    if (!geqrt) {
#pragma unroll
                        for (int r = 0; r < RPL; r += CV) PVec<CT>::st(dst + r, col + r);
                    } else {
#pragma unroll
                        for (int r = 0; r < RPL; ++r) dst[r] = (rb + r > c0 + i) ? col[r] : CT(0);
                    }
                }
            };
            put_x(0);
            __syncwarp();
            const int nstep = (geqrt && cb == NB - 1) ? kIB - 1 : kIB;  // the last column has no reflector
            T *ptop = &V(top0 + c0, col0 + c0 + jc);
            const int64_t dtop = LAYOUT == 0 ? 1 : args.lda;
            const bool out_top = tid < kIB && (!geqrt || (mail && !last));
            const bool post = mail && !last;  // the new top row: to the next role, from the last one to the matrix
            unsigned long long *pbox = box + ((size_t)cb * kIB * kIB + jc) * MW;
            int avail = geqrt ? kIB * NB : 0;
#pragma unroll 1
            for (int i = 0; i < nstep; ++i) {
                const int pb = i & 1;
                const bool own = geqrt && rb == c0 + i - i % RPL;
                const CT *xw = xs + (pb * NWR + wid) * 32;
                CT xr[RPL];
#pragma unroll
                for (int r = 0; r < RPL; r += CV) PVec<CT>::ld(xw + half * RPL + r, xr + r);
                Sq sq = Ar::sq(xw[lane & (2 * RPL - 1)]);
                if (geqrt) {
                    CT piv = col[0];
#pragma unroll
                    for (int r = 1; r < RPL; ++r) piv = (i % RPL == r) ? col[r] : piv;
                    if (own) rowb[pb * kIB + jc] = piv;
                }
#pragma unroll
                for (int o = RPL; o > 0; o >>= 1) sq = Ar::merge_xor(sq, o);
                CT d;
                {
                    constexpr int NA = Cfg::F4 ? 4 : 2;
                    Mac a[NA];
#pragma unroll
                    for (int u = 0; u < NA; ++u) a[u] = Ar::mac0();
#pragma unroll
                    for (int r = 0; r < RPL; ++r) Ar::mac(a[r % NA], xr[r], col[r]);
#pragma unroll
                    for (int h2 = NA / 2; h2 >= 1; h2 >>= 1)
#pragma unroll
                        for (int u = 0; u < h2; ++u) a[u] = Ar::mac_merge(a[u], a[u + h2]);
                    d = Ar::fin(a[0]);
                    d = d + vshfl_xor(d, 16);
                }
                if (NWR > 1) {
                    if (lane < kIB) part[(pb * kIB + lane) * NWR + wid] = d;
                    if (lane == 0) spart[pb * NWR + wid] = sq;
                    bar_named(1, NWR * 32);
                    Sq sw[NWR];
                    CT dw[NWR];
#pragma unroll
                    for (int w = 0; w < NWR; w += 2) PSq2<Sq>::ld(spart + pb * NWR + w, sw[w], sw[w + 1]);
                    if constexpr (NWR >= CV) {
#pragma unroll
                        for (int w = 0; w < NWR; w += CV) PVec<CT>::ld(part + (pb * kIB + jc) * NWR + w, dw + w);
                    } else {
#pragma unroll
                        for (int w = 0; w < NWR; ++w) dw[w] = part[(pb * kIB + jc) * NWR + w];
                    }
#pragma unroll
                    for (int h2 = NWR / 2; h2 >= 1; h2 >>= 1)
#pragma unroll
                        for (int w = 0; w < h2; ++w) {
                            sw[w] = Ar::merge(sw[w], sw[w + h2]);
                            dw[w] = dw[w] + dw[w + h2];
                        }
                    sq = sw[0];
                    d = dw[0];
                } else {
                    __syncwarp();
                }
                if (avail <= cb * kIB + i) avail = wait_rows(&s_rows, cb * kIB + i + 1, &s_fail, args.err);
                const CT *prow = geqrt ? rowb + pb * kIB : Rts + i * (kIB + 4);
                const CT rj = prow[jc];
                PRefl<CT> r = Ar::scalars(sq, prow[i]);
                if (Ar::small(sq, prow[i])) {  // known well before the scalars
                    bool zero = Ar::vanished(sq, prow[i]);
                    if (Ar::kFp64 ? (zero ? prow[i] != CT(0) : !vfinite(r.f)) : !zero) {
                        // A column too small for its type (FP64: its squares vanish, or tau /
                        // nu^2 overflows), or NaN.  One that is nothing against the columns before
                        // it counts as zero: what cancellation leaves of dependent columns,
                        // each some 1e-8 (1e-16) of the one before
                        int m = largest(i);
                        if (args.ref) {
                            const T *ref = reinterpret_cast<const T *>(args.ref) + zb * args.sRef;
                            for (int q = lane; q < B; q += 32) m = max(m, mag_bits(CT(__ldcg(ref + q * args.ref_ld))));
                            m = __reduce_max_sync(0xffffffffu, m);
                        }
                        const bool drop = negligible<CT>(mag_bits(zero ? prow[i] : r.nu), m);
                        bad = bad || (!drop && (zero || i < kIB - 1 || !Ar::kFp64));  // (FP64's last column needs no f)
                        zero = zero || drop;
                    }
                    if (zero) {  // identity reflector
                        r.nu = r.tau = r.tc = r.f = r.inv = CT(0);
                        r.beta = prow[i];
                    }
                }
                bad = bad || !vfinite(r.tau) || !vfinite(r.nu);
                const CT h = r.nu * rj + d;
                const CT w = jc > i ? r.f * h : CT(0);  // columns up to i are finished
#pragma unroll
                for (int q = 0; q < RPL; ++q) col[q] = col[q] - xr[q] * w;
                const CT top = jc > i ? rj - r.tc * h : r.beta;  // the pivot row's new value
                if (geqrt) {
#pragma unroll
                    for (int q = 0; q < RPL; ++q) col[q] = (own && jc >= i && i % RPL == q) ? top : col[q];
                }
                if (i < kIB - 1) put_x(i + 1);
                if (out_top && jc >= i) {
                    if (post) mail_put(pbox + i * kIB * MW, top, args.tag);
                    else ptop[i * dtop] = (T)top;
                }
                mytau = jc == i ? r.tau : mytau;
                myinv = jc == i ? r.inv : myinv;
                __syncwarp();
            }
            big = largest(kIB);
            if (bad && lane == 0) atomicCAS(args.err, kDevOk, kDevNonfinite);
            if (tid < kIB) stau[tid] = mytau;
            __syncwarp();
            // without the mailbox the diagonal block is handed on whole, here; the last
            // row of the last block has no reflector
            if (!geqrt && !mail && tid == 0) st_release(progress + p, cb + 1);
            if (geqrt && post && cb == NB - 1 && jc == kIB - 1 && rb + RPL == B)
                mail_put(pbox + (kIB - 1) * kIB * MW, col[RPL - 1], args.tag);
            // ---- V (each column scaled by its 1 / nu) back to the tile, and the
            // masked Y (unit lower for GEQRT)
#pragma unroll
            for (int r = 0; r < RPL; ++r)
                if (!geqrt || rb + r > c0 + jc) col[r] = col[r] * myinv;
            if (geqrt && post && rb >= c0 && rb < c0 + kIB) {  // the rows above the diagonal are the last role's to write
#pragma unroll
                for (int r = 0; r < RPL; ++r)
                    if (rb + r > c0 + jc) V(row0 + rb + r, col0 + c0 + jc) = (T)col[r];
            } else if (!geqrt || rb >= c0) {
                store_col<T, LAYOUT, CT, RPL>(V, row0 + rb, col0 + c0 + jc, col);
            }
#pragma unroll
            for (int r = 0; r < RPL; ++r) {
                CT y = col[r];
                if (geqrt) y = (rb + r == c0 + jc) ? CT(1) : (rb + r > c0 + jc ? y : CT(0));
                Yr[(size_t)(rb + r) * YLD + jc] = y;
            }
        }
        if constexpr (Cfg::FETCH == kFetchIdle) {
            if (wid == NWR && !geqrt)
                fetch_top<T, LAYOUT, CT, NB>(V, top0, col0, cb, follow, from, args.tag, progress + p - 1,
                                             Rbuf + (cb & 1) * kIB * (kIB + 4), &s_rows, &s_fail, args.err);
        }
        if (tid == 0) s_ok = !ld_shared_volatile(&s_fail);
        bar_named(2, NT);
        if (!s_ok) return;
        if (tid == 0) *reinterpret_cast<volatile int *>(&s_used) = cb + 1;
        // without the mailbox: the block's rows of the top tile are written back above
        // (the release covers what the barrier ordered before it)
        if (geqrt && !mail && tid == 0) st_release(progress, cb + 1);
        if (tid < kIB) tau_out[c0 + tid] = (T)stau[tid];

        // ---- Gram matrix of the block's reflectors
        if constexpr (Cfg::F4) {
            // 4 x 4 blocks, two row halves per warp, a range of rows per warp
            constexpr int RW = B / NW;
            const int lb = (lane >> 2) & 3, ib = lane & 3;
            CT g[4][4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int v = 0; v < 4; ++v) g[u][v] = CT(0);
#pragma unroll 4
            for (int r = half; r < RW; r += 2) {
                const CT *yr = Yr + (size_t)(wid * RW + r) * YLD;
                CT a[4], e[4];
                PVec<CT>::ld(yr + 4 * lb, a);
                PVec<CT>::ld(yr + 4 * ib, e);
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int v = 0; v < 4; ++v) g[u][v] += a[u] * e[v];
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
#pragma unroll
                for (int v = 0; v < 4; ++v) g[u][v] += vshfl_xor(g[u][v], 16);
                if (half == 0) PVec<CT>::st(Gp + wid * kIB * kIB + (4 * lb + u) * kIB + 4 * ib, g[u]);
            }
        } else {
            // one pair l < m per thread (two threads per pair from 256 threads on)
            constexpr int HS = NT >= 256 ? 2 : 1;
            constexpr int NP = kIB * (kIB - 1) / 2;
            for (int idx = tid; idx < (NP * HS + 31) / 32 * 32; idx += NT) {
                const int pi = idx / HS, h = idx % HS;
                int l = 0, m = 0;
                if (pi < NP) {
                    m = 1;
                    while (m * (m + 1) / 2 <= pi) ++m;
                    l = pi - m * (m - 1) / 2;
                }
                Mac acc = Ar::mac0();
                if (pi < NP) {
                    constexpr int RH = B / HS;
                    const CT *yr = Yr + (size_t)h * RH * YLD;
#pragma unroll 4
                    for (int r = 0; r < RH; ++r) Ar::mac(acc, yr[r * YLD + l], yr[r * YLD + m]);
                }
                CT v = Ar::fin(acc);
                if (HS == 2) v = v + vshfl_xor(v, 1);
                if (pi < NP && h == 0) G[l * kIB + m] = v;
            }
        }

        // ---- Z = Y^T C over the trailing columns of the tile: thread = columns
        // jA, jA + 32 of its warp's 64, rows of its range
        if constexpr (NB > 1) {
            if (nrest > 0) {
                const bool res = wid < wr;
                const int nc = res ? nr : ns, K = res ? KR : KST, w0 = res ? wid : wid - wr;
                const int wcol = Cfg::wcol(nc);
                const int wc = wcol > 0 ? w0 % wcol : 0, kseg = wcol > 0 ? w0 / wcol : 0;
                const int jA = wc * 64 + lane, jB = jA + 32;
                const bool onA = kseg < K && jA < nc, onB = kseg < K && jB < nc;
                const int RK = B / K;
                CT *zp = (res ? Zp : ZpS) + (size_t)kseg * kIB * nc;
                Mac z0[kIB], z1[kIB];
#pragma unroll
                for (int l = 0; l < kIB; ++l) z0[l] = z1[l] = Ar::mac0();
                auto row_mac = [&](int r, CT va, CT vb) {
                    CT y[kIB];
                    ld16<CT>(Yr + (size_t)r * YLD, y);
#pragma unroll
                    for (int l = 0; l < kIB; ++l) {
                        Ar::mac(z0[l], y[l], va);
                        Ar::mac(z1[l], y[l], vb);
                    }
                };
                if (onA) {
                    if (RESC > 0 && res) {
                        const CT *pA = Cs + (size_t)(B - nr - S0 + jA) * CLD;
                        const CT *pB = onB ? pA + (size_t)32 * CLD : pA;
#pragma unroll 1
                        for (int r = kseg * RK; r < (kseg + 1) * RK; r += CV) {
                            CT cA[CV], cB[CV];
                            PVec<CT>::ld(pA + r, cA);
                            PVec<CT>::ld(pB + r, cB);
#pragma unroll
                            for (int u = 0; u < CV; ++u) row_mac(r + u, cA[u], cB[u]);
                        }
                    } else if (Cfg::STREAM) {
                        // streamed columns: from L2, the next SU rows in flight
                        constexpr int SU = Cfg::F4 ? 8 : 4;
                        const int64_t cA0 = col0 + jbase + jA, cB0 = onB ? cA0 + 32 : cA0;
                        T bA[SU], bB[SU], nA[SU], nB[SU];
                        auto fetch = [&](int r, T (&a)[SU], T (&b)[SU]) {
                            if (LAYOUT == 0) {
#pragma unroll
                                for (int u = 0; u < SU; u += TV) {
                                    PVec<T>::ldcg(&V(row0 + r + u, cA0), a + u);
                                    PVec<T>::ldcg(&V(row0 + r + u, cB0), b + u);
                                }
                            } else {
#pragma unroll
                                for (int u = 0; u < SU; ++u) {
                                    a[u] = __ldcg(&V(row0 + r + u, cA0));
                                    b[u] = __ldcg(&V(row0 + r + u, cB0));
                                }
                            }
                        };
                        const int rend = (kseg + 1) * RK;
                        fetch(kseg * RK, bA, bB);
#pragma unroll 1
                        for (int r = kseg * RK; r < rend; r += SU) {
                            if (r + SU < rend) fetch(r + SU, nA, nB);
#pragma unroll
                            for (int u = 0; u < SU; ++u) row_mac(r + u, CT(bA[u]), CT(bB[u]));
#pragma unroll
                            for (int u = 0; u < SU; ++u) {
                                bA[u] = nA[u];
                                bB[u] = nB[u];
                            }
                        }
                    }
                }
#pragma unroll
                for (int l = 0; l < kIB; ++l) {
                    if (onA) zp[(size_t)l * nc + jA] = Ar::fin(z0[l]);
                    if (onB) zp[(size_t)l * nc + jB] = Ar::fin(z1[l]);
                }
            }
        }
        CT nx[RPL];  // the next block's columns, loaded ahead of their update
        if constexpr (NB > 1) {
            if (nrest > 0 && refl) {
                if (Cfg::STREAM && ns > 0) {
                    load_col<T, LAYOUT, CT, RPL>(V, row0 + rb, col0 + jbase + jc, nx);
                } else if (RESC > 0) {
#pragma unroll
                    for (int r = 0; r < RPL; r += CV)
                        PVec<CT>::ld(Cs + (size_t)(jbase - S0 + jc) * CLD + rb + r, nx + r);
                }
            }
        }
        bar_named(2, NT);
        if constexpr (Cfg::F4) {
            for (int idx = tid; idx < kIB * kIB; idx += NT) {
                CT v = Gp[idx];
#pragma unroll
                for (int w = 1; w < NW; ++w) v += Gp[w * kIB * kIB + idx];
                G[idx] = v;
            }
        }
        // the trailing top rows, once the previous role's are in them
        if (tid == 0) {
            s_ok = (follow && nrest > 0) ? wait_geq(full + p - 1, cb + 1, args.err) : true;
            if (!s_ok) *reinterpret_cast<volatile int *>(&s_fail) = 1;  // for the fetch warp
        }
        bar_named(2, NT);
        if (!s_ok) return;

        // ---- W = T^T (Z + top rows) by forward substitution; top rows -= W.  The 16
        // unit right-hand sides after the columns give the rows of T.
        for (int j = tid; j < nrest + kIB; j += NT) {
            CT z[kIB], top[kIB];
            Mac zz[kIB];
            const bool unit = j >= nrest;
            if (unit) {
#pragma unroll
                for (int l = 0; l < kIB; ++l) zz[l] = Ar::mac_from(CT(j - nrest == l ? 1 : 0));
            } else {
                if (!geqrt) load_col<T, LAYOUT, CT, kIB>(V, top0 + c0, col0 + jbase + j, top);
                const bool str = j < ns;
                const CT *zp = str ? ZpS + j : Zp + (j - ns);
                const int nc = str ? ns : nr, K = str ? KST : KR;
#pragma unroll
                for (int l = 0; l < kIB; ++l) z[l] = zp[(size_t)l * nc];
                for (int k = 1; k < K; ++k) {
#pragma unroll
                    for (int l = 0; l < kIB; ++l) z[l] = z[l] + zp[(size_t)(k * kIB + l) * nc];
                }
                if (!geqrt) {
#pragma unroll
                    for (int l = 0; l < kIB; ++l) z[l] = z[l] + top[l];
                }
#pragma unroll
                for (int l = 0; l < kIB; ++l) zz[l] = Ar::mac_from(z[l]);
            }
#pragma unroll
            for (int l = 0; l < kIB; ++l) {
                z[l] = stau[l] * Ar::fin(zz[l]);
                const CT nz = -z[l];
#pragma unroll
                for (int m = l + 1; m < kIB; ++m) Ar::mac(zz[m], G[l * kIB + m], nz);
            }
            if (unit) {
#pragma unroll
                for (int k = 0; k < kIB; ++k) tblk_out[(size_t)cb * kIB * kIB + (j - nrest) + k * kIB] = (T)z[k];
            } else if constexpr (NB > 1) {
                st16<CT>(Ws + (size_t)j * YLD, z);
                if (!geqrt) {
#pragma unroll
                    for (int l = 0; l < kIB; ++l) top[l] = top[l] - z[l];
                    store_col<T, LAYOUT, CT, kIB>(V, top0 + c0, col0 + jbase + j, top);
                }
            }
        }
        bar_named(2, NT);
        if constexpr (NB > 1) {
            // a TSQRT role hands the trailing top rows on before updating its own tile
            if (!geqrt && tid == 0) st_release(full + p, cb + 1);
            if (nrest > 0) {
                // ---- C -= Y W: the next block's 16 columns first, into registers
                if (refl) {
                    if constexpr (!std::is_same<CT, dfx>::value) {
                        CT w[kIB];
                        ld16<CT>(Ws + (size_t)jc * YLD, w);
#pragma unroll
                        for (int r = 0; r < RPL; ++r) {
                            CT y[kIB];
                            ld16<CT>(Yr + (size_t)(rb + r) * YLD, y);
                            Mac acc = Ar::mac0();
#pragma unroll
                            for (int l = 0; l < kIB; ++l) Ar::mac(acc, y[l], w[l]);
                            col[r] = nx[r] - Ar::fin(acc);
                        }
                    } else {  // reflectors in a loop: unrolled, its code is bound by instruction fetch
                        Mac acc[RPL];
#pragma unroll
                        for (int r = 0; r < RPL; ++r) acc[r] = Ar::mac0();
#pragma unroll 1
                        for (int l = 0; l < kIB; ++l) {
                            const CT wl = Ws[(size_t)jc * YLD + l];
#pragma unroll
                            for (int r = 0; r < RPL; ++r) Ar::mac(acc[r], Yr[(size_t)(rb + r) * YLD + l], wl);
                        }
#pragma unroll
                        for (int r = 0; r < RPL; ++r) col[r] = nx[r] - Ar::fin(acc[r]);
                    }
                    // GEQRT: rows c0 .. c0+15 of these columns are final
                    if (geqrt && rb == c0) store_col<T, LAYOUT, CT, RPL>(V, row0 + rb, col0 + jbase + jc, col);
                }
                // ---- the other columns, two rows per thread
                if (nrest > kIB) {
                    constexpr int RS = B >= 64 ? B / 2 : B;
                    constexpr int CG = NT / RS > 0 ? NT / RS : 1;
                    const int slot = tid % RS, grp = tid / RS;
                    CT ya[kIB], yb[kIB];
                    ld16<CT>(Yr + (size_t)slot * YLD, ya);
                    ld16<CT>(Yr + (size_t)(slot + B / 2) * YLD, yb);
                    auto apply = [&](int j, CT &a, CT &b) {
                        CT w[kIB];
                        ld16<CT>(Ws + (size_t)j * YLD, w);
                        Mac a0 = Ar::mac0(), a1 = Ar::mac0();
#pragma unroll
                        for (int l = 0; l < kIB; ++l) {
                            Ar::mac(a0, ya[l], w[l]);
                            Ar::mac(a1, yb[l], w[l]);
                        }
                        a = a - Ar::fin(a0);
                        b = b - Ar::fin(a1);
                    };
                    // GEQRT: only rows from c0 on belong to this role
                    const bool wa = !geqrt || slot >= c0, wb = !geqrt || slot + B / 2 >= c0;
                    if (Cfg::STREAM && ns > kIB) {  // streamed columns, NQ per turn, the next ones in flight
                        constexpr int NQ = 4;
                        T ga[NQ], gb[NQ], ha[NQ], hb[NQ];
                        auto fetch = [&](int j, T (&a)[NQ], T (&b)[NQ]) {
                            const int64_t c = col0 + jbase + j;
                            if (LAYOUT == 0) {
#pragma unroll
                                for (int e = 0; e < NQ; ++e) {
                                    a[e] = __ldcg(&V(row0 + slot, c + e));
                                    b[e] = __ldcg(&V(row0 + slot + B / 2, c + e));
                                }
                            } else {
#pragma unroll
                                for (int e = 0; e < NQ; e += TV) {
                                    PVec<T>::ldcg(&V(row0 + slot, c + e), a + e);
                                    PVec<T>::ldcg(&V(row0 + slot + B / 2, c + e), b + e);
                                }
                            }
                        };
                        const int jbeg = kIB + grp * NQ;  // 16 columns at least, a multiple of 16
                        if (jbeg < ns) fetch(jbeg, ga, gb);
#pragma unroll 1
                        for (int j = jbeg; j < ns; j += CG * NQ) {
                            if (j + CG * NQ < ns) fetch(j + CG * NQ, ha, hb);
#pragma unroll
                            for (int e = 0; e < NQ; ++e) {
                                CT a = CT(ga[e]), b = CT(gb[e]);
                                apply(j + e, a, b);
                                ga[e] = (T)a;
                                gb[e] = (T)b;
                            }
                            const int64_t c = col0 + jbase + j;
                            if (LAYOUT == 0) {
#pragma unroll
                                for (int e = 0; e < NQ; ++e) {
                                    if (wa) V(row0 + slot, c + e) = ga[e];
                                    if (wb) V(row0 + slot + B / 2, c + e) = gb[e];
                                }
                            } else {
#pragma unroll
                                for (int e = 0; e < NQ; e += TV) {
                                    if (wa) PVec<T>::st(&V(row0 + slot, c + e), ga + e);
                                    if (wb) PVec<T>::st(&V(row0 + slot + B / 2, c + e), gb + e);
                                }
                            }
#pragma unroll
                            for (int e = 0; e < NQ; ++e) {
                                ga[e] = ha[e];
                                gb[e] = hb[e];
                            }
                        }
                    }
                    if constexpr (RESC > 0) {
                        // GEQRT: rows c0 .. c0+15 of the columns are final and go out
                        const bool oa = geqrt && slot >= c0 && slot < jbase;
                        const bool ob = geqrt && slot + B / 2 >= c0 && slot + B / 2 < jbase;
#pragma unroll 2
                        for (int j = (ns > kIB ? ns : kIB) + grp; j < nrest; j += CG) {
                            CT *pc = Cs + (size_t)(jbase - S0 + j) * CLD + slot;
                            CT a = pc[0], b = pc[B / 2];
                            apply(j, a, b);
                            pc[0] = a;
                            pc[B / 2] = b;
                            if (oa) V(row0 + slot, col0 + jbase + j) = (T)a;
                            if (ob) V(row0 + slot + B / 2, col0 + jbase + j) = (T)b;
                        }
                    }
                }
            }
            bar_named(2, NT);
        }
        if (geqrt && tid == 0) st_release(full, cb + 1);
    }
}

// ---------------------------------------------------------------------------
// Trailing update of tiles 32 and 64 and of FP64 tiles of 16, 16 reflectors at a time
// (FP32 tiles of 16: update16_kernel; tiles 128 and 256: the full-T update).
//
// A CTA takes a column strip and `group` consecutive tiles; a thread owns 16 rows
// of one column of the current tile, in registers from its load to its store.
// Per block of 16 reflectors: Z = V^T A over the thread's rows, the row segments
// joined through shared memory, W = T^T (Z + top rows) (FP32: by every segment's
// thread, so W needs no second exchange; FP64: by the first segment's), top rows
// -= W, A -= V W.  The top rows of the strip stay in shared memory while the CTA
// works through its group and pass from group to group block by block: the next
// group needs a block's top rows only when it forms that block's W, so the chain
// through the tiles is one load, one 16 x 16 product and one store per tile and
// block (a counter per block: one for the whole strip would not grow
// monotonically).
// V and T of the next blocks are staged ahead (three buffers: one barrier per
// block).  (tile group, strip) pairs come from a ticket in group-major order, so a
// CTA only waits on one that already runs.
//
// What bounds it: the chain of W through the tiles (about 1.5 us a tile), the FP32
// pipe in large batches, the FP64 unit for FP64.  Measured (GB300, all of a call's
// updates, before: one CTA per strip looping over the tiles, every product from
// shared memory with three barriers a block): FP32 n = 1024 tile 64 11.3 -> 1.35
// ms, n = 1296 tile 16 39 -> 11 ms; FP64 n = 1024 tile 64 22.5 -> 7.2 ms.
template <typename T, int B>
struct UpdCfg {
    static constexpr int NB = B / kIB;             // blocks per tile = row segments
    static constexpr bool F4 = sizeof(T) == 4;
    static constexpr int W = F4 ? 64 : 32;         // columns of a strip
    static constexpr int NT = W * NB;
    static constexpr int LDV = F4 ? 20 : 18;       // row stride of V (16-byte rows)
    static constexpr int VSZ = B * LDV + kIB * kIB;  // one staged block: V, then T (row l: T(0..15, l))
    static constexpr int PER = (B * kIB + NT - 1) / NT;
    static constexpr int MINB = F4 ? (B == 64 ? 2 : 3) : 1;  // CTAs per SM the registers allow
    static constexpr size_t smem_bytes() {
        return sizeof(T) * (3 * (size_t)VSZ + (size_t)B * W + (NB > 1 ? 2 * (size_t)NB * kIB * W + kIB * W : 0));
    }
};

template <typename T, int LAYOUT, int B>
__global__ void __launch_bounds__(UpdCfg<T, B>::NT, UpdCfg<T, B>::MINB) update_kernel(UpdateArgs args) {
    using C = UpdCfg<T, B>;
    constexpr int NB = C::NB, W = C::W, NT = C::NT, LDV = C::LDV, PER = C::PER;
    constexpr int VN = PVec<T>::VN;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *Vs = reinterpret_cast<T *>(smem_raw);  // [3][VSZ]
    T *Top = Vs + 3 * C::VSZ;                 // [B][W]
    T *Zp = Top + B * W;                      // [2][NB][16][W]
    T *Wx = Zp + 2 * NB * kIB * W;            // [16][W] (FP64)
    __shared__ int s_t, s_ok;
    const int tid = threadIdx.x;
    const int64_t zb = blockIdx.y;
    int *flags = args.flags + zb * args.sFlags;
    if (tid == 0) {
        s_t = atomicAdd(flags, 1);
        s_ok = 1;
    }
    __syncthreads();
    const int grp = s_t / args.nstrip, strip = s_t % args.nstrip;
    const int p0 = args.first_role + grp * args.group;
    if (p0 >= args.P) return;
    const int p1 = min(args.P, p0 + args.group);
    int *done = flags + 1 + strip * (args.fine ? NB : 1);
    const int64_t j0 = (int64_t)(args.pc + 1) * B + (int64_t)strip * W;
    const int col = tid % W, seg = tid / W;
    const bool live = j0 + col < args.n;
    View<T, LAYOUT> V{reinterpret_cast<T *>(args.a) + zb * args.sA, args.lda};
    const int64_t top0 = (int64_t)args.pr * B, col0 = (int64_t)args.pc * B;
    const int64_t jc = live ? j0 + col : j0;  // dead columns repeat the first one and store nothing
    const T *tblk = reinterpret_cast<const T *>(args.tblk) + zb * args.sTblk;
    const int nblk = (p1 - p0) * NB;

    // staging of block u of the group (tile p0 + u / NB, block u % NB): V masked to
    // unit lower for the top tile, and T
    T sv[PER];
    T st[kIB * kIB / NT > 0 ? kIB * kIB / NT : 1];
    auto fetch = [&](int u) {
        const int p = p0 + u / NB, c0 = (u % NB) * kIB;
        const int64_t r0 = (int64_t)(args.pr + p) * B;
#pragma unroll
        for (int e = 0; e < PER; ++e) {
            const int idx = tid + e * NT;
            const int r = LAYOUT == 0 ? idx % B : idx / kIB, l = LAYOUT == 0 ? idx / B : idx % kIB;
            T v = __ldcg(&V(r0 + r, col0 + c0 + l));
            if (p == 0) v = r == c0 + l ? T(1) : (r > c0 + l ? v : T(0));
            sv[e] = v;
        }
#pragma unroll
        for (int e = 0; e < (int)(sizeof(st) / sizeof(T)); ++e) {
            const int idx = tid + e * NT;
            if (idx < kIB * kIB) st[e] = __ldcg(tblk + ((size_t)p * NB + u % NB) * kIB * kIB + idx);
        }
    };
    auto stage = [&](int u) {
        T *buf = Vs + (u % 3) * C::VSZ;
#pragma unroll
        for (int e = 0; e < PER; ++e) {
            const int idx = tid + e * NT;
            const int r = LAYOUT == 0 ? idx % B : idx / kIB, l = LAYOUT == 0 ? idx / B : idx % kIB;
            buf[r * LDV + l] = sv[e];
        }
#pragma unroll
        for (int e = 0; e < (int)(sizeof(st) / sizeof(T)); ++e) {
            const int idx = tid + e * NT;
            if (idx < kIB * kIB) buf[B * LDV + idx] = st[e];
        }
    };
    static_assert(B * kIB % NT == 0, "staging split");

    T a[kIB], an[kIB];
    auto load_tile = [&](int p, T (&v)[kIB]) {
        load_col<T, LAYOUT, T, kIB>(V, (int64_t)(args.pr + p) * B + seg * kIB, jc, v);
    };
    load_tile(p0, a);
    fetch(0);
    stage(0);
    if (nblk > 1) {
        fetch(1);
        stage(1);
    }
    if (nblk > 2) fetch(2);
    __syncthreads();
    T pend[kIB];       // new top rows, stored once every thread has read the old ones
    int pend_row = -1;
    for (int u = 0; u < nblk; ++u) {
        const int p = p0 + u / NB, cb = u % NB, c0 = cb * kIB;
        const bool head = p == 0;                    // the top tile itself (GEQRT)
        const bool in_global = !head && p == p0;     // the top rows come from the previous group
        const T *vb = Vs + (u % 3) * C::VSZ, *tb = vb + B * LDV;
        if (cb == 0 && p + 1 < p1) load_tile(p + 1, an);
        // Z over my rows
        T z[kIB];
#pragma unroll
        for (int l = 0; l < kIB; ++l) z[l] = T(0);
#pragma unroll
        for (int r = 0; r < kIB; ++r) {
            T y[kIB];
            ld16<T>(vb + (seg * kIB + r) * LDV, y);
#pragma unroll
            for (int l = 0; l < kIB; ++l) z[l] += y[l] * a[r];
        }
        if (NB > 1) {
            T *zp = Zp + ((u & 1) * NB + seg) * kIB * W + col;
#pragma unroll
            for (int l = 0; l < kIB; ++l) zp[l * W] = z[l];
        }
        if (tid == 0 && in_global && p > args.first_role && (args.fine || cb == 0))
            s_ok = wait_geq(done + (args.fine ? cb : 0), p - args.first_role, args.err);
        __syncthreads();
        if (!s_ok) return;
        if (pend_row >= 0) {
#pragma unroll
            for (int l = 0; l < kIB; ++l) Top[(pend_row + l) * W + col] = pend[l];
            pend_row = -1;
        }
        if (u + 2 < nblk) {
            stage(u + 2);
            if (u + 3 < nblk) fetch(u + 3);
        }
        // another group follows: each block's counter only grows tile by tile
        const bool release = p + 1 == p1 && p + 1 < args.P && (args.fine || cb == NB - 1);
        // W = T^T (Z + top rows); top rows -= W
        T w[kIB];
        if (C::F4 || seg == 0) {
            T top[kIB];
            if (!head) {
                if (in_global) {
                    load_col<T, LAYOUT, T, kIB>(V, top0 + c0, jc, top);
                } else {
#pragma unroll
                    for (int l = 0; l < kIB; ++l) top[l] = Top[(c0 + l) * W + col];
                }
            }
            if (NB > 1) {
#pragma unroll
                for (int l = 0; l < kIB; ++l) {
                    const T *zp = Zp + (u & 1) * NB * kIB * W + l * W + col;
                    z[l] = zp[0];
#pragma unroll
                    for (int q = 1; q < NB; ++q) z[l] += zp[q * kIB * W];
                }
            }
            if (!head) {
#pragma unroll
                for (int l = 0; l < kIB; ++l) z[l] += top[l];
                // every segment has read the rows that the first one overwrites below
                if (C::F4 && NB > 1 && in_global && p + 1 == p1) __syncthreads();
            }
#pragma unroll
            for (int l = 0; l < kIB; ++l) {  // T(m, l) at tb[m + 16 l]
                T tl[kIB];
#pragma unroll
                for (int q = 0; q <= l; q += VN) PVec<T>::ld(tb + l * kIB + q, tl + q);
                T acc = T(0);
#pragma unroll
                for (int m = 0; m <= l; ++m) acc += tl[m] * z[m];
                w[l] = acc;
            }
            if (!head) {
                // out: the last tile of the group hands the rows on (and the last tile
                // of the panel leaves them final)
                if (seg == 0) {
#pragma unroll
                    for (int l = 0; l < kIB; ++l) pend[l] = top[l] - w[l];
                    if (p + 1 == p1) {
                        if (live) store_col<T, LAYOUT, T, kIB>(V, top0 + c0, jc, pend);
                        if (release) {
                            bar_named(1, W);
                            if (col == 0) st_release(done + (args.fine ? cb : 0), p - args.first_role + 1);
                        }
                    } else {
                        pend_row = c0;
                    }
                }
            }
            if (!C::F4 && NB > 1) {
#pragma unroll
                for (int l = 0; l < kIB; ++l) Wx[l * W + col] = w[l];
            }
        }
        if (!C::F4 && NB > 1) {
            __syncthreads();
            if (seg > 0) {
#pragma unroll
                for (int l = 0; l < kIB; ++l) w[l] = Wx[l * W + col];
            }
        }
        // A -= V W
#pragma unroll
        for (int r = 0; r < kIB; ++r) {
            T y[kIB];
            ld16<T>(vb + (seg * kIB + r) * LDV, y);
            T acc = T(0);
#pragma unroll
            for (int l = 0; l < kIB; ++l) acc += y[l] * w[l];
            a[r] -= acc;
        }
        if (head) {
            // rows c0 .. c0+15 of the top tile are final for this tile
            if (p + 1 == p1) {
                if (seg == cb && live) store_col<T, LAYOUT, T, kIB>(V, top0 + c0, jc, a);
                if (release) {
                    __syncthreads();
                    if (tid == 0) st_release(done + (args.fine ? cb : 0), p - args.first_role + 1);
                }
            } else if (seg == cb) {
#pragma unroll
                for (int l = 0; l < kIB; ++l) Top[(c0 + l) * W + col] = a[l];
            }
        }
        if (cb == NB - 1) {
            if (!head && live)
                store_col<T, LAYOUT, T, kIB>(V, (int64_t)(args.pr + p) * B + seg * kIB, jc, a);
#pragma unroll
            for (int r = 0; r < kIB; ++r) a[r] = an[r];
        }
    }
}

// ---------------------------------------------------------------------------
// Trailing update of FP32 tiles of 16: a CTA takes a strip of 16 columns through all
// tiles, four threads per column, four rows (and four reflectors) each.
//
// What bounds it: the latency of a tile, times the tiles; a 16 x 16 product is too
// little work to pass the strip on for.  With one thread per column a tile was 650
// dependent-ish instructions of one warp (3.1 k cycles); four threads share them (Z by
// a reduce-scatter over the quad, W and Z gathered through shared memory), V, T and the
// strip's tile arrive by asynchronous copies five tiles ahead, and 16 columns a CTA
// give each warp a scheduler to itself.  Measured (GB300, n = 1296, all updates of the
// call): 11.2 -> 5.0 ms.
constexpr int kU16W = 16, kU16T = 4 * kU16W, kU16S = 6;  // columns, threads, stages
__device__ __forceinline__ void copy16_async(float *dst, const float *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
template <int LAYOUT>
__global__ void __launch_bounds__(kU16T) update16_kernel(UpdateArgs args) {
    constexpr int VS = 272, TS = 272, AS = 288, ST = VS + TS + AS;
    __shared__ __align__(16) float sm[kU16S * ST];
    __shared__ __align__(16) float ex[kU16T / 32][8 * 20];  // a quad's 16 values
    const int tid = threadIdx.x, qd = tid & 3, col = tid >> 2;
    const int64_t zb = blockIdx.y;
    View<float, LAYOUT> V{reinterpret_cast<float *>(args.a) + zb * args.sA, args.lda};
    const float *tblk = reinterpret_cast<const float *>(args.tblk) + zb * args.sTblk;
    const int64_t col0 = (int64_t)args.pc * 16, j0 = col0 + 16 + (int64_t)blockIdx.x * kU16W;
    const int64_t top0 = (int64_t)args.pr * 16;
    const int p0 = args.first_role, P = args.P;
    // 16-word rows, every four of them 4 (8) words further: the quad's 16-byte (4-byte) reads spread over the banks
    auto pad4 = [](int r) { return r * 16 + (r / 4) * 4; };
    auto pad8 = [](int r) { return r * 16 + (r / 4) * 8; };
    auto fetch = [&](int p) {
        if (p < P) {
            float *st = sm + (p % kU16S) * ST;
            const int64_t row0 = (int64_t)(args.pr + p) * 16;
            const int i = tid >> 2, q4 = 4 * (tid & 3);
            if (LAYOUT == 0) {  // [reflector][row], [column][row]
                copy16_async(st + i * 16 + q4, &V(row0 + q4, col0 + i));
                copy16_async(st + VS + TS + i * 16 + q4, &V(row0 + q4, j0 + i));
            } else {  // [row][reflector], [row][column]
                copy16_async(st + pad4(i) + q4, &V(row0 + i, col0 + q4));
                copy16_async(st + VS + TS + pad8(i) + q4, &V(row0 + i, j0 + q4));
            }
            copy16_async(st + VS + pad4(i) + q4, tblk + (size_t)p * kIB * kIB + i * 16 + q4);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float *exq = ex[tid >> 5] + ((tid & 31) >> 2) * 20;
    auto gather = [&](const float (&own)[4], float (&all)[16]) {  // the quad's 4 x 4 values
        __syncwarp();
        *reinterpret_cast<float4 *>(exq + 4 * qd) = make_float4(own[0], own[1], own[2], own[3]);
        __syncwarp();
        ld16<float>(exq, all);
    };
    auto load4 = [&](int64_t r0, float (&v)[4]) {
        load_col<float, LAYOUT, float, 4>(V, r0 + 4 * qd, j0 + col, v);
    };
    auto store4 = [&](int64_t r0, const float (&v)[4]) {
        store_col<float, LAYOUT, float, 4>(V, r0 + 4 * qd, j0 + col, v);
    };

    float top[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (p0 > 0) load4(top0, top);
    for (int i = 0; i < kU16S - 1; ++i) fetch(p0 + i);
#pragma unroll 1
    for (int p = p0; p < P; ++p) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kU16S - 2) : "memory");
        __syncthreads();  // tile p is here; the slot of tile p - 1 is free
        fetch(p + kU16S - 1);
        const float *st = sm + (p % kU16S) * ST;
        const bool head = p == 0;  // the top tile itself (GEQRT): unit lower V, W = T^T Z
        float v[4][16], a[4];
        if (LAYOUT == 0) {
#pragma unroll
            for (int l = 0; l < 16; ++l) {
                const float4 x = *reinterpret_cast<const float4 *>(st + l * 16 + 4 * qd);
                v[0][l] = x.x;
                v[1][l] = x.y;
                v[2][l] = x.z;
                v[3][l] = x.w;
            }
            const float4 x = *reinterpret_cast<const float4 *>(st + VS + TS + col * 16 + 4 * qd);
            a[0] = x.x;
            a[1] = x.y;
            a[2] = x.z;
            a[3] = x.w;
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                ld16<float>(st + pad4(4 * qd + e), v[e]);
                a[e] = st[VS + TS + pad8(4 * qd + e) + col];
            }
        }
        if (head) {
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
                for (int l = 0; l < 16; ++l)
                    v[e][l] = 4 * qd + e > l ? v[e][l] : (4 * qd + e == l ? 1.0f : 0.0f);
        }
        // Z = V^T A: the quad's partial sums, reflectors 4 qd .. 4 qd + 3 to this thread
        float z[16], k8[8], zo[4];
#pragma unroll
        for (int l = 0; l < 16; ++l) {
            z[l] = v[0][l] * a[0];
#pragma unroll
            for (int e = 1; e < 4; ++e) z[l] = fmaf(v[e][l], a[e], z[l]);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float keep = (qd & 2) ? z[8 + i] : z[i], send = (qd & 2) ? z[i] : z[8 + i];
            k8[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float keep = (qd & 1) ? k8[4 + i] : k8[i], send = (qd & 1) ? k8[i] : k8[4 + i];
            zo[i] = keep + __shfl_xor_sync(0xffffffffu, send, 1);
            if (!head) zo[i] += top[i];
        }
        // W = T^T Z, top rows -= W
        float wo[4], w[16];
        gather(zo, z);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            float t[16], s0 = 0.0f, s1 = 0.0f;
            ld16<float>(st + VS + pad4(4 * qd + e), t);
#pragma unroll
            for (int m = 0; m < 16; m += 2) {
                s0 = fmaf(t[m], z[m], s0);
                s1 = fmaf(t[m + 1], z[m + 1], s1);
            }
            wo[e] = s0 + s1;
            if (!head) top[e] -= wo[e];
        }
        gather(wo, w);
        // A -= V W
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
            for (int l = 0; l < 16; l += 2) {
                s0 = fmaf(v[e][l], w[l], s0);
                s1 = fmaf(v[e][l + 1], w[l + 1], s1);
            }
            a[e] -= s0 + s1;
        }
        if (head) {
#pragma unroll
            for (int e = 0; e < 4; ++e) top[e] = a[e];
        } else {
            store4((int64_t)(args.pr + p) * 16, a);
        }
    }
    store4(top0, top);
}

// One panel kernel per tile size.
template <typename T, int LAYOUT, typename CT, int B>
int launch_panel_b(const PanelArgs &a, dim3 grid, cudaStream_t s) {
    using Cfg = PanelCfg<CT, B>;
    static std::atomic<bool> attr_set{false};
    constexpr size_t smem = Cfg::smem_bytes();
    static_assert(smem <= 227 * 1024, "panel shared memory");
    if (!attr_set) {
        AVS_CUDA_TRY(cudaFuncSetAttribute(panel_kernel<T, LAYOUT, CT, B>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)smem));
        attr_set = true;
    }
    panel_kernel<T, LAYOUT, CT, B><<<grid, Cfg::NTL, smem, s>>>(a);
    AVS_CUDA_TRY(cudaGetLastError());
    return AVS_SUCCESS;
}
template <typename T, int LAYOUT, typename CT>
int launch_panel_ct(const PanelArgs &a, dim3 grid, cudaStream_t s) {
    switch (a.b) {
        case 16: return launch_panel_b<T, LAYOUT, CT, 16>(a, grid, s);
        case 32: return launch_panel_b<T, LAYOUT, CT, 32>(a, grid, s);
        case 64: return launch_panel_b<T, LAYOUT, CT, 64>(a, grid, s);
        case 128: return launch_panel_b<T, LAYOUT, CT, 128>(a, grid, s);
        case 256: return launch_panel_b<T, LAYOUT, CT, 256>(a, grid, s);
        default: return AVS_ERR_UNSUPPORTED;
    }
}

// The panels' mailbox, cleared of any word that could pass for one of this call's
// (tags 1, 2, ...): b rows of 16 values for each of nt tiles.
template <typename T>
int panel_mail_reset(const Stage1Work &w, int64_t n, cudaStream_t s) {
    if (!w.mail) return AVS_SUCCESS;
    const size_t bytes = 2 * sizeof(T) * (size_t)n * kIB;
    const int batch = w.batch > 0 ? w.batch : 1;
    if (batch == 1) AVS_CUDA_TRY(cudaMemsetAsync(w.mail, 0, bytes, s));
    else AVS_CUDA_TRY(cudaMemset2DAsync(w.mail, sizeof(double) * (size_t)w.sMail, 0, bytes, batch, s));
    return AVS_SUCCESS;
}

// FP64 tiles with the double-float trailing updates (AVS_PREC_FP64X2) run
// the panel in double-float arithmetic too (CT = dfx: FP64 storage, each value
// converted on load and rounded back on store); GB300 issues FP64 at 1/64 of
// the FP32 rate and the panel's reflectors and applies are FP64-issue-bound.
template <typename T, int LAYOUT>
int launch_panel(T *dA, int64_t lda, int b, int pr, int pc, int P, int first_role, const Stage1Work &w,
                 cudaStream_t s, const int *ready = nullptr, const T *ref = nullptr) {
    const bool dfp = sizeof(T) == 8 && w.df_update;
    const int batch = w.batch > 0 ? w.batch : 1;
    AVS_CUDA_TRY(cudaMemsetAsync(w.flags, 0, sizeof(int) * (size_t)(batch > 1 ? w.sFlags * batch : 2 * P + 1), s));
    PanelArgs a;
    a.a = dA;
    a.lda = lda;
    a.b = b;
    a.pr = pr;
    a.pc = pc;
    a.P = P;
    a.first_role = first_role;
    a.tau = w.tau;
    a.tblk = w.tblk;
    a.ticket = w.flags;
    a.progress = w.flags + 1;
    a.err = w.err;
    a.sA = w.sA;
    a.sTau = w.sTau;
    a.sTblk = w.sTblk;
    a.sFlags = w.sFlags;
    a.mail = P - first_role > 1 && first_role == 0 ? static_cast<unsigned long long *>(w.mail) : nullptr;
    a.tag = (unsigned)(pr + pc + 1);  // half-step k of a call: 2 k + 1 (QR) or 2 k + 2 (LQ)
    // the diagonal of the call's first panel: given (out of core), or in the matrix once that panel is through
    a.ref = w.ref ? w.ref : (pr + pc > 0 ? (ref ? ref : dA) : nullptr);
    a.ref_ld = w.ref ? 1 : lda + 1;
    a.sRef = w.sA;
    a.sMail = w.sMail;
    a.ready = ready;
    a.ready_need = b / kChainStrip;
    const dim3 grid(P - first_role, batch);
    if constexpr (sizeof(T) == 8) {
        if (dfp) return launch_panel_ct<T, LAYOUT, dfx>(a, grid, s);
    }
    return launch_panel_ct<T, LAYOUT, T>(a, grid, s);
}

template <typename T, int LAYOUT, int B>
int launch_update_b(UpdateArgs a, int64_t ncols, const Stage1Work &w, cudaStream_t s) {
    using C = UpdCfg<T, B>;
    static std::atomic<bool> attr_set{false};
    constexpr size_t smem = C::smem_bytes();
    static_assert(smem <= 227 * 1024, "update shared memory");
    if (!attr_set) {
        AVS_CUDA_TRY(cudaFuncSetAttribute(update_kernel<T, LAYOUT, B>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)smem));
        attr_set = true;
    }
    const int batch = w.batch > 0 ? w.batch : 1;
    a.nstrip = (int)((ncols + C::W - 1) / C::W);
    // Tiles per CTA.  One tile per CTA where latency counts (FP32 n = 1024 tile 64
    // 5.0 ms, all tiles in one CTA 6.5; FP64 n = 512 tile 32 18.0 against 27.7, and
    // FP64 always: its tiles take long), and all of them once the strips fill the GPU
    // twice over by themselves (2 x 152 SMs; 32 matrices of order 1024 tile 64 10.5 ms against
    // 15.0, 256 of order 256 tile 32 2.2 against 3.0).  The values do not depend on it.
    const bool whole = C::F4 && (int64_t)a.nstrip * batch >= 304;
    a.group = whole ? a.P : 1;
    // ticket and counters: one per block and strip in the work's own array, else (out
    // of core) one per strip in the panel's flags, which are free again
    a.fine = w.uflags != nullptr;
    a.flags = a.fine ? w.uflags : w.flags;
    a.sFlags = a.fine ? w.sUflags : w.sFlags;
    const size_t fb = sizeof(int) * (size_t)(1 + a.nstrip * (a.fine ? C::NB : 1));
    if (batch > 1)
        AVS_CUDA_TRY(cudaMemset2DAsync(a.flags, sizeof(int) * (size_t)a.sFlags, 0, fb, batch, s));
    else
        AVS_CUDA_TRY(cudaMemsetAsync(a.flags, 0, fb, s));
    const int ngrp = (a.P - a.first_role + a.group - 1) / a.group;
    update_kernel<T, LAYOUT, B><<<dim3((unsigned)a.nstrip * ngrp, batch), C::NT, smem, s>>>(a);
    AVS_CUDA_TRY(cudaGetLastError());
    return AVS_SUCCESS;
}
template <int LAYOUT>
int launch_update16(const UpdateArgs &a, int64_t ncols, const Stage1Work &w, cudaStream_t s) {
    update16_kernel<LAYOUT><<<dim3((unsigned)(ncols / kU16W), w.batch > 0 ? w.batch : 1), kU16T, 0, s>>>(a);
    AVS_CUDA_TRY(cudaGetLastError());
    return AVS_SUCCESS;
}
template <typename T, int LAYOUT>
int launch_update(T *dA, int64_t lda, int64_t n, int b, int pr, int pc, int P, const Stage1Work &w,
                  cudaStream_t s, int first_role = 0) {
    const int64_t ncols = n - (int64_t)(pc + 1) * b;
    if (ncols <= 0 || P <= first_role) return AVS_SUCCESS;
    UpdateArgs a{};
    a.a = dA;
    a.lda = lda;
    a.n = n;
    a.b = b;
    a.pr = pr;
    a.pc = pc;
    a.P = P;
    a.first_role = first_role;
    a.tblk = w.tblk;
    a.err = w.err;
    a.sA = w.sA;
    a.sTblk = w.sTblk;
    switch (b) {
        case 16:
            if constexpr (sizeof(T) == 4) return launch_update16<LAYOUT>(a, ncols, w, s);
            else return launch_update_b<T, LAYOUT, 16>(a, ncols, w, s);
        case 32: return launch_update_b<T, LAYOUT, 32>(a, ncols, w, s);
        case 64: return launch_update_b<T, LAYOUT, 64>(a, ncols, w, s);
        default: return AVS_ERR_UNSUPPORTED;  // the full-T update
    }
}

// The tau of the panel just launched (roles 0..P-1 of half-step k, tile index
// first + p) to the caller's array, when it asked for them.
template <typename T>
int copy_tau_out(void *out, const Stage1Work &w, int nt, int k, int first, int P, int b, cudaStream_t s) {
    if (!out) return AVS_SUCCESS;
    AVS_CUDA_TRY(cudaMemcpyAsync(reinterpret_cast<T *>(out) + ((size_t)k * nt + first) * b, w.tau,
                                 sizeof(T) * (size_t)P * b, cudaMemcpyDeviceToDevice, s));
    return AVS_SUCCESS;
}

}  // namespace

// Tensor-core trailing update (the parts of stage1_tc_update in `parts`) of
// one half-step, bracketed by a pair of the caller's events when it asked for
// timing.
int timed_update(float *X, int64_t n, int b, int pr, int pc, int P, const Stage1Work &w, const TcBufs &tb,
                 cudaStream_t s, int64_t *launches, int parts = kTcAll, float *xt_out = nullptr,
                 int *ready = nullptr) {
    const bool timed = w.ev_pairs && w.ev_used && *w.ev_used < w.ev_cap;
    if (timed) AVS_CUDA_TRY(cudaEventRecord(w.ev_pairs[2 * *w.ev_used], s));
    const int rc = stage1_tc_update(X, n, b, pr, pc, P, w, tb, s, launches, parts, xt_out, ready);
    if (rc != AVS_SUCCESS) return rc;
    if (timed) {
        AVS_CUDA_TRY(cudaEventRecord(w.ev_pairs[2 * *w.ev_used + 1], s));
        ++*w.ev_used;
    }
    return AVS_SUCCESS;
}

// GE2BND with tensor-core trailing updates (FP32 tiles, b = 128 or 256, one
// matrix, lda = n): QR half-steps on X, LQ half-steps as QR half-steps on the
// transposed trailing block in XT.
//
// Lookahead: the next half-step's panel works on the top tile row that the
// chain of the current update computes (the chain writes it into the other
// buffer as well, transposed, and counts finished strips per tile), so the
// panel runs on the aux stream (high priority) beside the chain, each role
// waiting for its own tile, and beside the rest of the update (A_p -= Y_p W_p
// and the transpose of the rows below) on the caller's stream; its T build
// follows on aux.  The Y copies and S_p = Y_p^T A_p need the panel only and
// run beside the T build; the chain waits for both.  Every kernel touches the
// same data in the same order as without the overlap:
//   QR half-step k: the chain writes X row tile k (columns >= k+1) and its
//     transpose, XT column tile k = the LQ panel, which overlaps the rest of
//     the update of X rows >= k+1 and the transpose X -> XT of rows and
//     columns >= k+1.
//   LQ half-step k: the chain writes XT row tile k+1 and its transpose, X
//     column tile k+1 (rows >= k+1) = the next QR panel, which overlaps the
//     update of XT rows >= k+2 and the transposes back (XT rows >= k+2, and
//     the one tile XT(k+1, k) -> X(k, k+1)).
int stage1_ge2bnd_tc(float *X, int64_t n, int b, const Stage1Work &w, cudaStream_t s, int64_t *launches) {
    const int nt = (int)(n / b);
    const int fmt = w.tc_split;
    const TcBufs tb = stage1_tc_carve(w.tc_ws, n, b, fmt);
    float *XT = tb.xt;
    const bool la = w.aux && w.la_fork && w.la_panel && w.la_tb;
    cudaStream_t a = la ? w.aux : s;
    int rc, dev = 0, sms = 0;
    AVS_CUDA_TRY(cudaGetDevice(&dev));
    AVS_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    if ((rc = panel_mail_reset<float>(w, n, s)) != AVS_SUCCESS) return rc;
    if ((rc = stage1_tc_planes(X, n, fmt, tb, s)) != AVS_SUCCESS) return rc;
    // panel + tau copy + T build of one half-step on the aux stream, after the
    // caller's stream has reached this point (or the point where it recorded
    // la_fork: forked = true); hand-offs back after the panel and after the T
    // build
    auto panel_tb = [&](float *M, int pr, int pc, int P, void *tau_out, int k, int first, const int *ready,
                        bool forked = false) -> int {
        int r;
        if (la) {
            if (!forked) AVS_CUDA_TRY(cudaEventRecord(w.la_fork, s));
            AVS_CUDA_TRY(cudaStreamWaitEvent(a, w.la_fork, 0));
        }
        if ((r = launch_panel<float, 0>(M, n, b, pr, pc, P, 0, w, a, ready, X)) != AVS_SUCCESS) return r;
        if ((r = copy_tau_out<float>(tau_out, w, nt, k, first, P, b, a)) != AVS_SUCCESS) return r;
        if (la) AVS_CUDA_TRY(cudaEventRecord(w.la_panel, a));
        if ((int64_t)(pc + 1) * b < n && (r = stage1_tbuild<float>(M, n, b, 0, pr, pc, P, w, a)) != AVS_SUCCESS)
            return r;
        if (la) AVS_CUDA_TRY(cudaEventRecord(w.la_tb, a));
        if (launches) *launches += (int64_t)(pc + 1) * b < n ? 3 : 1;
        return AVS_SUCCESS;
    };
    // one half-step's update on the caller's stream, with the next panel
    // (on M2, panel tile (pr2, pc2), P2 tiles) started beside its chain
    auto half_step = [&](float *M, int pr, int pc, int P, float *M2, int pr2, int pc2, int P2, void *tau_out,
                         int k2, int first2) -> int {
        int r;
        if (la) AVS_CUDA_TRY(cudaStreamWaitEvent(s, w.la_panel, 0));
        if ((r = timed_update(M, n, b, pr, pc, P, w, tb, s, launches, kTcS)) != AVS_SUCCESS) return r;
        if (la) AVS_CUDA_TRY(cudaStreamWaitEvent(s, w.la_tb, 0));
        // The panel starts beside the chain (its roles wait for their tiles)
        // only while its P2 CTAs, on at most P2 SMs, leave at least half of the
        // SMs to the chain and the call holds its reservation (w.la_ready: the
        // waiting panels of all running calls within half of the SMs);
        // otherwise after it.  The chain is launched first:
        // where the two streams share a hardware queue the panel then simply
        // runs after it, so the panel's waits never hold the chain back.
        int *ready = (la && w.la_ready && 2 * P2 <= sms) ? tb.ready : nullptr;
        if ((r = timed_update(M, n, b, pr, pc, P, w, tb, s, launches, kTcPlanes, nullptr, ready)) != AVS_SUCCESS)
            return r;
        if (ready) AVS_CUDA_TRY(cudaEventRecord(w.la_fork, s));
        if ((r = timed_update(M, n, b, pr, pc, P, w, tb, s, launches, kTcChain, M2, ready)) != AVS_SUCCESS) return r;
        if ((r = panel_tb(M2, pr2, pc2, P2, tau_out, k2, first2, ready, ready != nullptr)) != AVS_SUCCESS) return r;
        return timed_update(M, n, b, pr, pc, P, w, tb, s, launches, kTcUpdate);
    };
    auto finish = [&](int r) -> int {  // the aux stream joins the caller's before any return
        if (la) {
            cudaEventRecord(w.la_fork, a);
            cudaStreamWaitEvent(s, w.la_fork, 0);
        }
        return r;
    };
    if ((rc = panel_tb(X, 0, 0, nt, w.tau_q_out, 0, 0, nullptr)) != AVS_SUCCESS) return finish(rc);
    for (int k = 0; k + 1 < nt; ++k) {
        const int64_t k1b = (int64_t)(k + 1) * b, k2b = (int64_t)(k + 2) * b;
        const int P = nt - k, PL = nt - k - 1;
        // QR half-step k (its panel and T build done or in flight on aux), the LQ panel beside it
        if ((rc = half_step(X, k, k, P, XT, k + 1, k, PL, w.tau_p_out, k, k + 1)) != AVS_SUCCESS) return finish(rc);
        // X rows, columns >= k+1 -> XT
        if ((rc = stage1_tc_transpose_box(X, XT, n, k1b, n - k1b, k1b, n - k1b, fmt, tb, s)) != AVS_SUCCESS)
            return finish(rc);
        // LQ half-step k, the next QR panel beside it
        if ((rc = half_step(XT, k + 1, k, PL, X, k + 1, k + 1, P - 1, w.tau_q_out, k + 1, k + 1)) != AVS_SUCCESS)
            return finish(rc);
        // and back: XT rows >= k+2 (all columns >= k) -> X, and the LQ panel's top tile
        if ((rc = stage1_tc_transpose_box(XT, X, n, k2b, n - k2b, (int64_t)k * b, n - (int64_t)k * b, fmt, tb, s)) !=
            AVS_SUCCESS)
            return finish(rc);
        if ((rc = stage1_tc_transpose_box(XT, X, n, k1b, b, (int64_t)k * b, b, fmt, tb, s)) != AVS_SUCCESS)
            return finish(rc);
        if (launches) *launches += 3;
    }
    // the last QR panel (one tile, no trailing columns) ran on aux
    return finish(AVS_SUCCESS);
}

template <typename T>
int stage1_ge2bnd(T *dA, int64_t n, int64_t lda, int b, const Stage1Work &w, cudaStream_t s, int64_t *launches) {
    const int nt = (int)(n / b);
    int rc;
    if constexpr (sizeof(T) == 4) {
        if (w.tc_split && w.tc_ws && b >= 128 && lda == n && (w.batch <= 1))
            return stage1_ge2bnd_tc(reinterpret_cast<float *>(dA), n, b, w, s, launches);
    }
    if ((rc = panel_mail_reset<T>(w, n, s)) != AVS_SUCCESS) return rc;
    for (int k = 0; k < nt; ++k) {
        // QR half-step: GEQRT(k,k) + TSQRT(row,k), Q^T applied to the row panels.
        const int P = nt - k;
        if ((rc = launch_panel<T, 0>(dA, lda, b, k, k, P, 0, w, s)) != AVS_SUCCESS) return rc;
        if ((rc = copy_tau_out<T>(w.tau_q_out, w, nt, k, k, P, b, s)) != AVS_SUCCESS) return rc;
        if (b >= 128 && w.tfull)
            rc = stage1_update_full<T>(dA, lda, n, b, 0, k, k, P, w, s);
        else
            rc = launch_update<T, 0>(dA, lda, n, b, k, k, P, w, s);
        if (rc != AVS_SUCCESS) return rc;
        if (launches) *launches += (k + 1 < nt) ? ((b >= 128 && w.tfull) ? 4 : 2) : 1;
        if (k == nt - 1) break;
        // LQ half-step: the same on the transposed view, top tile (k, k+1).
        const int PL = nt - k - 1;
        if ((rc = launch_panel<T, 1>(dA, lda, b, k + 1, k, PL, 0, w, s)) != AVS_SUCCESS) return rc;
        if ((rc = copy_tau_out<T>(w.tau_p_out, w, nt, k, k + 1, PL, b, s)) != AVS_SUCCESS) return rc;
        if (b >= 128 && w.tfull)
            rc = stage1_update_full<T>(dA, lda, n, b, 1, k + 1, k, PL, w, s);
        else
            rc = launch_update<T, 1>(dA, lda, n, b, k + 1, k, PL, w, s);
        if (rc != AVS_SUCCESS) return rc;
        if (launches) *launches += (b >= 128 && w.tfull) ? 4 : 2;
    }
    return AVS_SUCCESS;
}

// Tiled QR (tiled_QR!, KAbasedSVD/src/tiledalgos.jl:6-15): the QR half-steps
// of GE2BND alone.  On return R is in the upper triangle and the reflectors
// below it (unit lower V in the diagonal tiles, full V in the tiles below);
// dtau (optional) receives the tau of panel k, tile row r, reflector l at
// dtau[(k * nt + r) * b + l] (rows r >= k).
template <typename T>
int stage1_geqrf(T *dA, int64_t n, int64_t lda, int b, const Stage1Work &w, T *dtau, cudaStream_t s,
                 int64_t *launches) {
    const int nt = (int)(n / b);
    int rc;
    const bool tc = sizeof(T) == 4 && w.tc_split && w.tc_ws && b >= 128 && lda == n && w.batch <= 1;
    TcBufs tb{};
    if (tc) tb = stage1_tc_carve(w.tc_ws, n, b, w.tc_split);
    if ((rc = panel_mail_reset<T>(w, n, s)) != AVS_SUCCESS) return rc;
    for (int k = 0; k < nt; ++k) {
        const int P = nt - k;
        if ((rc = launch_panel<T, 0>(dA, lda, b, k, k, P, 0, w, s)) != AVS_SUCCESS) return rc;
        if (launches) ++*launches;
        if (dtau)
            AVS_CUDA_TRY(cudaMemcpyAsync(dtau + ((size_t)k * nt + k) * b, w.tau, sizeof(T) * (size_t)P * b,
                                         cudaMemcpyDeviceToDevice, s));
        if (k == nt - 1) break;
        if constexpr (sizeof(T) == 4) {
            if (tc) {
                // operand planes of the trailing block as the update reads it now
                const int64_t r0 = (int64_t)k * b, j0 = (int64_t)(k + 1) * b;
                if ((rc = stage1_tc_planes_block(reinterpret_cast<float *>(dA), n, r0, j0, w.tc_split, tb, s)) !=
                    AVS_SUCCESS)
                    return rc;
                if ((rc = stage1_tbuild<float>(reinterpret_cast<float *>(dA), n, b, 0, k, k, P, w, s)) != AVS_SUCCESS)
                    return rc;
                if ((rc = timed_update(reinterpret_cast<float *>(dA), n, b, k, k, P, w, tb, s, launches)) !=
                    AVS_SUCCESS)
                    return rc;
                if (launches) *launches += 3;
                continue;
            }
        }
        if (b >= 128 && w.tfull)
            rc = stage1_update_full<T>(dA, lda, n, b, 0, k, k, P, w, s);
        else
            rc = launch_update<T, 0>(dA, lda, n, b, k, k, P, w, s);
        if (rc != AVS_SUCCESS) return rc;
        if (launches) *launches += (b >= 128 && w.tfull) ? 3 : 1;
    }
    return AVS_SUCCESS;
}

template <typename T>
int stage1_geqrt_tile(T *dA, int b, T *dtau, const Stage1Work &w, cudaStream_t s) {
    int rc = launch_panel<T, 0>(dA, b, b, 0, 0, 1, 0, w, s);
    if (rc != AVS_SUCCESS) return rc;
    AVS_CUDA_TRY(cudaMemcpyAsync(dtau, w.tau, sizeof(T) * (size_t)(b - 1), cudaMemcpyDeviceToDevice, s));
    return AVS_SUCCESS;
}

// dRB: contiguous 2b x b buffer [R; B] (ld 2b); role 1 of a two-tile panel.
template <typename T>
int stage1_tsqrt_pair(T *dRB, int b, T *dtau, const Stage1Work &w, cudaStream_t s) {
    int rc = launch_panel<T, 0>(dRB, 2 * b, b, 0, 0, 2, 1, w, s);
    if (rc != AVS_SUCCESS) return rc;
    AVS_CUDA_TRY(cudaMemcpyAsync(dtau, reinterpret_cast<T *>(w.tau) + b, sizeof(T) * (size_t)b,
                                 cudaMemcpyDeviceToDevice, s));
    return AVS_SUCCESS;
}

// One panel (P tiles down tile column pc from tile row pr, roles first_role..P-1)
// and its trailing update over the columns right of the panel up to ncols, on
// the view `layout` (0: columns, 1: transposed) of dA: the full-T update for
// tiles >= 128 when w.tfull is given (as in stage1_ge2bnd), else the
// 16-reflector-block one.  The building blocks of the out-of-core driver,
// which runs a half-step as a sequence of such slabs with the top tile row
// carried from slab to slab.
template <typename T>
int stage1_panel(T *dA, int64_t lda, int b, int layout, int pr, int pc, int P, int first_role, const Stage1Work &w,
                 cudaStream_t s) {
    return layout == 0 ? launch_panel<T, 0>(dA, lda, b, pr, pc, P, first_role, w, s)
                       : launch_panel<T, 1>(dA, lda, b, pr, pc, P, first_role, w, s);
}
template <typename T>
int stage1_update(T *dA, int64_t lda, int64_t ncols, int b, int layout, int pr, int pc, int P, int first_role,
                  const Stage1Work &w, cudaStream_t s) {
    if (b >= 128 && w.tfull) return stage1_update_full<T>(dA, lda, ncols, b, layout, pr, pc, P, w, s, first_role);
    return layout == 0 ? launch_update<T, 0>(dA, lda, ncols, b, pr, pc, P, w, s, first_role)
                       : launch_update<T, 1>(dA, lda, ncols, b, pr, pc, P, w, s, first_role);
}
template int stage1_panel<float>(float *, int64_t, int, int, int, int, int, int, const Stage1Work &, cudaStream_t);
template int stage1_panel<double>(double *, int64_t, int, int, int, int, int, int, const Stage1Work &, cudaStream_t);
template int stage1_update<float>(float *, int64_t, int64_t, int, int, int, int, int, int, const Stage1Work &,
                                  cudaStream_t);
template int stage1_update<double>(double *, int64_t, int64_t, int, int, int, int, int, int, const Stage1Work &,
                                   cudaStream_t);

template int stage1_ge2bnd<float>(float *, int64_t, int64_t, int, const Stage1Work &, cudaStream_t, int64_t *);
template int stage1_ge2bnd<double>(double *, int64_t, int64_t, int, const Stage1Work &, cudaStream_t, int64_t *);
template int stage1_geqrt_tile<float>(float *, int, float *, const Stage1Work &, cudaStream_t);
template int stage1_geqrf<float>(float *, int64_t, int64_t, int, const Stage1Work &, float *, cudaStream_t,
                                 int64_t *);
template int stage1_geqrf<double>(double *, int64_t, int64_t, int, const Stage1Work &, double *, cudaStream_t,
                                  int64_t *);
template int stage1_geqrt_tile<double>(double *, int, double *, const Stage1Work &, cudaStream_t);
template int stage1_tsqrt_pair<float>(float *, int, float *, const Stage1Work &, cudaStream_t);
template int stage1_tsqrt_pair<double>(double *, int, double *, const Stage1Work &, cudaStream_t);

}  // namespace avs
