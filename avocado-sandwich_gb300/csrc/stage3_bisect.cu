// Stage 3: singular values of an upper bidiagonal B (d, e) by per-value FP64
// bisection on the Golub-Kahan tridiagonal TGK(B) (zero diagonal,
// off-diagonal d0, e0, d1, e1, ..., d_{n-1}; eigenvalues +-sigma_i).
//
// Replaces LAPACK.bdsdc!('U','N', d, e) (KAbasedSVD/src/bulgechasing.jl:50-53,
// CUDAbasedSVD/SVD_GPU.jl:267,281), which the reference runs on the CPU.
// Method: Sturm counts from the LDL^T pivots of TGK - x I with the pivot guard
// of LAPACK dstebz (Kahan's bisection), every loop bounded.  Output is
// descending, like bdsdc.
//
// B is scaled by a power of two so that every singular value lies in [0, 1), and
// a value is found as the cell of a dyadic grid that contains it: FP32 counts
// first, double-float counts on the cell and its neighbours, and for FP64 results of
// widths below 2^-40 FP64 counts on that cell and its neighbours, each on a group of G lanes that
// splits the bracket at G K points a pass.  A bracket whose edges a finer
// arithmetic does not confirm is dropped and that arithmetic starts again from
// [0, 1).  Widths below the grid's cells (2^-52 of the scale): halving in FP64 from
// there.  An infinite entry gives the infinite bound for every value.
#include <algorithm>
#include <cfloat>
#include <cmath>

#include "avs_common.cuh"
#include "df64.cuh"

namespace avs {
namespace {

// scratch[0] = Gershgorin bound of TGK (Inf when it overflows, or an entry is Inf),
// scratch[1] = pivmin, scratch[2] = exponent k of the scaling by 2^-k, scratch[3] =
// the bound of the scaled matrix: below 1 for finite entries (taken from quarters of
// the entries, whose sums don't overflow), else Inf (one block).
__device__ void tgk_bound_body(const double *d, const double *e, int64_t n, double *scratch) {
    __shared__ double sb[32], sq[32], sm[32];
    double bound = 0.0, quarter = 0.0, maxsq = 0.0;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        const double di = fabs(d[i]);
        const double el = i > 0 ? fabs(e[i - 1]) : 0.0;
        const double er = i + 1 < n ? fabs(e[i]) : 0.0;
        bound = fmax(bound, di + el + er);
        quarter = fmax(quarter, 0.25 * di + 0.25 * el + 0.25 * er);
        maxsq = fmax(maxsq, fmax(di * di, er * er));
    }
    for (int o = 16; o > 0; o >>= 1) {
        bound = fmax(bound, __shfl_xor_sync(0xffffffffu, bound, o));
        quarter = fmax(quarter, __shfl_xor_sync(0xffffffffu, quarter, o));
        maxsq = fmax(maxsq, __shfl_xor_sync(0xffffffffu, maxsq, o));
    }
    if ((threadIdx.x & 31) == 0) {
        sb[threadIdx.x >> 5] = bound;
        sq[threadIdx.x >> 5] = quarter;
        sm[threadIdx.x >> 5] = maxsq;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double b2 = 0.0, b4 = 0.0, m2 = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
            b2 = fmax(b2, sb[w]);
            b4 = fmax(b4, sq[w]);
            m2 = fmax(m2, sm[w]);
        }
        scratch[0] = b2;
        scratch[1] = DBL_MIN * fmax(m2, 1.0);
        // exponent of the scale: b2 2^-k < 1, with room for the bound's rounding
        int k = 0;
        double scaled = b4;
        if (b4 <= DBL_MAX && b2 > 0.0) {
            k = b4 >= 1.0 ? ilogb(b4 * (1.0 + 1e-6)) + 3 : ilogb(b2 * (1.0 + 1e-6)) + 1;
            scaled = b4 >= 1.0 ? scalbn(b4, 2 - k) : scalbn(b2, -k);
        }
        scratch[2] = (double)k;
        scratch[3] = scaled;
    }
}

__global__ void tgk_bound_kernel(const double *d, const double *e, int64_t n, double *scratch) {
    tgk_bound_body(d, e, n, scratch);
}

// Pivot recurrence q_i = -x - a_i / q_{i-1} (a_i = squared off-diagonal of
// TGK), counting negative pivots.  The division is replaced by a reciprocal:
// a single-precision estimate (hardware rcp) refined by one Newton-Raphson
// step r' = r (2 - q r), which leaves a relative error near 2^-46; pivots
// outside the single-precision range fall back to an FP64 division.  The
// count is then exact for off-diagonals perturbed by ~1e-14 relatively.
__device__ __forceinline__ double recip_nr(double q) {
    const double aq = fabs(q);
    if (aq > 1e-36 && aq < 1e36) {
        const double r = (double)__frcp_rn((float)q);
        const double e = fma(-q, r, 1.0);
        return fma(r, e, r);
    }
    return 1.0 / q;
}

__device__ __forceinline__ int tgk_count(const double *__restrict__ d, const double *__restrict__ e, int64_t n,
                                         double x, double pivmin) {
    int cnt = 0;
    double q = -x;
    if (fabs(q) < pivmin) q = -pivmin;
    cnt += (q < 0.0);
    for (int64_t i = 0; i < n; ++i) {
        const double di = __ldg(d + i);
        q = fma(-(di * di), recip_nr(q), -x);
        if (fabs(q) < pivmin) q = -pivmin;
        cnt += (q < 0.0);
        if (i + 1 < n) {
            const double ei = __ldg(e + i);
            q = fma(-(ei * ei), recip_nr(q), -x);
            if (fabs(q) < pivmin) q = -pivmin;
            cnt += (q < 0.0);
        }
    }
    return cnt;
}

// The same count in FP32 (used only to narrow the bracket; every bracket it
// produces is re-checked with FP64 counts before it is trusted).
__device__ __forceinline__ int tgk_count_f32(const double *__restrict__ d, const double *__restrict__ e, int64_t n,
                                             float x, float pivmin) {
    int cnt = 0;
    float q = -x;
    if (fabsf(q) < pivmin) q = -pivmin;
    cnt += (q < 0.0f);
    for (int64_t i = 0; i < n; ++i) {
        const float di = (float)__ldg(d + i);
        q = -x - __fdividef(di * di, q);
        if (fabsf(q) < pivmin || !isfinite(q)) q = -pivmin;
        cnt += (q < 0.0f);
        if (i + 1 < n) {
            const float ei = (float)__ldg(e + i);
            q = -x - __fdividef(ei * ei, q);
            if (fabsf(q) < pivmin || !isfinite(q)) q = -pivmin;
            cnt += (q < 0.0f);
        }
    }
    return cnt;
}

// The k-th largest singular value of the upper bidiagonal (d, e) of order n by one
// thread, from the bound and pivot guard in scratch[0..1]: the allocation-free
// call's form, which has no room for the squared off-diagonals the multisection
// below reads.
__device__ double bisect_value(const double *d, const double *e, int64_t n, int64_t k, double rel_tol,
                               const double *scratch) {
    const double bound = scratch[0];
    const double pivmin = scratch[1];
    if (bound == 0.0) return 0.0;
    const double tol = rel_tol * bound;
    const int64_t target = 2 * n - 1 - k;  // TGK index (ascending) of the k-th largest sigma
    double lo = 0.0, hi = bound * (1.0 + 4.0 * DBL_EPSILON) + pivmin;
    // phase 1: FP32 counts shrink the bracket to ~2^-18 of its width
    if (bound < 1e30 && bound > 1e-30) {
        float flo = 0.0f, fhi = (float)hi;
        const float fpiv = fmaxf((float)pivmin, 1e-37f);
        for (int it = 0; it < 18; ++it) {
            const float mid = 0.5f * (flo + fhi);
            if (mid <= flo || mid >= fhi) break;
            if (tgk_count_f32(d, e, n, mid, fpiv) > target)
                fhi = mid;
            else
                flo = mid;
        }
        // widen by a few FP32 ulps of the bracket and verify it in FP64
        const double w = fmax((double)(fhi - flo), 1e-7 * bound);
        const double tlo = fmax(0.0, (double)flo - w), thi = fmin(hi, (double)fhi + w);
        if (tgk_count(d, e, n, tlo, pivmin) <= target) lo = tlo;
        if (tgk_count(d, e, n, thi, pivmin) > target) hi = thi;
    }
    // phase 2: FP64 bisection to the requested width
    for (int it = 0; it < 128 && hi - lo > tol; ++it) {
        const double mid = 0.5 * (lo + hi);
        if (mid <= lo || mid >= hi) break;
        if (tgk_count(d, e, n, mid, pivmin) > target)
            hi = mid;
        else
            lo = mid;
    }
    return 0.5 * (lo + hi);
}

__global__ void bisect_thread_kernel(const double *d, const double *e, int64_t n, double rel_tol,
                                     const double *scratch, double *sigma) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= n) return;
    sigma[k] = bisect_value(d, e, n, k, rel_tol, scratch);
}

// ---- multisection on the scaled problem (every pipeline call) -----------------
// The squared scaled off-diagonals a_i = (off_i 2^-k)^2: as double-float pairs,
// and in FP64 for FP64 results (sq, may be null).
__device__ __forceinline__ void tgk_prep_one(double off, int k, int64_t i, float2 *a, double *sq) {
    const double o = scalbn(off, -k);
    const double v = o * o;
    const float h = (float)v;
    a[i] = make_float2(h, (float)(v - (double)h));
    if (sq) sq[i] = v;
}
__global__ void tgk_prep_kernel(const double *d, const double *e, int64_t n, const double *scratch, float2 *a,
                                double *sq) {
    const int k = (int)scratch[2];
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < 2 * n - 1;
         i += (int64_t)gridDim.x * blockDim.x)
        tgk_prep_one((i & 1) ? e[i >> 1] : d[i >> 1], k, i, a, sq);
}

__device__ __forceinline__ float rcp_ftz(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float pow2f(int e) { return __int_as_float((127 + e) << 23); }  // |e| <= 126
__device__ __forceinline__ double pow2d(int e) { return __hiloint2double((1023 + e) << 20, 0); }

// Sturm counts at K shifts at once (one pass over a, K interleaved recurrences
// q = -x - a / q).  The a_i are at most 1 and |q| is kept at 1e-36 or more, so no
// quotient overflows.
template <int K>
__device__ __forceinline__ void tgk_count_f(const float2 *__restrict__ a, int m, const float (&x)[K], int (&cnt)[K]) {
    constexpr float pivmin = 1e-36f;
    float q[K];
#pragma unroll
    for (int j = 0; j < K; ++j) {
        q[j] = x[j] < pivmin ? -pivmin : -x[j];
        cnt[j] = 1;
    }
#pragma unroll 4
    for (int i = 0; i < m; ++i) {
        const float ai = __ldg(a + i).x;
#pragma unroll
        for (int j = 0; j < K; ++j) {
            q[j] = fmaf(-ai, rcp_ftz(q[j]), -x[j]);
            if (fabsf(q[j]) < pivmin) q[j] = -pivmin;
            cnt[j] += __float_as_uint(q[j]) >> 31;
        }
    }
}
// In double-float: the quotient is t = a r with r ~ 1/q plus its residual
// (a - t q) r, about 20 instructions a pivot and 75 cycles of chain where a
// reciprocal refined in double-float and a product take 60 and 200; its relative
// error is below 2^-46 (r is refined once in FP32), so the counts are exact for a
// matrix within about 1e-14 of TGK(B), as those of the FP64 recurrence are.
template <int K>
__device__ __forceinline__ void tgk_count_df(const float2 *__restrict__ a, int m, const df64 (&x)[K],
                                             int (&cnt)[K]) {
    constexpr float pivmin = 1e-36f;
    df64 q[K];
#pragma unroll
    for (int j = 0; j < K; ++j) {
        q[j] = x[j].hi < pivmin ? df64{-pivmin, 0.0f} : df_neg(x[j]);
        cnt[j] = 1;
    }
#pragma unroll 2
    for (int i = 0; i < m; ++i) {
        const float2 ai = __ldg(a + i);
#pragma unroll
        for (int j = 0; j < K; ++j) {
            float r = rcp_ftz(q[j].hi);
            r = fmaf(r, fmaf(-q[j].hi, r, 1.0f), r);
            const float t = __fmul_rn(ai.x, r);
            const float rem = __fadd_rn(__fmaf_rn(-t, q[j].lo, __fmaf_rn(-t, q[j].hi, ai.x)), ai.y);
            const df64 s = two_sum(-x[j].hi, -t);
            const float lo = __fsub_rn(s.lo, __fmaf_rn(rem, r, x[j].lo));
            q[j] = fast_two_sum(s.hi, lo);
            if (fabsf(q[j].hi) < pivmin) q[j] = df64{-pivmin, 0.0f};
            cnt[j] += __float_as_uint(q[j].hi) >> 31;
        }
    }
}
// In FP64: q = -x - a r (2 - q r) with r ~ 1/q from FP32 (one refinement, relative
// error 2^-23, so 2^-46 after the step): three FP64 instructions a pivot.  GB300
// issues an FP64 warp instruction in 64 cycles per scheduler, conversions
// included, so q's FP32 image and r's FP64 one are made with integer operations.
__device__ __forceinline__ double tgk_step_d(double a, double q, double x) {
    const unsigned hi = (unsigned)__double2hiint(q), lo = (unsigned)__double2loint(q);
    const unsigned ex = (hi >> 20) & 0x7ffu;
    if (ex - (1023u - 115u) < 230u) {
        const unsigned sgn = hi & 0x80000000u;
        const unsigned mag = ((((hi & 0x7fffffffu) - (896u << 20)) << 3) | (lo >> 29)) + ((lo >> 28) & 1u);
        const float qf = __uint_as_float(mag | sgn);
        float r = rcp_ftz(qf);
        r = fmaf(r, fmaf(-qf, r, 1.0f), r);
        const unsigned rb = __float_as_uint(r);
        const double rd =
            __hiloint2double((int)((((rb & 0x7fffffffu) >> 3) + (896u << 20)) | sgn), (int)(rb << 29));
        return fma(-(a * rd), fma(-q, rd, 2.0), -x);
    }
    return -x - a / q;
}
__device__ __forceinline__ int tgk_count_d(const double *__restrict__ sq, int m, double x) {
    double q = x < DBL_MIN ? -DBL_MIN : -x;
    int cnt = 1;
#pragma unroll 2
    for (int i = 0; i < m; ++i) {
        q = tgk_step_d(__ldg(sq + i), q, x);
        // |q| < DBL_MIN (no exponent): the pivot guard
        if ((__double2hiint(q) & 0x7ff00000) == 0) q = -DBL_MIN;
        cnt += (unsigned)__double2hiint(q) - 0x80000000u <= 0x7ff00000u;  // q < 0, no NaN
    }
    return cnt;
}

// A bracket [lo, lo + 2^c) in units of 2^-depth; top: its upper edge is confirmed.
struct Bracket {
    long long lo;
    int depth, c;
    bool top;
};

constexpr int kDepthF = 18;      // cells of the FP32 phase: its counts err by up to a few 1e-7
constexpr int kDepthDfMax = 51;  // the double-float grid: exact pairs to depth 48, below it shifts near 1
                                 // round at 2^-50 (a width of 1e-15 of the bound, the least in double-float)
constexpr int kDepthDfD = 40;    // double-float cells before the FP64 phase, which narrower widths take

// One group (G consecutive lanes) splits the bracket at G K points per pass until
// its cell has the wanted depth.  exceed(v0, depth, ex): ex[j] = count at
// (v0 + j) 2^-depth > target.  Returns false when the lower edge turns out to lie
// above the value or the upper edge is never confirmed.
template <int G, int K, typename F>
__device__ __forceinline__ bool multisect(Bracket &b, int want, int gl, unsigned gmask, F exceed) {
    constexpr int NI = G * K;
    constexpr int P = NI >= 128 ? 7 : NI >= 64 ? 6 : NI >= 32 ? 5 : NI >= 16 ? 4 : NI >= 8 ? 3 : 2;
    static_assert(NI == (1 << P), "parts");
    while (b.depth < want || b.c > 0) {
        const int p = min(P, want - b.depth + b.c);
        const long long lo = b.lo << (p - b.c);
        const int depth = b.depth + p - b.c;
        bool ex[K];
        exceed(lo + gl * K, depth, ex);
        int first = NI;
#pragma unroll
        for (int j = K - 1; j >= 0; --j)
            if (ex[j] && lo + gl * K + j > 0) first = gl * K + j;
#pragma unroll
        for (int o = G / 2; o >= 1; o >>= 1) first = min(first, __shfl_xor_sync(gmask, first, o));
        if (first == 0) return false;
        const int parts = 1 << p;
        if (first <= parts && first < NI) b.top = true;
        b.lo = lo + min(first, parts) - 1;
        b.depth = depth;
        b.c = 0;
    }
    return b.top;
}
// The cell and its neighbours: one cell below, two above.
__device__ __forceinline__ Bracket widen(const Bracket &b) {
    return Bracket{b.lo > 0 ? b.lo - 1 : 0, b.depth, 2, false};
}

// k-th largest singular value.  F64: FP64 result (sq given), else double-float.
template <int G, bool F64>
__device__ double bisect_grp(const float2 *a, const double *sq, int64_t n, int64_t k, double rel_tol,
                             const double *scratch, int gl, unsigned gmask) {
    const double bound = scratch[0], scaled = scratch[3];
    if (!(bound > 0.0 && scaled <= 1.0)) return bound;  // 0, or an entry is Inf
    const int ke = (int)scratch[2];
    const int m = (int)(2 * n - 1);
    const int target = (int)(2 * n - 1 - k);  // TGK index (ascending) of the k-th largest sigma
    // depth whose cells are at most rel_tol * bound wide
    const double tol = fmin(F64 ? fmax(rel_tol * scaled, 1e-17) : fmax(rel_tol, 1e-15) * scaled, 0.5);
    int want = -ilogb(tol);
    if (pow2d(-want) > tol) ++want;
    want = max(want, kDepthF + 2);

    Bracket b{0, 0, 0, true};
    constexpr int K = 4;
    multisect<G, K>(b, kDepthF, gl, gmask, [&](long long v0, int depth, bool(&ex)[K]) {
        float x[K];
        int c[K];
#pragma unroll
        for (int j = 0; j < K; ++j) x[j] = (float)(int)(v0 + j) * pow2f(-depth);
        tgk_count_f<K>(a, m, x, c);
#pragma unroll
        for (int j = 0; j < K; ++j) ex[j] = c[j] > target;
    });
    auto ex_df = [&](long long v0, int depth, bool(&ex)[K]) {
        df64 x[K];
        int c[K];
#pragma unroll
        for (int j = 0; j < K; ++j) {  // the upper bits rounded to 24, the rest
            const long long v = v0 + j;
            const float h = (float)(unsigned)(v >> 20);
            const int r = (int)(v - ((long long)(unsigned)h << 20));
            x[j] = fast_two_sum(h * pow2f(20 - depth), (float)r * pow2f(-depth));
        }
        tgk_count_df<K>(a, m, x, c);
#pragma unroll
        for (int j = 0; j < K; ++j) ex[j] = c[j] > target;
    };
    const int wdf = F64 ? min(kDepthDfD, want) : min(want, kDepthDfMax);
    b = widen(b);
    if (!multisect<G, K>(b, wdf, gl, gmask, ex_df)) {
        b = Bracket{0, 0, 0, true};
        multisect<G, K>(b, wdf, gl, gmask, ex_df);
    }
    // FP64 counts for widths that double-float does not reach well: above that, its cell
    // (the counts err by 1e-14 of the bound) is the bracket asked for.  Measured (GB300, a
    // width of 1e-6, n = 4096): 2.5 ms; with the FP64 phase 39.5, the default width 28.8.
    if constexpr (F64) if (want > kDepthDfD) {
        const int wd = min(max(want, kDepthDfD + 2), 52);
        auto ex_d = [&](long long v0, int depth, bool(&ex)[1]) {
            ex[0] = tgk_count_d(sq, m, (double)v0 * pow2d(-depth)) > target;
        };
        b = widen(b);
        if (!multisect<G, 1>(b, wd, gl, gmask, ex_d)) {
            b = Bracket{0, 0, 0, true};
            multisect<G, 1>(b, wd, gl, gmask, ex_d);
        }
    }
    double lo = (double)b.lo * pow2d(-b.depth), hi = ((double)b.lo + 1.0) * pow2d(-b.depth);
    // no count reached the target below the bound (a NaN entry, which no comparison
    // counts): the bound
    if (lo > scaled) return bound;
    if constexpr (F64) if (want > kDepthDfD) {
        // a width below the grid's cells (2^-52 of the scale): halving, as far down as
        // FP64 numbers and the requested width go.  Every lane of the group runs the
        // same counts; the default width ends on the grid (one halving more for a bound
        // within 1e-6 below a power of two).
        for (int it = 0; it < 128 && hi - lo > rel_tol * scaled; ++it) {
            const double mid = 0.5 * (lo + hi);
            if (mid <= lo || mid >= hi) break;
            if (tgk_count_d(sq, m, mid) > target)
                hi = mid;
            else
                lo = mid;
        }
    }
    return scalbn(0.5 * (lo + hi), ke);
}

// Lanes per value.  A pass costs one count's latency while every scheduler has
// one warp or so, and its issue beyond; the shifts counted per resolved bit grow
// with G (G K shifts for log2(G K) bits).  So: as many lanes as fill the GPU about
// once.  Measured (GB300, double-float, tolerance 1e-10, ms): n = 128 G = 32 0.11,
// 8 0.14, 2 0.19; n = 1024 G = 16 0.71, 8 0.91, 32 1.04; n = 4096 G = 4 4.4, 2 5.2,
// 8 5.3; n = 5760 G = 2 7.3, 4 9.1; above n = 12288 the pivots no longer fit in L1
// and a second warp hides their latency: n = 16384 G = 2 39, 1 42, 4 51.  FP64: n =
// 512 G = 32 0.92, 16 1.09; n = 1024 G = 16 2.2, 32 2.6; n = 4096 G = 8 14.9, 16
// 20.3.  Before (two lanes, double-float reciprocals; FP64: one thread per value):
// n = 128 0.39, 1024 2.9, 4096 11.7, 16384 65 ms; FP64 n = 1024 31.8, 4096 127 ms.
// The value found is the grid's cell whatever G is, as long as the counts at
// neighbouring grid points are ordered, i.e. the cells are wider than the counts'
// errors (about 2n 1e-14 at the very worst): so for tolerances of 5e-11 and more
// and orders up to 2048 the batch may take part in the choice (256 matrices of order
// 256: G = 1 1.4 ms, 2 1.5, 4 2.5) and a matrix still gets the values of its single
// call bit for bit; otherwise G depends on the order alone.
inline int bisect_lanes(int64_t n, int64_t batch, double rel_tol, bool f64) {
    const int64_t nv = (!f64 && rel_tol >= 5e-11 && n <= 2048) ? n * batch : n;
    const int least = f64 ? 8 : (n > 12288 ? 2 : 1);
    int g = 32;
    while (g > least && nv * g > (f64 ? 16384 : 20480)) g >>= 1;
    return g;
}

template <int G, bool F64>
__global__ void __launch_bounds__(128) bisect_kernel(const float2 *a, const double *sq, int64_t n, int64_t batch,
                                                     int64_t sA, int64_t sScr, double rel_tol, const double *scratch,
                                                     double *sigma) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t g = t / G;
    if (g >= n * batch) return;  // whole groups: G divides the block size
    const int gl = (int)(t % G);
    const int64_t zb = g / n, k = g % n;
    const unsigned gmask = (G == 32) ? 0xffffffffu : (((1u << (G & 31)) - 1u) << ((threadIdx.x & 31) & ~(G - 1)));
    const double v = bisect_grp<G, F64>(a + zb * sA, F64 ? sq + zb * sA : nullptr, n, k, rel_tol, scratch + zb * sScr,
                                        gl, gmask);
    if (gl == 0) sigma[g] = v;
}

template <bool F64>
int launch_bisect(const float2 *a, const double *sq, int64_t n, int64_t batch, int64_t sA, int64_t sScr,
                  double rel_tol, const double *scratch, double *sigma, cudaStream_t s) {
    const int G = bisect_lanes(n, batch, rel_tol, F64);
    const unsigned blocks = (unsigned)((n * batch * G + 127) / 128);
    switch (G) {
        case 1:
            if constexpr (!F64)
                bisect_kernel<1, F64><<<blocks, 128, 0, s>>>(a, sq, n, batch, sA, sScr, rel_tol, scratch, sigma);
            break;
        case 2:
            if constexpr (!F64)
                bisect_kernel<2, F64><<<blocks, 128, 0, s>>>(a, sq, n, batch, sA, sScr, rel_tol, scratch, sigma);
            break;
        case 4:
            if constexpr (!F64)
                bisect_kernel<4, F64><<<blocks, 128, 0, s>>>(a, sq, n, batch, sA, sScr, rel_tol, scratch, sigma);
            break;
        case 8: bisect_kernel<8, F64><<<blocks, 128, 0, s>>>(a, sq, n, batch, sA, sScr, rel_tol, scratch, sigma); break;
        case 16: bisect_kernel<16, F64><<<blocks, 128, 0, s>>>(a, sq, n, batch, sA, sScr, rel_tol, scratch, sigma); break;
        default: bisect_kernel<32, F64><<<blocks, 128, 0, s>>>(a, sq, n, batch, sA, sScr, rel_tol, scratch, sigma); break;
    }
    AVS_CUDA_TRY(cudaGetLastError());
    return AVS_SUCCESS;
}

template <typename T>
__global__ void cast_kernel(const double *src, T *dst, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = (T)src[i];
}

template <typename TI, typename TO>
__global__ void copy2d_kernel(const TI *src, int64_t lds, TO *dst, int64_t ldd, int64_t rows, int64_t cols) {
    for (int64_t c = blockIdx.y; c < cols; c += gridDim.y)
        for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < rows; r += (int64_t)gridDim.x * blockDim.x)
            dst[r + c * ldd] = (TO)src[r + c * lds];
}

// Threads per CTA: small enough that the values spread over every SM.
inline int bisect_threads(int64_t n) {
    int t = 128;
    while (t > 32 && (n + t - 1) / t < 2 * 152) t >>= 1;
    return t;
}

}  // namespace

// FP64 results (dsq: 2n doubles) or double-float ones (dsq null); dpairs 2n pairs.
static int bisect_single(const double *dd, const double *de, int64_t n, double rel_tol, double *dsigma,
                         double *dscratch, float2 *dpairs, double *dsq, cudaStream_t s, int64_t *launches) {
    if (n <= 0) return AVS_SUCCESS;
    if (n > ((int64_t)1 << 29)) return AVS_ERR_UNSUPPORTED;  // pivots are counted in 32 bits
    tgk_bound_kernel<<<1, 1024, 0, s>>>(dd, de, n, dscratch);
    AVS_CUDA_TRY(cudaGetLastError());
    const int pb = (int)std::min<int64_t>((2 * n + 255) / 256, 1024);
    tgk_prep_kernel<<<pb, 256, 0, s>>>(dd, de, n, dscratch, dpairs, dsq);
    AVS_CUDA_TRY(cudaGetLastError());
    if (launches) *launches += 3;
    return dsq ? launch_bisect<true>(dpairs, dsq, n, 1, 0, 0, rel_tol, dscratch, dsigma, s)
               : launch_bisect<false>(dpairs, nullptr, n, 1, 0, 0, rel_tol, dscratch, dsigma, s);
}
int stage3_bisect(const double *dd, const double *de, int64_t n, double rel_tol, double *dsigma, double *dscratch,
                  float2 *dpairs, double *dsq, cudaStream_t s, int64_t *launches) {
    if (!(rel_tol > 0.0)) rel_tol = 2.0 * DBL_EPSILON;
    return bisect_single(dd, de, n, rel_tol, dsigma, dscratch, dpairs, dsq, s, launches);
}
int stage3_bisect_df(const double *dd, const double *de, int64_t n, double rel_tol, double *dsigma, double *dscratch,
                     float2 *dpairs, cudaStream_t s, int64_t *launches) {
    if (!(rel_tol > 0.0)) rel_tol = 1e-14;
    return bisect_single(dd, de, n, rel_tol, dsigma, dscratch, dpairs, nullptr, s, launches);
}

// ---------------------------------------------------------------------------
// Allocation-free variant of the bisection (avs_bidiag_svals_noalloc).
//
// Some callers cannot call cudaMalloc at the moment they need singular values:
// a host that has handed all device memory to its own pool allocator (Julia's
// CUDA.jl, PyTorch's caching allocator) and forbids allocations behind the
// pool's back, or a latency-critical loop that must not pay cudaMalloc's
// implicit device synchronisation.  For them the scratch of the bisection --
// the Gershgorin bound and pivot guard of TGK(B), and a zero-padded copy of the
// superdiagonal -- lives in the file-scope device array below instead of a
// workspace.  Every GPU that loads the library holds it (about 512 KiB) until
// the process exits.  Every call shares it and it keeps the last call's
// contents; calls that overlap on the GPU race on it.
constexpr int64_t kNoAllocMaxN = 65536;
constexpr int64_t kNoAllocHead = 8;  // [0] bound, [1] pivmin, rest unused
static __device__ __align__(256) double g_noalloc_scratch[kNoAllocHead + kNoAllocMaxN + 1];

}  // namespace avs

#include <mutex>

namespace avs {
namespace {
constexpr int kMaxDevices = 64;
double *g_noalloc_ptr[kMaxDevices] = {};
std::mutex g_noalloc_mu;
}  // namespace

// Device address of the static scratch for the current device.  Host code may
// not use g_noalloc_scratch as a device pointer (it names a host-side shadow),
// so the address is looked up once per device with that device current.
static int noalloc_scratch(double **out) {
    int dev = 0;
    AVS_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return AVS_ERR_UNSUPPORTED;
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
        void *p = nullptr;
        AVS_CUDA_TRY(cudaGetSymbolAddress(&p, g_noalloc_scratch));
        g_noalloc_ptr[dev] = static_cast<double *>(p);
    }
    *out = g_noalloc_ptr[dev];
    return AVS_SUCCESS;
}

int bidiag_svals_noalloc(int64_t n, const double *dd, const double *de, double *dsigma, double rel_tol,
                         cudaStream_t s) {
    if (n < 0) return -1;
    if (n > kNoAllocMaxN) return AVS_ERR_TOO_LARGE;
    if (n > 0 && !dd) return -2;
    if (n > 1 && !de) return -3;
    if (n > 0 && !dsigma) return -4;
    if (n == 0) return AVS_SUCCESS;
    double *scr = nullptr;
    int rc = noalloc_scratch(&scr);
    if (rc != AVS_SUCCESS) return rc;
    double *te = scr + kNoAllocHead;
    // the previous call's contents are still there: rewrite the whole padded copy
    if (n > 1) AVS_CUDA_TRY(cudaMemcpyAsync(te, de, sizeof(double) * (size_t)(n - 1), cudaMemcpyDeviceToDevice, s));
    AVS_CUDA_TRY(cudaMemsetAsync(te + (n - 1), 0, sizeof(double) * 2, s));
    if (!(rel_tol > 0.0)) rel_tol = 2.0 * DBL_EPSILON;
    tgk_bound_kernel<<<1, 1024, 0, s>>>(dd, te, n, scr);
    AVS_CUDA_TRY(cudaGetLastError());
    const int threads = bisect_threads(n);
    bisect_thread_kernel<<<(unsigned)((n + threads - 1) / threads), threads, 0, s>>>(dd, te, n, rel_tol, scr, dsigma);
    AVS_CUDA_TRY(cudaGetLastError());
    AVS_CUDA_TRY(cudaStreamSynchronize(s));
    return AVS_SUCCESS;
}

template <typename T>
int cast_from_double(const double *src, T *dst, int64_t n, cudaStream_t s) {
    const int nb = (int)std::min<int64_t>((n + 255) / 256, 1024);
    cast_kernel<T><<<nb > 0 ? nb : 1, 256, 0, s>>>(src, dst, n);
    AVS_CUDA_TRY(cudaGetLastError());
    return AVS_SUCCESS;
}
template int cast_from_double<float>(const double *, float *, int64_t, cudaStream_t);
template int cast_from_double<double>(const double *, double *, int64_t, cudaStream_t);

template <typename TI, typename TO>
int copy_convert_2d(const TI *src, int64_t lds, TO *dst, int64_t ldd, int64_t rows, int64_t cols, cudaStream_t s) {
    dim3 grid((unsigned)std::min<int64_t>((rows + 255) / 256, 64), (unsigned)std::min<int64_t>(cols, 65535));
    copy2d_kernel<TI, TO><<<grid, 256, 0, s>>>(src, lds, dst, ldd, rows, cols);
    AVS_CUDA_TRY(cudaGetLastError());
    return AVS_SUCCESS;
}
template int copy_convert_2d<float, float>(const float *, int64_t, float *, int64_t, int64_t, int64_t, cudaStream_t);
template int copy_convert_2d<double, double>(const double *, int64_t, double *, int64_t, int64_t, int64_t,
                                             cudaStream_t);
template int copy_convert_2d<float, double>(const float *, int64_t, double *, int64_t, int64_t, int64_t,
                                            cudaStream_t);
template int copy_convert_2d<double, float>(const double *, int64_t, float *, int64_t, int64_t, int64_t,
                                            cudaStream_t);

// ---------------------------------------------------------------------------
// Batched: `batch` bidiagonals of order n stacked at stride n (d, e), singular
// values to dsigma (stride n); pairs and squares at stride 2n.
namespace {
__global__ void tgk_bound_batched(const double *d, const double *e, int64_t n, double *scratch) {
    const int64_t zb = blockIdx.x;
    tgk_bound_body(d + zb * n, e + zb * n, n, scratch + zb * 4);
}
__global__ void tgk_prep_batched(const double *d, const double *e, int64_t n, int batch, const double *scratch,
                                 float2 *a, double *sq) {
    const int64_t m = 2 * n - 1;
    const int64_t total = m * (int64_t)batch;
    for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < total; g += (int64_t)gridDim.x * blockDim.x) {
        const int64_t zb = g / m, i = g % m;
        tgk_prep_one((i & 1) ? e[zb * n + (i >> 1)] : d[zb * n + (i >> 1)], (int)scratch[zb * 4 + 2], i,
                     a + zb * 2 * n, sq ? sq + zb * 2 * n : nullptr);
    }
}
}  // namespace

static int bisect_batch(const double *dd, const double *de, int64_t n, int batch, double rel_tol, double *dsigma,
                        double *dscratch, float2 *dpairs, double *dsq, cudaStream_t s, int64_t *launches) {
    if (n <= 0 || batch <= 0) return AVS_SUCCESS;
    if (n > ((int64_t)1 << 29)) return AVS_ERR_UNSUPPORTED;
    tgk_bound_batched<<<batch, 256, 0, s>>>(dd, de, n, dscratch);
    AVS_CUDA_TRY(cudaGetLastError());
    const int64_t total = (2 * n - 1) * (int64_t)batch;
    tgk_prep_batched<<<(unsigned)std::min<int64_t>((total + 255) / 256, 8192), 256, 0, s>>>(dd, de, n, batch, dscratch,
                                                                                           dpairs, dsq);
    AVS_CUDA_TRY(cudaGetLastError());
    if (launches) *launches += 3;
    return dsq ? launch_bisect<true>(dpairs, dsq, n, batch, 2 * n, 4, rel_tol, dscratch, dsigma, s)
               : launch_bisect<false>(dpairs, nullptr, n, batch, 2 * n, 4, rel_tol, dscratch, dsigma, s);
}
int stage3_bisect_batched(const double *dd, const double *de, int64_t n, int batch, double rel_tol, double *dsigma,
                          double *dscratch, float2 *dpairs, double *dsq, cudaStream_t s, int64_t *launches) {
    if (!(rel_tol > 0.0)) rel_tol = 2.0 * DBL_EPSILON;
    return bisect_batch(dd, de, n, batch, rel_tol, dsigma, dscratch, dpairs, dsq, s, launches);
}
int stage3_bisect_df_batched(const double *dd, const double *de, int64_t n, int batch, double rel_tol,
                             double *dsigma, double *dscratch, float2 *dpairs, cudaStream_t s, int64_t *launches) {
    if (!(rel_tol > 0.0)) rel_tol = 4e-14;
    return bisect_batch(dd, de, n, batch, rel_tol, dsigma, dscratch, dpairs, nullptr, s, launches);
}

}  // namespace avs
