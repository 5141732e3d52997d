// Stage 2a: blocked band reduction, upper band of width B -> upper band of
// width T (T < B, T | B), the first stage of the hierarchical bulge chase.
//
// Reference: one stage of bidiag! (BRD/src/bulgechasing2.jl:22-45) with
// factor B / T, i.e. cbw = B, tbw = ts = T: a sweep reduces T rows at once;
// its first op is LQ_QMUL on those rows, then QR_QMUL / LQ_QMUL pairs chase
// the bulge down the band (bulgechasing2.jl:4-20).  The reference also uses
// the halving form of this step in bidiagonalize (KAbasedSVD/src/
// bulgechasing.jl:33-42).
//
// Sweep s (rows p = sT .. p+T-1), step m, with c0 = p + T + mB:
//   R op (LQ_QMUL): the T pivot rows [rho, rho+T) (rho = p for m = 0, else
//     c0 - B) over the columns [c0, c0+B) are factored X = L Q (T
//     Householder reflectors from the right); the rows below, [rho+T, c0+B),
//     are multiplied by Q^T = I - V T V^T; X becomes [L 0].
//   L op (QR_QMUL): the rows [c0, c0+B) over the T pivot columns [c0, c0+T)
//     are factored QR (T reflectors from the left); the columns to their
//     right, [c0+T, c0+2B), are multiplied by Q^T = I - V T^T V^T.
// Every index range is clipped to n.  With T = 1 this is the element chase
// of stage2_chase.cu.  Op k of sweep s touches nothing that ops >= k+4 of sweep s-1
// touch, and of op k+3 one T x T corner only: the triangle its factorisation leaves in
// its pivot rows (columns), at the far end of op k's rows (columns), final before op
// k+3's apply.  So op k starts once sweep s-1 has finished op k+2, and reads the corner
// between its own factorisation and its apply, when sweep s-1 has announced it (done
// counts 2 per op and 1 for the corner); the result is bit-identical to running the
// sweeps one after another.
//
// One thread-block cluster of C CTAs owns a sweep.  Every CTA loads the
// panel and factors it itself (same data, same code: the same bits) and applies
// the block reflector to its share of the rows (R op) or columns (L op): W = A V (Z
// = V^T A), Y = W T (T^T Z) by forward substitution from the Gram matrix that the
// factorisation leaves (T^-1 = diag(1/tau) + striu(V^T V), one thread per row or
// column), A -= Y V^T (V Y); operands in shared memory, on the FP32 (or FP64) pipe.
// In double-float every product chain keeps an unnormalised pair (12 instead of 15
// instructions a multiply-add; n = 2048, band 128: 20.3 -> 18.8 ms).
// What bounds it: the latency of an op along the sweep wavefront (the panel's 16
// reflectors are half of it: 12 to 15 k of about 20 to 37 k cycles).  Measured (GB300,
// the whole stage, before: every column's work inside the panel's chain, T formed
// by one warp, one reflector per thread in the first product): band 64 n = 1024 3.3
// -> 2.4 ms, 128 n = 4096 15.4 -> 11.6 ms, 256 n = 16384 115 -> 84 ms; then, with a lag
// of three ops instead of four, 2.4 -> 2.0, 11.6 -> 9.6, 84 -> 67 ms.
// The band is in compact storage A(r, c) at AB[(r - c + 2B) + c * ldab],
// ldab = 3B + 1 (band_ku / band_ldab): rows c-2B .. c+B of column c (band,
// upper bulge up to 2B-1, lower bulge up to B-1), laid out so that every
// column segment an op moves starts on 16 bytes: staging and write-back move
// 16-byte vectors.
//
// Arithmetic: the element type R throughout (FP32 for the FP32-class modes,
// double-float for AVS_PREC_FP64X2, FP64 for the FP64 path), reflector scalars
// included.
#include <cooperative_groups.h>

#include <algorithm>
#include <type_traits>

#include "avs_common.cuh"
#include "band_scale.cuh"
#include "df64.cuh"
#include "reflect.cuh"
#include "vec16.cuh"

namespace cg = cooperative_groups;

namespace avs {
namespace {

template <int B, int T, int C>
struct BandCfg {
    static constexpr int NT = 256;                // threads per CTA
    static constexpr int NW = NT / 32;            // warps
    static constexpr int MR = 2 * B - T;          // rows (R op) / columns (L op) of the apply, at most
    static constexpr int PER = (MR + C - 1) / C;  // per CTA
    static constexpr int RQ = 4096 / B;           // granule that makes every micro-tile split exact
    static constexpr int RPC = (PER + RQ - 1) / RQ * RQ;  // rows (R op) / columns (L op) per CTA
    static constexpr int LDP = B + 4;             // panel: column stride (QR form, B rows)
    static constexpr int LDA_R = RPC + 4;         // R op staging: column stride (RPC rows)
    static constexpr int LDA_L = B + 4;           // L op staging: column stride (B rows)
    static constexpr int ASZ = (B * LDA_R > RPC * LDA_L) ? B * LDA_R : RPC * LDA_L;
    static constexpr int LDW = RPC + 4;           // W / Y buffer: [k][r or cc]
    // GEMM 1: 4 rows (R op) or 4 columns (L op) x 4 reflectors per thread, the sum
    // over the band's width split KS ways (partial W joined by the substitution)
    static constexpr int NG4 = RPC / 4;
    static constexpr int KS = NT / (NG4 * (T / 4));
    static constexpr int BK = B / KS;
    // GEMM 2, R op: 4 rows x CPT2R columns per thread
    static constexpr int NCG_R = NT / NG4;
    static constexpr int CPT2R = B / NCG_R;
    // GEMM 2, L op: 4 rows x CPT2L columns per thread
    static constexpr int NIG = B / 4;
    static constexpr int NCG_L = NT / NIG;
    static constexpr int CPT2L = RPC / NCG_L;
    static_assert(B % 32 == 0 && T <= 32 && T < B && B % T == 0, "band stage shape");
    static_assert(KS >= 1 && KS * NG4 * (T / 4) == NT && BK % 4 == 0 && RPC <= NT, "GEMM 1 split");
    static_assert(CPT2R % 4 == 0 && CPT2R * NCG_R == B, "R op GEMM 2 split");
    static_assert(NT % NIG == 0 && CPT2L % 4 == 0 && CPT2L * NCG_L == RPC, "L op GEMM 2 split");
    template <typename R>
    static constexpr size_t smem_bytes() {
        return sizeof(R) * ((size_t)T * LDP + ASZ + (size_t)KS * T * LDW + (size_t)T * (T + 1) + T);
    }
};

// Multiply-adds run on MacAr<R> accumulators (double-float: an unnormalised
// pair); the sum of one over a warp, and the value of lane src.
__device__ __forceinline__ bool positive(float a) { return a > 0.0f; }
__device__ __forceinline__ bool positive(double a) { return a > 0.0; }
__device__ __forceinline__ bool positive(dfx a) { return a.v.hi > 0.0f; }
__device__ __forceinline__ float wsum(float v) { return warp_sum(v); }
__device__ __forceinline__ double wsum(double v) { return warp_sum(v); }
__device__ __forceinline__ dfx wsum(df64 s) {
#pragma unroll 1
    for (int o = 16; o > 0; o >>= 1)
        s = MacAr<dfx>::mac_merge(s, df64{__shfl_xor_sync(0xffffffffu, s.hi, o), __shfl_xor_sync(0xffffffffu, s.lo, o)});
    return MacAr<dfx>::fin(s);
}
__device__ __forceinline__ float ldcg_elem(const float *p) { return __ldcg(p); }
__device__ __forceinline__ double ldcg_elem(const double *p) { return __ldcg(p); }
__device__ __forceinline__ dfx ldcg_elem(const dfx *p) {
    const float2 v = __ldcg(reinterpret_cast<const float2 *>(p));
    return dfx(df64{v.x, v.y});
}
__device__ __forceinline__ float wshfl(float v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ double wshfl(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ dfx wshfl(dfx v, int src) {
    return dfx(df64{__shfl_sync(0xffffffffu, v.v.hi, src), __shfl_sync(0xffffffffu, v.v.lo, src)});
}

template <typename R>
struct Vec4;
template <>
struct Vec4<float> {
    static __device__ __forceinline__ void ld(const float *p, float (&o)[4]) {
        const float4 v = *reinterpret_cast<const float4 *>(p);
        o[0] = v.x;
        o[1] = v.y;
        o[2] = v.z;
        o[3] = v.w;
    }
};
template <>
struct Vec4<double> {
    static __device__ __forceinline__ void ld(const double *p, double (&o)[4]) {
        const double2 a = *reinterpret_cast<const double2 *>(p);
        const double2 b = *reinterpret_cast<const double2 *>(p + 2);
        o[0] = a.x;
        o[1] = a.y;
        o[2] = b.x;
        o[3] = b.y;
    }
};

template <>
struct Vec4<dfx> {
    static __device__ __forceinline__ void ld(const dfx *p, dfx (&o)[4]) {
        const float4 a = *reinterpret_cast<const float4 *>(p);
        const float4 b = *reinterpret_cast<const float4 *>(p + 2);
        o[0] = dfx(df64{a.x, a.y});
        o[1] = dfx(df64{a.z, a.w});
        o[2] = dfx(df64{b.x, b.y});
        o[3] = dfx(df64{b.z, b.w});
    }
};

// 16-byte vectors of the element type: 4 floats, 2 doubles or 2 pairs.
template <typename R>
struct Vec16;
template <>
struct Vec16<float> {
    static constexpr int N = 4;
    static __device__ __forceinline__ void ld(const float *p, float (&o)[4]) {
        const float4 v = __ldcg(reinterpret_cast<const float4 *>(p));
        o[0] = v.x;
        o[1] = v.y;
        o[2] = v.z;
        o[3] = v.w;
    }
    static __device__ __forceinline__ void st(float *p, const float (&v)[4]) {
        *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
    }
};
template <>
struct Vec16<double> {
    static constexpr int N = 2;
    static __device__ __forceinline__ void ld(const double *p, double (&o)[2]) {
        const double2 v = __ldcg(reinterpret_cast<const double2 *>(p));
        o[0] = v.x;
        o[1] = v.y;
    }
    static __device__ __forceinline__ void st(double *p, const double (&v)[2]) {
        *reinterpret_cast<double2 *>(p) = make_double2(v[0], v[1]);
    }
};

template <>
struct Vec16<dfx> {
    static constexpr int N = 2;
    static __device__ __forceinline__ void ld(const dfx *p, dfx (&o)[2]) {
        const float4 v = __ldcg(reinterpret_cast<const float4 *>(p));
        o[0] = dfx(df64{v.x, v.y});
        o[1] = dfx(df64{v.z, v.w});
    }
    static __device__ __forceinline__ void st(dfx *p, const dfx (&v)[2]) {
        *reinterpret_cast<float4 *>(p) = make_float4(v[0].v.hi, v[0].v.lo, v[1].v.hi, v[1].v.lo);
    }
};

// Staging copy global (L2) -> shared of NV 16-byte vectors spread over NT
// threads: vector idx = tid + u * NT comes from src(idx) (nullptr: zeros) and
// goes to dst(idx, v).  The loads of a batch of 8 are all in flight before the
// first store, so a thread waits for about one L2 latency per batch instead of
// one per vector.
template <typename R, int NT, int NV, typename Src, typename Dst>
__device__ __forceinline__ void stage_in_vec(int tid, Src src, Dst dst) {
    constexpr int N = Vec16<R>::N;
    constexpr int PER = (NV + NT - 1) / NT;
    constexpr int BATCH = PER < 8 ? PER : 8;
#pragma unroll
    for (int u0 = 0; u0 < PER; u0 += BATCH) {
        R v[BATCH][N];
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
            const int idx = tid + (u0 + u) * NT;
            const R *p = (u0 + u < PER && idx < NV) ? src(idx) : nullptr;
            if (p) {
                Vec16<R>::ld(p, v[u]);
            } else {
#pragma unroll
                for (int e = 0; e < N; ++e) v[u][e] = R(0);
            }
        }
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
            const int idx = tid + (u0 + u) * NT;
            if (u0 + u < PER && idx < NV) dst(idx, v[u]);
        }
    }
}

__device__ __forceinline__ void cl_arrive() { asm volatile("barrier.cluster.arrive.aligned;" ::: "memory"); }
__device__ __forceinline__ void cl_wait() { asm volatile("barrier.cluster.wait.aligned;" ::: "memory"); }

// Householder QR of the panel P (B rows x T columns, column k at P + k*LDP,
// zero rows below the valid part), LAPACK convention per column: beta =
// -sign(alpha) ||x||, v = x / (alpha - beta) below the diagonal, v_k = 1,
// tau = (beta - alpha) / beta; tau = 0 when the part below the diagonal is
// zero.  On return P holds R on and above the diagonal and V below it;
// s_tau the taus; gram[j * (T+1) + k] = v_j^T v_k for j < k.  Warp w owns
// columns w, w + NW, ...; lane l rows l, l + 32, ....  The owner of column k+1
// applies H_k to that column first, forms H_{k+1}, publishes it (arrives at a named
// barrier) and only then applies H_k to its other columns: a step's chain is one
// dot product, one norm and the scalars (with the other columns' work on it, the
// panel took 16.4 k cycles at B = 128).
template <typename R, int B, int T, int NW>
__device__ __forceinline__ void panel_qr(R *P, R *s_tau, R *gram) {
    constexpr int LDP = B + 4;
    constexpr int CPW = (T + NW - 1) / NW;
    constexpr int RPL = B / 32;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    R x[CPW][RPL];
#pragma unroll
    for (int jj = 0; jj < CPW; ++jj) {
        const int j = w + NW * jj;
#pragma unroll
        for (int u = 0; u < RPL; ++u) x[jj][u] = (j < T) ? P[j * LDP + lane + 32 * u] : R(0);
    }
    // H_k of column k in slot JK of its owner
    auto generate = [&](auto slot_c, int k) {
        constexpr int JK = decltype(slot_c)::value;
        auto sq = MacAr<R>::mac0();
#pragma unroll
        for (int u = 0; u < RPL; ++u) {
            const int i = lane + 32 * u;
            if (i > k) MacAr<R>::mac(sq, x[JK][u], x[JK][u]);
        }
        const R s = wsum(sq);
        const R alpha = wshfl(x[JK][0], k);  // T <= 32: row k is in slot 0
        R tau = R(0), beta = alpha, scal = R(0);
        if (positive(s)) reflector_scalars(alpha, s, tau, beta, scal);
#pragma unroll
        for (int u = 0; u < RPL; ++u) {
            const int i = lane + 32 * u;
            if (i > k) x[JK][u] = x[JK][u] * scal;
            else if (i == k) x[JK][u] = beta;
            P[k * LDP + i] = x[JK][u];
        }
        if (lane == 0) s_tau[k] = tau;
        __syncwarp();
    };
    R v[RPL], tau;
    // H_k (v, tau) to the column in slot JJ: right of k the apply, left of k the Gram
    // entry v_j^T v_k (x holds v_j below its diagonal)
    auto apply = [&](auto slot_c, int j, int k) {
        constexpr int JJ = decltype(slot_c)::value;
        auto dot = MacAr<R>::mac0();
#pragma unroll
        for (int u = 0; u < RPL; ++u) MacAr<R>::mac(dot, v[u], x[JJ][u]);
        const R d = wsum(dot);
        if (j > k) {
            const R t = -(d * tau);
#pragma unroll
            for (int u = 0; u < RPL; ++u) {
                auto m = MacAr<R>::mac_from(x[JJ][u]);
                MacAr<R>::mac(m, t, v[u]);
                x[JJ][u] = MacAr<R>::fin(m);
            }
        } else if (lane == 0) {
            gram[j * (T + 1) + k] = d;
        }
    };
    auto slots = [&](auto f) {  // f for every column slot of the warp
        f(std::integral_constant<int, 0>{});
        if constexpr (CPW > 1) f(std::integral_constant<int, 1>{});
        if constexpr (CPW > 2) f(std::integral_constant<int, 2>{});
        if constexpr (CPW > 3) f(std::integral_constant<int, 3>{});
    };
    static_assert(CPW <= 4 && T % NW == 0, "panel columns");
    // barriers 1 and 2 in turn: column k's owner arrives, the other warps wait
    auto publish = [&](int k) {
        asm volatile("bar.arrive %0, %1;" ::"r"(1 + (k & 1)), "n"(32 * NW) : "memory");
    };
    if (w == 0) {
        generate(std::integral_constant<int, 0>{}, 0);
        publish(0);
    }
#pragma unroll 1
    for (int k = 0; k < T; ++k) {
        if (w != k % NW) asm volatile("bar.sync %0, %1;" ::"r"(1 + (k & 1)), "n"(32 * NW) : "memory");
        tau = s_tau[k];
#pragma unroll
        for (int u = 0; u < RPL; ++u) {
            const int i = lane + 32 * u;
            v[u] = (i > k) ? P[k * LDP + i] : (i == k ? R(1) : R(0));
        }
        const int kn = k + 1;
        const bool next = kn < T && w == kn % NW;
        if (next) {
            slots([&](auto sl) {
                if (kn / NW == decltype(sl)::value) {
                    apply(sl, kn, k);
                    generate(sl, kn);
                }
            });
            publish(kn);
        }
        slots([&](auto sl) {
            const int j = w + NW * decltype(sl)::value;
            if (j != k && !(next && j == kn)) apply(sl, j, k);
        });
    }
}

// Y from the partial W of one row (R op: Y = W T) or column (L op: Y = T^T Z): the
// same forward substitution y_k = tau_k (w_k - sum_{l<k} G_lk y_l).  Wy: KS
// partial sums [k][LDW] in, Y in the first on return; one thread per row.
template <typename R, int T, int KS, int LDW>
__device__ __forceinline__ void substitute(const R *s_tau, const R *gram, R *Wy, int row) {
    typename MacAr<R>::Mac w[T];
#pragma unroll
    for (int k = 0; k < T; ++k) {
        w[k] = MacAr<R>::mac_from(Wy[k * LDW + row]);
#pragma unroll
        for (int q = 1; q < KS; ++q) w[k] = MacAr<R>::mac_merge(w[k], MacAr<R>::mac_from(Wy[(q * T + k) * LDW + row]));
    }
#pragma unroll
    for (int k = 0; k < T; ++k) {
        const R y = s_tau[k] * MacAr<R>::fin(w[k]);
#pragma unroll
        for (int m = k + 1; m < T; ++m) MacAr<R>::mac(w[m], -gram[k * (T + 1) + m], y);
        Wy[k * LDW + row] = y;
    }
}
// The same with a lane per reflector: lane l of a group of T holds w_l of one row, y_k
// passes by shuffle.  A loop of T short steps instead of T^2 / 2 multiply-adds in a row.
template <typename R, int T, int KS, int LDW, int RPC, int NT>
__device__ __forceinline__ void substitute_lanes(const R *s_tau, const R *gram, R *Wy) {
    constexpr int GRP = NT / T;
    static_assert(RPC % GRP == 0, "rows per group");
    const int l = threadIdx.x % T, grp = threadIdx.x / T;
#pragma unroll 1
    for (int row = grp; row < RPC; row += GRP) {
        auto w = MacAr<R>::mac_from(Wy[l * LDW + row]);
#pragma unroll 1
        for (int q = 1; q < KS; ++q) w = MacAr<R>::mac_merge(w, MacAr<R>::mac_from(Wy[(q * T + l) * LDW + row]));
        R y = R(0);
#pragma unroll 1
        for (int k = 0; k < T; ++k) {
            const R yk = wshfl(s_tau[k] * MacAr<R>::fin(w), (threadIdx.x & 31 & ~(T - 1)) + k);
            if (l == k) y = yk;
            if (l > k) MacAr<R>::mac(w, -gram[k * (T + 1) + l], yk);
        }
        Wy[l * LDW + row] = y;
    }
}

template <int B, int T, typename R, int C>
__global__ void __launch_bounds__(256, sizeof(R) == 4 ? 2 : 1) band_stage_kernel(R *ab_base, int64_t n, int64_t ldab, int *ticket,
                                                          int *done_base, int *err, int batch, int64_t sAB,
                                                          int64_t sDone) {
    using Cfg = BandCfg<B, T, C>;
    // double-float: short loops (one row or column of the products at a time, the
    // substitution a lane per reflector), since unrolled as FP32 is the op's code does not
    // fit the instruction caches (band 64 n = 1024 7.0 -> 6.5 ms, 128 n = 2048 14.5 -> 12.6)
    constexpr bool kSmall = std::is_same<R, dfx>::value;
    constexpr int NT = Cfg::NT, NW = Cfg::NW, LDP = Cfg::LDP, RPC = Cfg::RPC, LDW = Cfg::LDW;
    constexpr int ku = band_ku(B);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R *P = reinterpret_cast<R *>(smem_raw);  // [T][LDP] panel (QR form), then V
    R *As = P + T * LDP;                      // apply staging
    R *Wy = As + Cfg::ASZ;                    // [KS][T][LDW]: partial W / Z, then Y in the first
    R *gram = Wy + Cfg::KS * T * LDW;         // [T][T+1]
    R *s_tau = gram + T * (T + 1);            // [T]
    __shared__ int s_j;
    cg::cluster_group cluster = cg::this_cluster();
    const int q = (int)cluster.block_rank();
    const int tid = threadIdx.x;

    const int64_t nsw = (n - 2 - T >= 0) ? (n - 2 - T) / T + 1 : 0;
    for (;;) {
        if (q == 0 && tid == 0) s_j = atomicAdd(ticket, 1);
        cluster.sync();
        const int64_t tk = *cluster.map_shared_rank(&s_j, 0);
        cluster.sync();
        const int64_t sw = tk / batch, zb = tk % batch;  // sweep-major over the batch
        if (sw >= nsw) return;
        R *ab = ab_base + zb * sAB;
        int *done = done_base + zb * sDone;
        auto at = [&](int64_t r, int64_t c) -> R * { return ab + (ku + r - c) + c * ldab; };
        const int64_t p = sw * T;
        const int nsteps = (int)((n - 2 - p - T) / B) + 1;
        const int ops_prev = (sw > 0) ? 2 * ((int)((n - 2 - p) / B) + 1) : 0;
        for (int op = 0; op < 2 * nsteps; ++op) {
            const int m = op >> 1;
            const bool rop = (op & 1) == 0;
            const int64_t c0 = p + T + (int64_t)m * B;
            // A wait that runs out records kDevTimeout; the cluster still runs its
            // barriers to the end (later waits return at once), so no CTA is left
            // at a cluster barrier.
            if (tid == 0 && sw > 0) wait_geq(done + sw - 1, 2 * min(op + 3, ops_prev), err);
            const bool corner = sw > 0 && op + 3 < ops_prev;  // op + 3's pivot corner is still to come
            __syncthreads();
            const int L = (int)(n - c0 < B ? n - c0 : (int64_t)B);  // R op: columns; L op: rows
            if (rop) {
                const int64_t rho = (m == 0) ? p : c0 - B;
                const int64_t r_lo = rho + T + (int64_t)q * RPC;
                const int64_t r_hi = (c0 + B < n) ? c0 + B : n;
                constexpr int VN = Vec16<R>::N;
                // panel (QR form): P[k][c'] = A(rho + k, c0 + c'); column c' of the
                // pivot rows is T / VN vectors
                stage_in_vec<R, NT, T / VN * B>(
                    tid,
                    [&](int idx) -> const R * {
                        const int cc = idx / (T / VN), pt = idx % (T / VN);
                        return (cc < L) ? at(rho + pt * VN, c0 + cc) : nullptr;
                    },
                    [&](int idx, const R(&v)[VN]) {
                        const int cc = idx / (T / VN), pt = idx % (T / VN);
#pragma unroll
                        for (int e = 0; e < VN; ++e) P[(pt * VN + e) * LDP + cc] = v[e];
                    });
                // this CTA's rows of the apply, column-major [c][r] (a vector that
                // starts below r_hi ends below c0 + B, inside the column's segment;
                // its rows at or past r_hi are zeroed)
                stage_in_vec<R, NT, RPC / VN * B>(
                    tid,
                    [&](int idx) -> const R * {
                        const int cc = idx / (RPC / VN), pt = idx % (RPC / VN);
                        return (cc < L && r_lo + pt * VN < r_hi) ? at(r_lo + pt * VN, c0 + cc) : nullptr;
                    },
                    [&](int idx, R(&v)[VN]) {
                        const int pt = idx % (RPC / VN);
#pragma unroll
                        for (int e = 1; e < VN; ++e)
                            if (r_lo + pt * VN + e >= r_hi) v[e] = R(0);
                        Vec16<R>::st(As + (idx / (RPC / VN)) * Cfg::LDA_R + pt * VN, v);
                    });
                __syncthreads();
                cl_arrive();  // done reading the pivot rows
                panel_qr<R, B, T, NW>(P, s_tau, gram);
                __syncthreads();
                cl_wait();  // every CTA has read the pivot rows: L and zeros, a share per CTA
                for (int idx = q * (T * B / C) + tid; idx < (q + 1) * (T * B / C); idx += NT) {
                    const int k = idx % T, j = idx / T;
                    if (j >= T && j < L) *at(rho + k, c0 + j) = R(0);
                }
                if (q == 0) {  // the T x T corner, the next sweep's
                    for (int idx = tid; idx < T * T; idx += NT) {
                        const int k = idx % T, j = idx / T;
                        if (j < L) *at(rho + k, c0 + j) = (j <= k) ? P[k * LDP + j] : R(0);
                    }
                }
                __syncthreads();
                if (q == 0 && tid == 0) st_release(done + sw, 2 * op + 1);
                const int64_t rc = c0 + B - T - r_lo;  // the corner's first row in this CTA's rows
                const bool mine = corner && rc > -T && rc < RPC;
                if (mine && tid == 0) wait_geq(done + sw - 1, 2 * (op + 3) + 1, err);
                for (int idx = tid; idx < T * T; idx += NT) {  // explicit V: unit diagonal, zeros above
                    const int k = idx / T, i = idx % T;
                    if (i <= k) P[k * LDP + i] = (i == k) ? R(1) : R(0);
                }
                __syncthreads();
                if (mine) {
                    for (int idx = tid; idx < T * T; idx += NT) {
                        const int64_t r = rc + idx % T;
                        const int c = B - T + idx / T;
                        if (r >= 0 && r < RPC && r_lo + r < r_hi && c < L)
                            As[c * Cfg::LDA_R + r] = ldcg_elem(at(r_lo + r, c0 + c));
                    }
                    __syncthreads();
                }
                // W = A V: thread = 4 rows x 4 reflectors, BK columns of the sum
                {
                    const int g = tid % Cfg::NG4, k0 = (tid / Cfg::NG4) % (T / 4) * 4, ks = tid / (Cfg::NG4 * (T / 4));
                    typename MacAr<R>::Mac acc[4][4];
#pragma unroll
                    for (int a = 0; a < 4; ++a)
#pragma unroll
                        for (int b2 = 0; b2 < 4; ++b2) acc[a][b2] = MacAr<R>::mac0();
                    if constexpr (kSmall) {
#pragma unroll 1
                        for (int c = ks * Cfg::BK; c < (ks + 1) * Cfg::BK; ++c) {
                            R a4[4];
                            Vec4<R>::ld(As + c * Cfg::LDA_R + 4 * g, a4);
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk) {
                                const R vk = P[(k0 + kk) * LDP + c];
#pragma unroll
                                for (int rr = 0; rr < 4; ++rr) MacAr<R>::mac(acc[kk][rr], a4[rr], vk);
                            }
                        }
                    } else {
#pragma unroll 2
                    for (int c = ks * Cfg::BK; c < (ks + 1) * Cfg::BK; c += 4) {
                        R a4[4][4], v4[4][4];
#pragma unroll
                        for (int cc = 0; cc < 4; ++cc) Vec4<R>::ld(As + (c + cc) * Cfg::LDA_R + 4 * g, a4[cc]);
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk) Vec4<R>::ld(P + (k0 + kk) * LDP + c, v4[kk]);
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                            for (int cc = 0; cc < 4; ++cc)
#pragma unroll
                                for (int rr = 0; rr < 4; ++rr) MacAr<R>::mac(acc[kk][rr], a4[cc][rr], v4[kk][cc]);
                    }
                    }
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                        for (int rr = 0; rr < 4; ++rr) Wy[(ks * T + k0 + kk) * LDW + 4 * g + rr] = MacAr<R>::fin(acc[kk][rr]);
                }
                __syncthreads();
                if constexpr (kSmall) substitute_lanes<R, T, Cfg::KS, LDW, RPC, NT>(s_tau, gram, Wy);
                else if (tid < RPC) substitute<R, T, Cfg::KS, LDW>(s_tau, gram, Wy, tid);
                __syncthreads();
                // A -= Y V^T: thread = 4 rows x CPT2R columns; straight to global
                {
                    constexpr int CPT = Cfg::CPT2R;
                    const int g = tid % Cfg::NG4, cgp = tid / Cfg::NG4;
                    const int cb = cgp * CPT;
                    typename MacAr<R>::Mac acc[4][CPT];
#pragma unroll
                    for (int cc = 0; cc < CPT; ++cc)
#pragma unroll
                        for (int rr = 0; rr < 4; ++rr) acc[rr][cc] = MacAr<R>::mac_from(As[(cb + cc) * Cfg::LDA_R + 4 * g + rr]);
#pragma unroll(kSmall ? 1 : 16)
                    for (int k = 0; k < T; ++k) {
                        R y4[4];
                        Vec4<R>::ld(Wy + k * LDW + 4 * g, y4);
#pragma unroll
                        for (int c4 = 0; c4 < CPT; c4 += 4) {
                            R v4[4];
                            Vec4<R>::ld(P + k * LDP + cb + c4, v4);
#pragma unroll
                            for (int cc = 0; cc < 4; ++cc)
#pragma unroll
                                for (int rr = 0; rr < 4; ++rr)
                                    MacAr<R>::mac(acc[rr][c4 + cc], -y4[rr], v4[cc]);
                        }
                    }
                    constexpr int VN = Vec16<R>::N;
#pragma unroll
                    for (int cc = 0; cc < CPT; ++cc) {
                        const int c = cb + cc;
                        if (c < L) {
#pragma unroll
                            for (int r0 = 0; r0 < 4; r0 += VN) {
                                const int64_t r = r_lo + 4 * g + r0;
                                if (r + VN <= r_hi) {
                                    R v[VN];
#pragma unroll
                                    for (int e = 0; e < VN; ++e) v[e] = MacAr<R>::fin(acc[r0 + e][cc]);
                                    Vec16<R>::st(at(r, c0 + c), v);
                                } else {
#pragma unroll
                                    for (int e = 0; e < VN; ++e)
                                        if (r + e < r_hi) *at(r + e, c0 + c) = MacAr<R>::fin(acc[r0 + e][cc]);
                                }
                            }
                        }
                    }
                }
            } else {
                const int Tc = (int)(n - c0 < T ? n - c0 : (int64_t)T);  // pivot columns
                const int64_t cc_lo = c0 + T + (int64_t)q * RPC;
                const int64_t c_hi = (c0 + 2 * B < n) ? c0 + 2 * B : n;
                constexpr int VN = Vec16<R>::N;
                // panel: P[k][i] = A(c0 + i, c0 + k); a vector that starts below L
                // stays inside the column's segment, its rows at or past L are zeroed
                stage_in_vec<R, NT, B / VN * T>(
                    tid,
                    [&](int idx) -> const R * {
                        const int k = idx / (B / VN), pt = idx % (B / VN);
                        return (pt * VN < L && k < Tc) ? at(c0 + pt * VN, c0 + k) : nullptr;
                    },
                    [&](int idx, R(&v)[VN]) {
                        const int pt = idx % (B / VN);
#pragma unroll
                        for (int e = 1; e < VN; ++e)
                            if (pt * VN + e >= L) v[e] = R(0);
                        Vec16<R>::st(P + (idx / (B / VN)) * LDP + pt * VN, v);
                    });
                // this CTA's columns of the apply, column-major [cc][i]
                stage_in_vec<R, NT, B / VN * RPC>(
                    tid,
                    [&](int idx) -> const R * {
                        const int cc = idx / (B / VN), pt = idx % (B / VN);
                        return (pt * VN < L && cc_lo + cc < c_hi) ? at(c0 + pt * VN, cc_lo + cc) : nullptr;
                    },
                    [&](int idx, R(&v)[VN]) {
                        const int pt = idx % (B / VN);
#pragma unroll
                        for (int e = 1; e < VN; ++e)
                            if (pt * VN + e >= L) v[e] = R(0);
                        Vec16<R>::st(As + (idx / (B / VN)) * Cfg::LDA_L + pt * VN, v);
                    });
                __syncthreads();
                cl_arrive();  // done reading the pivot columns
                panel_qr<R, B, T, NW>(P, s_tau, gram);
                __syncthreads();
                cl_wait();  // R and zeros, a share per CTA
                for (int idx = q * (T * B / C) + tid; idx < (q + 1) * (T * B / C); idx += NT) {
                    const int i = idx % B, k = idx / B;
                    if (i >= T && i < L && k < Tc) *at(c0 + i, c0 + k) = R(0);
                }
                if (q == 0) {  // the T x T corner, the next sweep's
                    for (int idx = tid; idx < T * T; idx += NT) {
                        const int i = idx % T, k = idx / T;
                        if (i < L && k < Tc) *at(c0 + i, c0 + k) = (i <= k) ? P[k * LDP + i] : R(0);
                    }
                }
                __syncthreads();
                if (q == 0 && tid == 0) st_release(done + sw, 2 * op + 1);
                const int64_t rc = c0 + 2 * B - T - cc_lo;  // the corner's first column in this CTA's columns
                const bool mine = corner && rc > -T && rc < RPC;
                if (mine && tid == 0) wait_geq(done + sw - 1, 2 * (op + 3) + 1, err);
                for (int idx = tid; idx < T * T; idx += NT) {
                    const int k = idx / T, i = idx % T;
                    if (i <= k) P[k * LDP + i] = (i == k) ? R(1) : R(0);
                }
                __syncthreads();
                if (mine) {
                    for (int idx = tid; idx < T * T; idx += NT) {
                        const int i = B - T + idx % T;
                        const int64_t c = rc + idx / T;
                        if (c >= 0 && c < RPC && cc_lo + c < c_hi && i < L)
                            As[c * Cfg::LDA_L + i] = ldcg_elem(at(c0 + i, cc_lo + c));
                    }
                    __syncthreads();
                }
                // Z = V^T A: thread = 4 columns (g + cc NG4: lanes one column apart, so
                // their column reads spread over the banks) x 4 reflectors, BK rows of the sum
                {
                    const int g = tid % Cfg::NG4, k0 = (tid / Cfg::NG4) % (T / 4) * 4, ks = tid / (Cfg::NG4 * (T / 4));
                    typename MacAr<R>::Mac acc[4][4];
#pragma unroll
                    for (int a = 0; a < 4; ++a)
#pragma unroll
                        for (int b2 = 0; b2 < 4; ++b2) acc[a][b2] = MacAr<R>::mac0();
                    if constexpr (kSmall) {
#pragma unroll 1
                        for (int i = ks * Cfg::BK; i < (ks + 1) * Cfg::BK; ++i) {
                            R a4[4];
#pragma unroll
                            for (int cc = 0; cc < 4; ++cc) a4[cc] = As[(g + cc * Cfg::NG4) * Cfg::LDA_L + i];
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk) {
                                const R vk = P[(k0 + kk) * LDP + i];
#pragma unroll
                                for (int cc = 0; cc < 4; ++cc) MacAr<R>::mac(acc[kk][cc], vk, a4[cc]);
                            }
                        }
                    } else {
#pragma unroll 2
                    for (int i = ks * Cfg::BK; i < (ks + 1) * Cfg::BK; i += 4) {
                        R a4[4][4], v4[4][4];
#pragma unroll
                        for (int cc = 0; cc < 4; ++cc)
                            Vec4<R>::ld(As + (g + cc * Cfg::NG4) * Cfg::LDA_L + i, a4[cc]);
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk) Vec4<R>::ld(P + (k0 + kk) * LDP + i, v4[kk]);
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                            for (int cc = 0; cc < 4; ++cc)
#pragma unroll
                                for (int ii = 0; ii < 4; ++ii) MacAr<R>::mac(acc[kk][cc], v4[kk][ii], a4[cc][ii]);
                    }
                    }
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                        for (int cc = 0; cc < 4; ++cc) Wy[(ks * T + k0 + kk) * LDW + g + cc * Cfg::NG4] = MacAr<R>::fin(acc[kk][cc]);
                }
                __syncthreads();
                if constexpr (kSmall) substitute_lanes<R, T, Cfg::KS, LDW, RPC, NT>(s_tau, gram, Wy);
                else if (tid < RPC) substitute<R, T, Cfg::KS, LDW>(s_tau, gram, Wy, tid);
                __syncthreads();
                // A -= V Y: thread = 4 rows x CPT2L columns; straight to global
                {
                    constexpr int CPT = Cfg::CPT2L;
                    const int ig = tid % Cfg::NIG, cgp = tid / Cfg::NIG;
                    const int cb = cgp * CPT;
                    typename MacAr<R>::Mac acc[4][CPT];
#pragma unroll
                    for (int cc = 0; cc < CPT; ++cc)
#pragma unroll
                        for (int ii = 0; ii < 4; ++ii) acc[ii][cc] = MacAr<R>::mac_from(As[(cb + cc) * Cfg::LDA_L + 4 * ig + ii]);
#pragma unroll(kSmall ? 1 : 16)
                    for (int k = 0; k < T; ++k) {
                        R v4[4];
                        Vec4<R>::ld(P + k * LDP + 4 * ig, v4);
#pragma unroll
                        for (int c4 = 0; c4 < CPT; c4 += 4) {
                            R y4[4];
                            Vec4<R>::ld(Wy + k * LDW + cb + c4, y4);
#pragma unroll
                            for (int cc = 0; cc < 4; ++cc)
#pragma unroll
                                for (int ii = 0; ii < 4; ++ii)
                                    MacAr<R>::mac(acc[ii][c4 + cc], -v4[ii], y4[cc]);
                        }
                    }
                    constexpr int VN = Vec16<R>::N;
#pragma unroll
                    for (int cc = 0; cc < CPT; ++cc) {
                        const int64_t c = cc_lo + cb + cc;
                        if (c < c_hi) {
#pragma unroll
                            for (int i0 = 0; i0 < 4; i0 += VN) {
                                const int i = 4 * ig + i0;
                                if (i + VN <= L) {
                                    R v[VN];
#pragma unroll
                                    for (int e = 0; e < VN; ++e) v[e] = MacAr<R>::fin(acc[i0 + e][cc]);
                                    Vec16<R>::st(at(c0 + i, c), v);
                                } else {
#pragma unroll
                                    for (int e = 0; e < VN; ++e)
                                        if (i + e < L) *at(c0 + i + e, c) = MacAr<R>::fin(acc[i0 + e][cc]);
                                }
                            }
                        }
                    }
                }
            }
            // the op's stores, made visible at GPU scope by one fence per CTA (after
            // the CTA barrier), then the cluster barrier, then the release
            __syncthreads();
            if (tid == 0) __threadfence();
            cluster.sync();
            if (q == 0 && tid == 0) st_release(done + sw, 2 * (op + 1));
        }
    }
}

template <int B, int T, typename R, int C>
int launch_band_stage(R *dAB, int64_t n, int64_t ldab, const Stage2Work &w, cudaStream_t s, int num_sms, int batch,
                      int64_t sAB, int64_t sDone) {
    using Cfg = BandCfg<B, T, C>;
    const size_t smem = Cfg::template smem_bytes<R>();
    auto kern = band_stage_kernel<B, T, R, C>;
    AVS_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    if (C > 8) AVS_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.blockDim = dim3(Cfg::NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3(C * 64);
    int max_clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&max_clusters, kern, &cfg) != cudaSuccess || max_clusters <= 0) {
        cudaGetLastError();
        max_clusters = std::max(1, num_sms / C);
    }
    const int64_t nsw = (n - 2 - T >= 0) ? (n - 2 - T) / T + 1 : 0;
    if (nsw == 0) return AVS_SUCCESS;
    // sweeps in flight: a sweep's 2 n / B ops over a lag of 3 ops
    const int64_t want = std::max<int64_t>(1, (2 * (n / B) / 3 + 2) * (int64_t)batch);
    const int64_t clusters = std::min<int64_t>(std::min<int64_t>(want, max_clusters), nsw * (int64_t)batch);
    cfg.gridDim = dim3((unsigned)(clusters * C));
    AVS_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, dAB, n, ldab, w.flags, w.flags + 1, w.err, batch, sAB, sDone));
    return AVS_SUCCESS;
}

// dense (leading dimension lda, matrix stride sA) -> compact band of width
// bw (ku = band_ku(bw)), scaled (band_scale.cuh), zeros outside 0 <= c - r <= bw
template <typename TI, typename R>
__global__ void dense_to_band_kernel(const TI *a, int64_t n, int64_t lda, int64_t sA, int bw, R *ab, int64_t ldab,
                                     int64_t sAB, const int *scale) {
    const int64_t c = blockIdx.x;
    const int64_t zb = blockIdx.y;
    const int ku = band_ku(bw);
    const TI f = pow2<TI>(-band_exponent(scale, zb));
    const TI *az = a + zb * sA;
    R *abz = ab + zb * sAB + c * ldab;
    for (int i = threadIdx.x; i < ldab; i += blockDim.x) {
        const int64_t r = c - ku + i;
        abz[i] = (r >= 0 && r <= c && c - r <= bw) ? (R)(az[r + c * lda] * f) : R(0);
    }
}

// compact band (width bw1 storage) holding a band of width bw2 -> compact
// band of width bw2 (ku2 = 2 bw2 - 1) of storage type St (float2: double-float
// pairs; double)
template <typename R, typename St>
__global__ void band_to_band_kernel(const R *ab1, int64_t n, int bw1, int64_t ldab1, int64_t sAB1, int bw2, St *ab2,
                                    int64_t ldab2, int64_t sAB2) {
    const int64_t c = blockIdx.x;
    const int64_t zb = blockIdx.y;
    const int ku1 = band_ku(bw1), ku2 = 2 * bw2 - 1;
    const R *src = ab1 + zb * sAB1;
    St *dst = ab2 + zb * sAB2 + c * ldab2;
    for (int i = threadIdx.x; i < ldab2; i += blockDim.x) {
        const int64_t r = c - ku2 + i;
        const bool in = (r >= 0 && r <= c && c - r <= bw2);
        const R v = in ? src[(ku1 + r - c) + c * ldab1] : R(0);
        if constexpr (std::is_same<R, dfx>::value) {
            dst[i] = make_float2(v.v.hi, v.v.lo);
        } else if constexpr (std::is_same<St, float2>::value) {
            const float h = (float)v;
            dst[i] = make_float2(h, (float)((double)v - (double)h));
        } else {
            dst[i] = (St)v;
        }
    }
}

// compact band (width bw storage) -> dense column-major n x n: every entry the
// compact storage holds (rows c-2bw .. c+bw of column c), scaled back, zeros elsewhere
template <typename R>
__global__ void band_to_dense_kernel(const R *ab, int64_t n, int bw, int64_t ldab, R *a, int64_t lda,
                                     const int *scale) {
    const int64_t c = blockIdx.x;
    const int ku = band_ku(bw);
    const R f = pow2<R>(band_exponent(scale, 0));
    for (int64_t r = threadIdx.x; r < n; r += blockDim.x) {
        const int64_t i = ku + r - c;
        a[r + c * lda] = (i >= 0 && i < ldab) ? ab[i + c * ldab] * f : R(0);
    }
}

// CTAs per cluster: the apply's 2B - T rows (columns) split C ways; FP64
// operands at band 256 take 16 CTAs (a non-portable cluster size) so that a
// CTA's staging fits in shared memory.
template <int B, typename R>
constexpr int band_cluster() {
    return B == 256 ? (sizeof(R) == 8 ? 16 : 8) : (B == 128 ? 8 : 2);
}

}  // namespace

template <typename R>
int band_stage(R *dAB, int64_t n, int bw, int tbw, int64_t ldab, const Stage2Work &w, cudaStream_t s, int num_sms,
               int batch, int64_t sAB, int64_t sDone) {
    if (n < 3) return AVS_SUCCESS;
    if (ldab != band_ldab(bw)) return AVS_ERR_INTERNAL;
    AVS_CUDA_TRY(cudaMemsetAsync(w.flags, 0, sizeof(int) * (size_t)((n + 1) * (int64_t)batch + 1), s));
#define AVS_BAND_CASE(BB, TT)                                                                                   \
    if (bw == BB && tbw == TT)                                                                                  \
        return launch_band_stage<BB, TT, R, band_cluster<BB, R>()>(dAB, n, ldab, w, s, num_sms, batch, sAB, sDone);
    AVS_BAND_CASE(256, 32)
    AVS_BAND_CASE(256, 16)
    AVS_BAND_CASE(128, 32)
    AVS_BAND_CASE(128, 16)
    AVS_BAND_CASE(64, 16)
#undef AVS_BAND_CASE
    return AVS_ERR_UNSUPPORTED;
}
template int band_stage<float>(float *, int64_t, int, int, int64_t, const Stage2Work &, cudaStream_t, int, int,
                               int64_t, int64_t);
template int band_stage<double>(double *, int64_t, int, int, int64_t, const Stage2Work &, cudaStream_t, int, int,
                                int64_t, int64_t);
template int band_stage<dfx>(dfx *, int64_t, int, int, int64_t, const Stage2Work &, cudaStream_t, int, int, int64_t,
                             int64_t);

bool band_stage_supported(int bw, int tbw) {
    return ((bw == 256 || bw == 128) && (tbw == 32 || tbw == 16)) || (bw == 64 && tbw == 16);
}

template <typename TI, typename R>
int dense_to_band(const TI *dA, int64_t n, int64_t lda, int64_t sA, int bw, R *dAB, int64_t ldab, int64_t sAB,
                  int batch, const int *scale, cudaStream_t s) {
    if (n <= 0) return AVS_SUCCESS;
    dense_to_band_kernel<TI, R><<<dim3((unsigned)n, (unsigned)batch), 128, 0, s>>>(dA, n, lda, sA, bw, dAB, ldab, sAB,
                                                                                  scale);
    AVS_CUDA_TRY(cudaGetLastError());
    return AVS_SUCCESS;
}
template int dense_to_band<float, float>(const float *, int64_t, int64_t, int64_t, int, float *, int64_t, int64_t,
                                         int, const int *, cudaStream_t);
template int dense_to_band<double, double>(const double *, int64_t, int64_t, int64_t, int, double *, int64_t,
                                           int64_t, int, const int *, cudaStream_t);
template int dense_to_band<double, dfx>(const double *, int64_t, int64_t, int64_t, int, dfx *, int64_t, int64_t, int,
                                        const int *, cudaStream_t);

template <typename R, typename St>
int band_to_band(const R *dAB1, int64_t n, int bw1, int64_t ldab1, int64_t sAB1, int bw2, St *dAB2, int64_t ldab2,
                 int64_t sAB2, int batch, cudaStream_t s) {
    if (n <= 0) return AVS_SUCCESS;
    band_to_band_kernel<R, St><<<dim3((unsigned)n, (unsigned)batch), 128, 0, s>>>(dAB1, n, bw1, ldab1, sAB1, bw2,
                                                                                 dAB2, ldab2, sAB2);
    AVS_CUDA_TRY(cudaGetLastError());
    return AVS_SUCCESS;
}
template int band_to_band<float, float2>(const float *, int64_t, int, int64_t, int64_t, int, float2 *, int64_t,
                                         int64_t, int, cudaStream_t);
template int band_to_band<double, double>(const double *, int64_t, int, int64_t, int64_t, int, double *, int64_t,
                                          int64_t, int, cudaStream_t);
template int band_to_band<dfx, float2>(const dfx *, int64_t, int, int64_t, int64_t, int, float2 *, int64_t, int64_t,
                                       int, cudaStream_t);

template <typename R>
int band_to_dense(const R *dAB, int64_t n, int bw, int64_t ldab, R *dA, int64_t lda, const int *scale,
                  cudaStream_t s) {
    if (n <= 0) return AVS_SUCCESS;
    band_to_dense_kernel<R><<<(unsigned)n, 256, 0, s>>>(dAB, n, bw, ldab, dA, lda, scale);
    AVS_CUDA_TRY(cudaGetLastError());
    return AVS_SUCCESS;
}
template int band_to_dense<float>(const float *, int64_t, int, int64_t, float *, int64_t, const int *,
                                  cudaStream_t);
template int band_to_dense<double>(const double *, int64_t, int, int64_t, double *, int64_t, const int *,
                                   cudaStream_t);

}  // namespace avs
