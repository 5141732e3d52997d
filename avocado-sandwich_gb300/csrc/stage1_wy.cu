// Stage 1, trailing update with the full compact-WY factor of each tile
// (tiles of 128 and 256).
//
// The reflectors a panel role generated for its tile (GEQRT: b - 1 of them,
// TSQRT: b) are applied to the trailing columns as one block reflector
// Q_p = I - Y_p T_p Y_p^T, in the reference's order (GEQRT first, then the
// TSQRT tiles top to bottom, TiledMatrix.jl:107-113 / QRkernels.jl:131-197):
//
//   GEQRT tile:  Z = Y0^T Top,          W = T0^T Z,  Top -= Y0 W
//   TSQRT tile:  Z = Top + V_p^T A_p,   W = T_p^T Z, Top -= W, A_p -= V_p W
//
// The T build forms T_p (b x b, upper triangular) from the 16 x 16 diagonal blocks
// the panel kernel produced and the Gram matrix G = Y_p^T Y_p: by doubling
// (gram_kernel, tdouble_kernel), or column block by column block, T[0:c0, J] =
// -T[0:c0, 0:c0] G[0:c0, J] T_JJ (tbuild_kernel: 8-byte tiles of 256).
//
// update_full_kernel: one CTA per (tile, column strip).  Only W and the strip of
// the top tile row pass from tile to tile (W_p needs Top after tile p-1), so
// V_p^T A_p runs as soon as the CTA starts, then the CTA waits for the previous
// tile's release of the strip, forms W, hands the strip on and updates its own
// tile.  CTAs take (tile, strip) pairs in tile-major order from a ticket, so a
// CTA only waits on one that already runs.  What bounded it with one CTA per strip
// looping over the tiles: the strips were the launch's only parallelism (64
// columns each, 2 to 62 CTAs on 152 SMs at n = 4096) and every tile's three
// products ran in sequence; then the chain of W through the tiles (two CTAs on an SM
// instead of one gained nothing, warps stood at the barrier behind the wait).  So W
// runs by row blocks of 32: T is upper triangular, a block of W needs the top strip's
// rows up to that block only, and each block has its own counter and is handed on as
// soon as it is made, so the blocks of a strip pipeline through the tiles; T's block is
// loaded before the wait.  Two CTAs (16-column FP64 strips: three) share an SM.
// Measured (GB300, all updates of a call: one CTA per strip -> CTA per tile and strip
// -> row blocks): FP32 n = 4096 tile 128 45.8 -> 20.2 -> 12 ms, double-float n = 2048
// tile 128 34.5 -> 18.6 -> 11 ms (24.0 before the integer conversions).
// The two products with V are register-blocked GEMMs (8 rows x CB columns per
// thread, K = b streamed through shared memory in chunks that the next chunk's
// loads overlap).  FP64 tiles use 16-column strips when 32-column strips would leave
// SMs idle; in double-float the products accumulate with the compensated dot
// product.
#include <algorithm>
#include <type_traits>

#include "avs_common.cuh"
#include "df64.cuh"
#include "tblk.cuh"
#include "vec16.cuh"

namespace avs {
namespace {

constexpr int kWIB = 16;     // diagonal block size of T (the panel's compact-WY blocks)
constexpr int kWNT = 256;    // threads per CTA

template <typename T>
struct WCfg {
    static constexpr int W = upd_strip(sizeof(T), false);  // strip width
    static constexpr int KC = sizeof(T) == 8 ? 8 : 16;   // K chunk
};

// Memory type <-> compute type (all warps convert here: double-float on the integer pipe).
template <typename CT, typename T>
__device__ __forceinline__ CT to_ct(T v) {
    if constexpr (std::is_same<CT, dfx>::value) return dfx(df_from_double_int(v));
    else return CT(v);
}
template <typename T, typename CT>
__device__ __forceinline__ T from_ct(CT v) {
    if constexpr (std::is_same<CT, dfx>::value) return df_to_double_int(v.v);
    else return (T)v;
}

struct TBuildArgs {
    const void *a;
    int64_t lda;
    int b;
    int pr, pc, P;
    const void *tblk;  // [P][b/16][256]
    void *tfull;       // [P][b*b], T(l, i) at l + i*b
    int64_t sA, sTblk, sTfull;  // per-matrix strides (blockIdx.y = matrix)
    int first_role;    // tiles first_role..P-1 (1: the top tile's T was built earlier)
};

// ---------------------------------------------------------------------------
// T build of 8-byte tiles of 256 from the Gram matrix that gram_kernel left in tfull's
// upper triangle.  One CTA per tile: b/16 - 1 dependent column blocks (with the Gram
// matrix on the same CTA too: FP64 QR n = 1024 43.1 -> 37.2 ms, FP64X2 n = 2048 133 -> 112).
template <typename T, typename CT = T>
__global__ void __launch_bounds__(kWNT) tbuild_kernel(TBuildArgs args) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int b = args.b;
    const int nb = b / kWIB;
    const int p = blockIdx.x + args.first_role;
    const int64_t zb = blockIdx.y;
    const int tid = threadIdx.x;
    T *Tf = reinterpret_cast<T *>(args.tfull) + zb * args.sTfull + (size_t)p * b * b;
    const T *tb = reinterpret_cast<const T *>(args.tblk) + zb * args.sTblk + (size_t)p * nb * kWIB * kWIB;

    // ---- diagonal blocks and zeros below them; first column block
    for (int idx = tid; idx < b * b; idx += kWNT) {
        const int l = idx % b, i = idx / b;
        const int bl = l / kWIB, bi = i / kWIB;
        if (bl == bi) Tf[l + (size_t)i * b] = tb[(size_t)bi * kWIB * kWIB + (l % kWIB) + (i % kWIB) * kWIB];
        else if (bl > bi) Tf[l + (size_t)i * b] = T(0);
    }
    __syncthreads();
    // ---- column blocks J = 1..nb-1: CT[0:c0, J] = -CT[0:c0,0:c0] G[0:c0, J] T_JJ.
    // G's block (in Tf's column block J) and T_JJ are staged in shared memory;
    // thread r owns row r: 16 accumulators over m (CT upper triangular, zeros
    // below the diagonal), one coalesced load of CT(r, m) per m, then the 16 x 16
    // product with T_JJ in registers.
    CT *Gs = reinterpret_cast<CT *>(smem_raw);  // c0 x kWIB, Gs[m * kWIB + q]
    CT *TJ = Gs + b * kWIB;      // kWIB x kWIB, TJ[qq + q * kWIB]
    for (int J = 1; J < nb; ++J) {
        const int c0 = J * kWIB;
        for (int idx = tid; idx < c0 * kWIB; idx += kWNT) {
            const int m = idx % c0, q = idx / c0;
            Gs[m * kWIB + q] = CT(Tf[m + (size_t)(c0 + q) * b]);
        }
        for (int idx = tid; idx < kWIB * kWIB; idx += kWNT) TJ[idx] = CT(tb[(size_t)J * kWIB * kWIB + idx]);
        __syncthreads();
        const int r = tid;
        if (r < c0) {
            CT acc[kWIB];
#pragma unroll
            for (int q = 0; q < kWIB; ++q) acc[q] = CT(0);
#pragma unroll 8
            for (int m = 0; m < c0; ++m) {
                const CT t = CT(Tf[r + (size_t)m * b]);
#pragma unroll
                for (int q = 0; q < kWIB; ++q) acc[q] += t * Gs[m * kWIB + q];
            }
#pragma unroll
            for (int q = 0; q < kWIB; ++q) {
                CT v = CT(0);
#pragma unroll
                for (int qq = 0; qq < kWIB; ++qq) v += acc[qq] * TJ[qq + q * kWIB];
                Tf[r + (size_t)(c0 + q) * b] = (T)(-v);
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// T build by doubling (FP32 tiles of 128 and 256, FP64 and double-float tiles of
// 128).  gram_kernel forms the Gram matrix's 64 x 64 tiles on or above the diagonal,
// one CTA each, into the upper triangle of tfull; tdouble_kernel, one CTA per tile,
// starts from the 16 x 16 diagonal blocks and joins neighbours of size s = 16, 32,
// ..: T = [T1, -T1 G12 T2; 0, T2], two products per level with all pairs in
// parallel, T's upper block triangle packed in shared memory by 16-column blocks
// (column block J: rows 0 .. 16(J+1), column-major, at offset 256 J (J+1) / 2).
// What bounded the build column block by column block: b/16 - 1 dependent steps on
// one SM per tile, after a Gram matrix on the same SM.  Measured (GB300, a whole
// panel's T, before -> after): FP32 tile 256 295 -> 130 us, tile 128 61 -> 32 us;
// double-float tile 128 500 -> 150 us.
constexpr int kGT = 64;    // Gram tile
constexpr int kGK = 32;    // rows per staged chunk

template <typename T, int LAYOUT, typename CT>
__global__ void __launch_bounds__(kWNT) gram_kernel(TBuildArgs args) {
    using M = MacAr<CT>;
    constexpr int LD = kGT + 4;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    CT *sI = reinterpret_cast<CT *>(smem_raw);  // [kGK][LD]
    CT *sJ = sI + kGK * LD;
    const int b = args.b;
    int J = 0;
    while ((J + 1) * (J + 2) / 2 <= (int)blockIdx.x) ++J;
    const int I = (int)blockIdx.x - J * (J + 1) / 2;  // tile pair I <= J
    const int p = blockIdx.y + args.first_role;
    const int64_t zb = blockIdx.z;
    const bool geqrt = (p == 0);
    const int tid = threadIdx.x;
    View<const T, LAYOUT> V{reinterpret_cast<const T *>(args.a) + zb * args.sA, args.lda};
    const int64_t row0 = (int64_t)(args.pr + p) * b;
    const int64_t col0 = (int64_t)args.pc * b;
    T *Tf = reinterpret_cast<T *>(args.tfull) + zb * args.sTfull + (size_t)p * b * b;
    constexpr int PER = kGK * kGT / kWNT;
    T nI[PER], nJ[PER];
    auto fetch = [&](int k0, int m0, T (&v)[PER]) {
#pragma unroll
        for (int e = 0; e < PER; ++e) {
            const int idx = tid + e * kWNT;
            const int k = LAYOUT == 0 ? idx % kGK : idx / kGT, m = LAYOUT == 0 ? idx / kGK : idx % kGT;
            const int t = k0 + k, c = m0 + m;
            T x = __ldcg(&V(row0 + t, col0 + c));
            if (geqrt) x = (t == c) ? T(1) : (t > c ? x : T(0));
            v[e] = x;
        }
    };
    auto stage = [&](CT *s, const T (&v)[PER]) {
#pragma unroll
        for (int e = 0; e < PER; ++e) {
            const int idx = tid + e * kWNT;
            const int k = LAYOUT == 0 ? idx % kGK : idx / kGT, m = LAYOUT == 0 ? idx / kGK : idx % kGT;
            s[k * LD + m] = to_ct<CT>(v[e]);
        }
    };
    const int l0 = 4 * (tid % 16), i0 = 4 * (tid / 16);
    const CT *bJ = I == J ? sI : sJ;
    typename M::Mac g[4][4];
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y) g[x][y] = M::mac0();
    fetch(0, I * kGT, nI);
    if (I != J) fetch(0, J * kGT, nJ);
    for (int k0 = 0; k0 < b; k0 += kGK) {
        __syncthreads();
        stage(sI, nI);
        if (I != J) stage(sJ, nJ);
        __syncthreads();
        if (k0 + kGK < b) {
            fetch(k0 + kGK, I * kGT, nI);
            if (I != J) fetch(k0 + kGK, J * kGT, nJ);
        }
#pragma unroll 4
        for (int k = 0; k < kGK; ++k) {
            CT a[4], c[4];
#pragma unroll
            for (int q = 0; q < 4; q += PVec<CT>::VN) {
                PVec<CT>::ld(sI + k * LD + l0 + q, a + q);
                PVec<CT>::ld(bJ + k * LD + i0 + q, c + q);
            }
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int y = 0; y < 4; ++y) M::mac(g[x][y], a[x], c[y]);
        }
    }
#pragma unroll
    for (int y = 0; y < 4; ++y)
#pragma unroll
        for (int x = 0; x < 4; ++x)
            Tf[I * kGT + l0 + x + (size_t)(J * kGT + i0 + y) * b] = (T)M::fin(g[x][y]);
}

__host__ __device__ constexpr int tb_off(int J) { return 128 * J * (J + 1); }

template <typename CT, int B>
constexpr size_t tdouble_smem() {  // packed T, then the products G12 T2 of a level
    return sizeof(CT) * ((size_t)tb_off(B / kWIB) + (size_t)B * B / 4);
}

template <typename T, typename CT, int B>
__global__ void __launch_bounds__(kWNT) tdouble_kernel(TBuildArgs args) {
    using M = MacAr<CT>;
    constexpr int NB = B / kWIB, VN = PVec<CT>::VN;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    CT *Tp = reinterpret_cast<CT *>(smem_raw);
    CT *X = Tp + tb_off(NB);
    const int p = blockIdx.x + args.first_role;
    const int64_t zb = blockIdx.y;
    const int tid = threadIdx.x;
    T *Tf = reinterpret_cast<T *>(args.tfull) + zb * args.sTfull + (size_t)p * B * B;
    const T *tb = reinterpret_cast<const T *>(args.tblk) + zb * args.sTblk + (size_t)p * NB * kWIB * kWIB;
    auto col = [&](int i) -> CT * { return Tp + tb_off(i / kWIB) + (i % kWIB) * (kWIB * (i / kWIB + 1)); };
    // the Gram blocks above the diagonal blocks, and the diagonal blocks of T
    for (int idx = tid; idx < B * B; idx += kWNT) {
        const int r = idx % B, i = idx / B;
        if (r / kWIB < i / kWIB) col(i)[r] = to_ct<CT>(__ldcg(Tf + r + (size_t)i * B));
    }
    for (int idx = tid; idx < NB * kWIB * kWIB; idx += kWNT) {
        const int J = idx / (kWIB * kWIB), e = idx % (kWIB * kWIB);
        col(J * kWIB + e / kWIB)[J * kWIB + e % kWIB] = to_ct<CT>(tb[idx]);
    }
    __syncthreads();
#pragma unroll 1
    for (int s = kWIB; s < B; s *= 2) {
        const int per = (s / 4) * (s / 4);  // 4 x 4 tiles of a pair
        const int tasks = B / (2 * s) * per;
        for (int u = tid; u < tasks; u += kWNT) {  // X = G12 T2 (T2 upper triangular)
            const int q = u / per, r = 4 * (u % per % (s / 4)), c = 4 * (u % per / (s / 4));
            const int r1 = q * 2 * s, r2 = r1 + s;
            typename M::Mac a[4][4];
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int y = 0; y < 4; ++y) a[x][y] = M::mac0();
            const CT *t0 = col(r2 + c) + r2, *t1 = col(r2 + c + 1) + r2, *t2 = col(r2 + c + 2) + r2,
                     *t3 = col(r2 + c + 3) + r2;
            const int mend = c / kWIB * kWIB + kWIB;
#pragma unroll 2
            for (int m = 0; m < mend; ++m) {
                CT g[4];
                const CT *gp = col(r2 + m) + r1 + r;
#pragma unroll
                for (int e = 0; e < 4; e += VN) PVec<CT>::ld(gp + e, g + e);
                const CT tv[4] = {t0[m], t1[m], t2[m], t3[m]};
#pragma unroll
                for (int x = 0; x < 4; ++x)
#pragma unroll
                    for (int y = 0; y < 4; ++y) M::mac(a[x][y], g[x], tv[y]);
            }
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int y = 0; y < 4; y += VN) {
                    CT v[VN];
#pragma unroll
                    for (int e = 0; e < VN; ++e) v[e] = M::fin(a[x][y + e]);
                    PVec<CT>::st(X + (size_t)(q * s + r + x) * s + c + y, v);
                }
        }
        __syncthreads();
        for (int u = tid; u < tasks; u += kWNT) {  // T12 = -T1 X (T1 upper triangular)
            const int q = u / per, r = 4 * (u % per % (s / 4)), c = 4 * (u % per / (s / 4));
            const int r1 = q * 2 * s, r2 = r1 + s;
            typename M::Mac a[4][4];
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int y = 0; y < 4; ++y) a[x][y] = M::mac0();
#pragma unroll 2
            for (int m = r / kWIB * kWIB; m < s; ++m) {
                CT t[4], xv[4];
                const CT *tp = col(r1 + m) + r1 + r;
                const CT *xp = X + (size_t)(q * s + m) * s + c;
#pragma unroll
                for (int e = 0; e < 4; e += VN) {
                    PVec<CT>::ld(tp + e, t + e);
                    PVec<CT>::ld(xp + e, xv + e);
                }
#pragma unroll
                for (int x = 0; x < 4; ++x)
#pragma unroll
                    for (int y = 0; y < 4; ++y) M::mac(a[x][y], t[x], xv[y]);
            }
#pragma unroll
            for (int y = 0; y < 4; ++y) {
                CT *dst = col(r2 + c + y) + r1 + r;
#pragma unroll
                for (int x = 0; x < 4; x += VN) {
                    CT v[VN];
#pragma unroll
                    for (int e = 0; e < VN; ++e) v[e] = -M::fin(a[x + e][y]);
                    PVec<CT>::st(dst + x, v);
                }
            }
        }
        __syncthreads();
    }
    // out, zeros below the diagonal blocks
    for (int idx = tid; idx < B * B; idx += kWNT) {
        const int r = idx % B, i = idx / B;
        Tf[idx] = (r < kWIB * (i / kWIB + 1)) ? from_ct<T>(col(i)[r]) : T(0);
    }
}

// ---------------------------------------------------------------------------
// Trailing update with full T.
struct UpdFullArgs {
    void *a;
    int64_t lda;
    int64_t n;
    int b;
    int pr, pc, P;
    const void *tfull;
    int64_t sA, sTfull;  // per-matrix strides (blockIdx.y = matrix)
    int first_role;      // 1: the top tile's own reflectors were applied earlier
    int nstrip;
    int *flags;          // [0] ticket, then a counter per row block of each strip: tiles finished with it; zeroed
    int64_t sFlags;      // ints between matrices
    int *err;
};

// A-operand sources of the products with V.
enum ASrc { kVrows = 0, kVcols = 1 };

template <typename T, int B, int WW = WCfg<T>::W>
struct UCfg {
    static constexpr int W = WW;
    static constexpr int KC = WCfg<T>::KC;
    static constexpr int MB = 8;                  // rows per thread
    static constexpr int TM = B / MB;             // threads along rows
    static constexpr int TC = kWNT / TM;          // threads along columns
    static constexpr int CB = W / TC;             // columns per thread
    // A thread's 8 rows are groups of VN consecutive ones, B VN / 8 apart, and the strip
    // buffers are row-major: a product's operands are 16-byte loads, 3 for 32
    // products in FP32 (12 single ones bound it by shared memory)
    static constexpr int VN = sizeof(T) == 4 ? 4 : 2;
    static constexpr int GS = B * VN / MB;        // rows between a thread's groups
    static __device__ __forceinline__ int row(int m0, int i) { return (i / VN) * GS + m0 * VN + i % VN; }
    static constexpr int LDW = W + VN;            // row stride of the strip buffers
    static constexpr int LDC = B + 4;             // leading dimension of A chunks (m)
    static constexpr int PER = KC * B / kWNT;     // chunk elements per thread
    // W = T^T Z: row blocks of KB; a thread's 8 rows are pairs, one per quarter of the tile
    static constexpr int KB = upd_row_block(sizeof(T), B);
    static constexpr int NBK = B / KB;
    static constexpr int GSC = B / 4;
    static __device__ __forceinline__ int crow(int m0, int i) { return (i / 2) * GSC + m0 * 2 + i % 2; }
    static constexpr int CHUNK = (2 * KC > KB ? 2 * KC : KB) * LDC;  // A operands staged
    // CTAs per SM (shared memory allows them; the registers are held to it)
    static constexpr int MINB = B == 128 ? (sizeof(T) == 8 && W == 16 ? 3 : 2) : (sizeof(T) == 8 && W == 16 ? 2 : 1);
    static_assert(CB >= 1 && PER >= 1, "update configuration");
};

// T: element type in memory; CT: compute type (T itself, or dfx for FP64 data
// updated in double-float arithmetic).
template <typename T, int LAYOUT, int B, int WW = WCfg<T>::W, typename CT = T>
struct UpdCtx {
    using C = UCfg<T, B, WW>;
    View<T, LAYOUT> V;
    const T *Tf;      // T of the current tile, ld B
    int64_t row0, col0;
    bool geqrt;
    // element (k, m) of the A operand for source s (chunk-relative k0 added by caller)
    __device__ __forceinline__ CT a_elem(int s, int k, int m) const {
        if (s == kVrows) {  // V(k, m): Z = V^T ...
            if (geqrt && k <= m) return (k == m) ? CT(1) : CT(0);
            return to_ct<CT>(V(row0 + k, col0 + m));
        } else {  // V(m, k): ... -= V W
            if (geqrt && m <= k) return (m == k) ? CT(1) : CT(0);
            return to_ct<CT>(V(row0 + m, col0 + k));
        }
    }
    // chunk element index -> (k, m), coalesced for the source
    __device__ __forceinline__ void map(int s, int idx, int &k, int &m) const {
        const bool kfast = (s == kVrows) == (LAYOUT == 0);
        if (kfast) { k = idx % C::KC; m = idx / C::KC; } else { m = idx % B; k = idx / B; }
    }
};

// Double-float: compensated accumulation (Dot2, Ogita-Rump-Oishi) on the pair
// (s, c) = (a.hi, a.lo): the product's error terms and the sum's rounding error go
// to c, renormalised once per product.
__device__ __forceinline__ void dot2(df64 &a, df64 x, df64 y) {
    const float pr = __fmul_rn(x.hi, y.hi);
    float ep = __fmaf_rn(x.hi, y.hi, -pr);
    ep = __fmaf_rn(x.hi, y.lo, ep);
    ep = __fmaf_rn(x.lo, y.hi, ep);
    const float t = __fadd_rn(a.hi, pr);
    const float z = __fsub_rn(t, a.hi);
    const float es = __fadd_rn(__fsub_rn(a.hi, __fsub_rn(t, z)), __fsub_rn(pr, z));
    a.hi = t;
    a.lo = __fadd_rn(a.lo, __fadd_rn(es, ep));
}

// acc (+|-)= A(k, m)^T-view ... : acc[i][j] += sign * sum_k A(k, m0+i) * Bop(k, c0+j)
template <typename T, int LAYOUT, int B, int WW = WCfg<T>::W, typename CT = T>
__device__ __forceinline__ void gemm(const UpdCtx<T, LAYOUT, B, WW, CT> &ctx, const int src,
                                     CT (&acc)[8][UCfg<T, B, WW>::CB], const CT *Bop, CT *chunk0, CT *chunk1,
                                     bool neg) {
    using C = UCfg<T, B, WW>;
    const int tid = threadIdx.x;
    const int m0 = tid % C::TM;
    const int c0 = (tid / C::TM) * C::CB;
    // rows and columns of the products at chunk row k
    auto load_av = [&](const CT *cur, int k, CT (&av)[8]) {
#pragma unroll
        for (int i = 0; i < 8; i += C::VN) PVec<CT>::ld(cur + k * C::LDC + C::row(m0, i), av + i);
    };
    auto load_bv = [&](int k, CT (&bv)[C::CB]) {
        const CT *p = Bop + k * C::LDW + c0;
        if constexpr (C::CB % C::VN == 0) {
#pragma unroll
            for (int j = 0; j < C::CB; j += C::VN) PVec<CT>::ld(p + j, bv + j);
        } else {
#pragma unroll
            for (int j = 0; j < C::CB; ++j) bv[j] = p[j];
        }
    };
    CT pre[C::PER];
    // prologue: chunk 0 into registers
#pragma unroll
    for (int e = 0; e < C::PER; ++e) {
        int k, m;
        ctx.map(src, tid + e * kWNT, k, m);
        pre[e] = ctx.a_elem(src, k, m);
    }
    CT *bufs[2] = {chunk0, chunk1};
    const int nchunk = B / C::KC;
    for (int ch = 0; ch < nchunk; ++ch) {
        CT *cur = bufs[ch & 1];
#pragma unroll
        for (int e = 0; e < C::PER; ++e) {
            int k, m;
            ctx.map(src, tid + e * kWNT, k, m);
            cur[k * C::LDC + m] = pre[e];
        }
        __syncthreads();
        if (ch + 1 < nchunk) {
            const int k0n = (ch + 1) * C::KC;
#pragma unroll
            for (int e = 0; e < C::PER; ++e) {
                int k, m;
                ctx.map(src, tid + e * kWNT, k, m);
                pre[e] = ctx.a_elem(src, k0n + k, m);
            }
        }
        const int k0 = ch * C::KC;
        if constexpr (std::is_same<CT, dfx>::value) {
            // renormalised once per call below
#pragma unroll 4
            for (int k = 0; k < C::KC; ++k) {
                CT av[8], bv[C::CB];
                load_av(cur, k, av);
                load_bv(k0 + k, bv);
#pragma unroll
                for (int j = 0; j < C::CB; ++j)
                    if (neg) bv[j] = -bv[j];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
#pragma unroll
                    for (int j = 0; j < C::CB; ++j) {
                        dot2(acc[i][j].v, av[i].v, bv[j].v);
                    }
                }
            }
            continue;
        }
#pragma unroll 4
        for (int k = 0; k < C::KC; ++k) {
            CT av[8], bv[C::CB];
            load_av(cur, k, av);
            load_bv(k0 + k, bv);
            if (neg) {
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < C::CB; ++j) acc[i][j] -= av[i] * bv[j];
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
#pragma unroll
                    for (int j = 0; j < C::CB; ++j) acc[i][j] += av[i] * bv[j];
                }
            }
        }
    }
    if constexpr (std::is_same<CT, dfx>::value) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < C::CB; ++j) acc[i][j].v = two_sum(acc[i][j].v.hi, acc[i][j].v.lo);
    }
    __syncthreads();
}

template <typename T, int LAYOUT, int B, typename CT = T, int WW = WCfg<T>::W>
__global__ void __launch_bounds__(kWNT, UCfg<T, B, WW>::MINB) update_full_kernel(UpdFullArgs args) {
    using C = UCfg<T, B, WW>;
    static_assert(sizeof(CT) == sizeof(T), "compute type of the element's size");
    constexpr int KB = C::KB, NBK = C::NBK, W = C::W;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    CT *Buf = reinterpret_cast<CT *>(smem_raw);    // B x LDW, row-major: the tile's strip
    CT *Zb = Buf + (size_t)B * C::LDW;             // B x LDW: Z, then W
    CT *ch0 = Zb + (size_t)B * C::LDW;             // KC x LDC, twice; KB x LDC for T
    CT *ch1 = ch0 + (size_t)C::KC * C::LDC;
    __shared__ int s_t, s_ok;
    const int tid = threadIdx.x;
    const int64_t zb = blockIdx.y;
    int *flags = args.flags + zb * args.sFlags;
    if (tid == 0) s_t = atomicAdd(flags, 1);
    __syncthreads();
    const int p = args.first_role + s_t / args.nstrip, strip = s_t % args.nstrip;
    if (p >= args.P) return;
    int *done = flags + 1 + strip * NBK;
    const int64_t j0 = (int64_t)(args.pc + 1) * B + (int64_t)strip * W;  // whole tiles of columns: strips are full
    View<T, LAYOUT> V{reinterpret_cast<T *>(args.a) + zb * args.sA, args.lda};
    const int64_t top0 = (int64_t)args.pr * B;
    const int m0 = tid % C::TM;
    const int c0 = (tid / C::TM) * C::CB;
    // rows [0, R) of a strip: element u of the thread (tid + u kWNT) in memory order
    auto elem = [&](int R, int idx, int &t, int &c) {
        t = LAYOUT == 0 ? idx % R : idx / W;
        c = LAYOUT == 0 ? idx / R : idx % W;
    };

    CT acc[8][C::CB];
    UpdCtx<T, LAYOUT, B, WW, CT> ctx;
    ctx.V = V;
    ctx.row0 = (int64_t)(args.pr + p) * B;
    ctx.col0 = (int64_t)args.pc * B;
    ctx.geqrt = (p == 0);
    const T *Tf = reinterpret_cast<const T *>(args.tfull) + zb * args.sTfull + (size_t)p * B * B;
    {  // the tile's strip, NL loads in flight
        constexpr int NL = 8;
        static_assert(B * W % (kWNT * NL) == 0, "strip loads");
#pragma unroll 1
        for (int base = tid; base < B * W; base += kWNT * NL) {
            T v[NL];
            int t, c;
#pragma unroll
            for (int u = 0; u < NL; ++u) {
                elem(B, base + u * kWNT, t, c);
                v[u] = __ldcg(&V(ctx.row0 + t, j0 + c));
            }
#pragma unroll
            for (int u = 0; u < NL; ++u) {
                elem(B, base + u * kWNT, t, c);
                Buf[t * C::LDW + c] = to_ct<CT>(v[u]);
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < C::CB; ++j) acc[i][j] = CT(0);
    gemm(ctx, kVrows, acc, Buf, ch0, ch1, false);   // V_p^T A_p (the top tile: Y0^T Top)
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < C::CB; ++j) {
            Zb[C::row(m0, i) * C::LDW + c0 + j] = acc[i][j];
            acc[i][j] = CT(0);
        }

    // ---- W = T^T (Z + Top), Top -= W, row block by row block: T is upper triangular,
    // so a block of W needs the top strip's rows up to that block only, and each block
    // is handed on at once
    constexpr int PT = KB * W / kWNT;   // top elements per thread and block
    constexpr int PF = KB * B / kWNT;   // T elements per thread and block
    static_assert(PT >= 1 && PF >= 1, "chain split");
#pragma unroll 1
    for (int m = 0; m < NBK; ++m) {
        T tv[PF], top[PT];
#pragma unroll
        for (int e = 0; e < PF; ++e) {  // T(k, i), k in the block, i >= m KB
            const int idx = tid + e * kWNT, k = idx % KB, i = idx / KB;
            tv[e] = i >= m * KB ? Tf[m * KB + k + (size_t)i * B] : T(0);
        }
        if (p > args.first_role) {
            if (tid == 0) s_ok = wait_geq(done + m, p - args.first_role, args.err);
            __syncthreads();
            if (!s_ok) return;
        }
        if (p > 0) {
            int t, c;
#pragma unroll
            for (int u = 0; u < PT; ++u) {
                elem(KB, tid + u * kWNT, t, c);
                top[u] = __ldcg(&V(top0 + m * KB + t, j0 + c));
            }
        }
        __syncthreads();  // Zb complete (m = 0), the previous block's T no longer read
#pragma unroll
        for (int e = 0; e < PF; ++e) {
            const int idx = tid + e * kWNT, k = idx % KB, i = idx / KB;
            ch0[k * C::LDC + i] = to_ct<CT>(tv[e]);
        }
        if (p > 0) {
            int t, c;
#pragma unroll
            for (int u = 0; u < PT; ++u) {
                elem(KB, tid + u * kWNT, t, c);
                CT &z = Zb[(m * KB + t) * C::LDW + c];
                z = z + to_ct<CT>(top[u]);
            }
        }
        __syncthreads();
        auto product = [&](auto first_c) {  // the thread's pairs from `first` on reach past the block
            constexpr int G0 = decltype(first_c)::value;
#pragma unroll 4
            for (int k = 0; k < KB; ++k) {
                CT av[8], bv[C::CB];
#pragma unroll
                for (int g = G0; g < 4; ++g) {
                    if constexpr (sizeof(CT) == 8) {
                        PVec<CT>::ld(ch0 + k * C::LDC + C::crow(m0, 2 * g), av + 2 * g);
                    } else {
                        const float2 v = *reinterpret_cast<const float2 *>(ch0 + k * C::LDC + C::crow(m0, 2 * g));
                        av[2 * g] = v.x;
                        av[2 * g + 1] = v.y;
                    }
                }
                const CT *bp = Zb + (m * KB + k) * C::LDW + c0;
                if constexpr (C::CB % C::VN == 0) {
#pragma unroll
                    for (int j = 0; j < C::CB; j += C::VN) PVec<CT>::ld(bp + j, bv + j);
                } else {
#pragma unroll
                    for (int j = 0; j < C::CB; ++j) bv[j] = bp[j];
                }
#pragma unroll
                for (int i = 2 * G0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < C::CB; ++j) {
                        if constexpr (std::is_same<CT, dfx>::value) dot2(acc[i][j].v, av[i].v, bv[j].v);
                        else acc[i][j] += av[i] * bv[j];
                    }
            }
        };
        switch (m * KB / C::GSC) {
            case 0: product(std::integral_constant<int, 0>{}); break;
            case 1: product(std::integral_constant<int, 1>{}); break;
            case 2: product(std::integral_constant<int, 2>{}); break;
            default: product(std::integral_constant<int, 3>{}); break;
        }
        __syncthreads();  // the block's Z no longer read: W in its place
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = C::crow(m0, i);
            if (r >= m * KB && r < (m + 1) * KB) {
#pragma unroll
                for (int j = 0; j < C::CB; ++j) {
                    if constexpr (std::is_same<CT, dfx>::value) acc[i][j].v = two_sum(acc[i][j].v.hi, acc[i][j].v.lo);
                    Zb[r * C::LDW + c0 + j] = acc[i][j];
                }
            }
        }
        __syncthreads();
        if (p > 0) {
            int t, c;
#pragma unroll
            for (int u = 0; u < PT; ++u) {
                elem(KB, tid + u * kWNT, t, c);
                V(top0 + m * KB + t, j0 + c) = from_ct<T>(to_ct<CT>(top[u]) - Zb[(m * KB + t) * C::LDW + c]);
            }
            __syncthreads();
            if (tid == 0) st_release(done + m, p - args.first_role + 1);
        }
    }

    // ---- A_p -= V W (the top tile: Top -= Y0 W)
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < C::CB; ++j) acc[i][j] = Buf[C::row(m0, i) * C::LDW + c0 + j];
    gemm(ctx, kVcols, acc, Zb, ch0, ch1, true);
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < C::CB; ++j) Buf[C::row(m0, i) * C::LDW + c0 + j] = acc[i][j];
    __syncthreads();
    for (int idx = tid; idx < B * W; idx += kWNT) {
        int t, c;
        elem(B, idx, t, c);
        V(ctx.row0 + t, j0 + c) = from_ct<T>(Buf[t * C::LDW + c]);
    }
    if (p == 0) {
        __syncthreads();
        if (tid < NBK) st_release(done + tid, 1);
    }
}

template <typename T, int B, int WW = WCfg<T>::W>
size_t upd_full_smem() {
    using C = UCfg<T, B, WW>;
    return sizeof(T) * (2 * (size_t)B * C::LDW + (size_t)C::CHUNK);
}

template <typename T, int LAYOUT, int B, typename CT = T, int WW = WCfg<T>::W>
int launch_upd_full(T *dA, int64_t lda, int64_t n, int pr, int pc, int P, const Stage1Work &w, cudaStream_t s,
                    int first_role) {
    using C = UCfg<T, B, WW>;
    static std::atomic<bool> attr{false};
    const size_t smem = upd_full_smem<T, B, WW>();
    if (!attr) {
        AVS_CUDA_TRY(cudaFuncSetAttribute(update_full_kernel<T, LAYOUT, B, CT, WW>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        attr = true;
    }
    const int64_t ncols = n - (int64_t)(pc + 1) * B;
    if (ncols <= 0) return AVS_SUCCESS;
    const int nstrip = (int)upd_strips(ncols, C::W);
    const int batch = w.batch > 0 ? w.batch : 1;
    // ticket and counters take the place of the panel's 16 x 16 T blocks, which the T
    // build has read; the buffer's size goes with the order (tblk_elems), not with the
    // tiles of this launch, and holds them for every order
    const int64_t sFl = w.sTblk * (int64_t)(sizeof(T) / sizeof(int));
    const size_t used = sizeof(int) * (size_t)upd_counters(ncols, B, sizeof(T), C::W);
    int *flags = reinterpret_cast<int *>(w.tblk);
    if (batch > 1) AVS_CUDA_TRY(cudaMemset2DAsync(flags, sizeof(int) * (size_t)sFl, 0, used, batch, s));
    else AVS_CUDA_TRY(cudaMemsetAsync(flags, 0, used, s));
    UpdFullArgs a{dA, lda, n, B, pr, pc, P, w.tfull, w.sA, w.sTfull, first_role, nstrip, flags, sFl, w.err};
    update_full_kernel<T, LAYOUT, B, CT, WW><<<dim3((unsigned)nstrip * (P - first_role), batch), kWNT, smem, s>>>(a);
    AVS_CUDA_TRY(cudaGetLastError());
    return AVS_SUCCESS;
}

// FP64 tiles: the update in FP64, or in double-float when the work asks for it.
// FP64 tiles: 32-column strips, or 16 when the 32-column strips (times the
// batch) would not give every SM two CTAs: a strip's tiles follow one another
// through W, which takes half as long for half the columns.  A column's values
// do not depend on the strip width (columns are independent, the sums run in
// the same order), so single and batched calls agree bit for bit.
template <typename T, int LAYOUT, int B>
int launch_upd_full_any(T *dA, int64_t lda, int64_t n, int pr, int pc, int P, const Stage1Work &w, cudaStream_t s,
                        int first_role) {
    if constexpr (sizeof(T) == 8) {
        static int sms = 0;
        if (sms == 0) {
            int dev = 0;
            AVS_CUDA_TRY(cudaGetDevice(&dev));
            AVS_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        }
        const int64_t ncols = n - (int64_t)(pc + 1) * B;
        const bool narrow = ((ncols + 31) / 32) * (int64_t)(w.batch > 0 ? w.batch : 1) < 2 * (int64_t)sms;
        if (w.df_update)
            return narrow ? launch_upd_full<T, LAYOUT, B, dfx, upd_strip(8, true)>(dA, lda, n, pr, pc, P, w, s, first_role)
                          : launch_upd_full<T, LAYOUT, B, dfx>(dA, lda, n, pr, pc, P, w, s, first_role);
        return narrow ? launch_upd_full<T, LAYOUT, B, T, upd_strip(8, true)>(dA, lda, n, pr, pc, P, w, s, first_role)
                      : launch_upd_full<T, LAYOUT, B>(dA, lda, n, pr, pc, P, w, s, first_role);
    }
    return launch_upd_full<T, LAYOUT, B>(dA, lda, n, pr, pc, P, w, s, first_role);
}

template <typename T, int LAYOUT, typename CT, int B>
int launch_tdouble(const TBuildArgs &a, int nrole, int batch, cudaStream_t s) {
    static std::atomic<bool> attr{false};
    constexpr size_t smem = tdouble_smem<CT, B>(), gsm = sizeof(CT) * 2 * kGK * (kGT + 4);
    static_assert(smem <= 227 * 1024 && gsm <= 48 * 1024, "T build shared memory");
    if (!attr) {
        AVS_CUDA_TRY(cudaFuncSetAttribute(tdouble_kernel<T, CT, B>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)smem));
        attr = true;
    }
    constexpr int NG = (B / kGT) * (B / kGT + 1) / 2;
    gram_kernel<T, LAYOUT, CT><<<dim3(NG, nrole, batch), kWNT, gsm, s>>>(a);
    AVS_CUDA_TRY(cudaGetLastError());
    tdouble_kernel<T, CT, B><<<dim3(nrole, batch), kWNT, smem, s>>>(a);
    AVS_CUDA_TRY(cudaGetLastError());
    return AVS_SUCCESS;
}

// Tiles of 128, and FP32 tiles of 256, by doubling; 8-byte tiles of 256, whose
// packed T does not fit in shared memory, column block by column block.  FP64
// tiles with the double-float updates build T in double-float too (FP64 storage;
// GB300 issues FP64 at 1/64 of the FP32 rate).
template <typename T, int LAYOUT>
int launch_tbuild(const T *dA, int64_t lda, int b, int pr, int pc, int P, const Stage1Work &w, cudaStream_t s,
                  int first_role = 0) {
    const int batch = w.batch > 0 ? w.batch : 1, nrole = P - first_role;
    TBuildArgs a{dA, lda, b, pr, pc, P, w.tblk, w.tfull, w.sA, w.sTblk, w.sTfull, first_role};
    if constexpr (sizeof(T) == 4) {
        return b == 256 ? launch_tdouble<T, LAYOUT, float, 256>(a, nrole, batch, s)
                        : launch_tdouble<T, LAYOUT, float, 128>(a, nrole, batch, s);
    } else {
        if (b == 128)
            return w.df_update ? launch_tdouble<T, LAYOUT, dfx, 128>(a, nrole, batch, s)
                               : launch_tdouble<T, LAYOUT, double, 128>(a, nrole, batch, s);
        constexpr size_t smem = sizeof(T) * (256 * kWIB + kWIB * kWIB), gsm = sizeof(T) * 2 * kGK * (kGT + 4);
        static_assert(smem <= 48 * 1024 && gsm <= 48 * 1024, "T build shared memory");
        constexpr int NG = (256 / kGT) * (256 / kGT + 1) / 2;
        if (w.df_update) {
            gram_kernel<T, LAYOUT, dfx><<<dim3(NG, nrole, batch), kWNT, gsm, s>>>(a);
            tbuild_kernel<T, dfx><<<dim3(nrole, batch), kWNT, smem, s>>>(a);
        } else {
            gram_kernel<T, LAYOUT, T><<<dim3(NG, nrole, batch), kWNT, gsm, s>>>(a);
            tbuild_kernel<T><<<dim3(nrole, batch), kWNT, smem, s>>>(a);
        }
        AVS_CUDA_TRY(cudaGetLastError());
        return AVS_SUCCESS;
    }
}

}  // namespace

// T build alone (for the tensor-core update path).
template <typename T>
int stage1_tbuild(const T *dA, int64_t lda, int b, int layout, int pr, int pc, int P, const Stage1Work &w,
                  cudaStream_t s) {
    return layout == 0 ? launch_tbuild<T, 0>(dA, lda, b, pr, pc, P, w, s)
                       : launch_tbuild<T, 1>(dA, lda, b, pr, pc, P, w, s);
}
template int stage1_tbuild<float>(const float *, int64_t, int, int, int, int, int, const Stage1Work &, cudaStream_t);
template int stage1_tbuild<double>(const double *, int64_t, int, int, int, int, int, const Stage1Work &,
                                   cudaStream_t);

// Full-T trailing update of one half-step (tiles 128 and 256), tiles
// first_role..P-1 of the panel.
template <typename T>
int stage1_update_full(T *dA, int64_t lda, int64_t n, int b, int layout, int pr, int pc, int P, const Stage1Work &w,
                       cudaStream_t s, int first_role) {
    int rc;
    if (layout == 0) {
        if ((rc = launch_tbuild<T, 0>(dA, lda, b, pr, pc, P, w, s, first_role)) != AVS_SUCCESS) return rc;
        return b == 256 ? launch_upd_full_any<T, 0, 256>(dA, lda, n, pr, pc, P, w, s, first_role)
                        : launch_upd_full_any<T, 0, 128>(dA, lda, n, pr, pc, P, w, s, first_role);
    }
    if ((rc = launch_tbuild<T, 1>(dA, lda, b, pr, pc, P, w, s, first_role)) != AVS_SUCCESS) return rc;
    return b == 256 ? launch_upd_full_any<T, 1, 256>(dA, lda, n, pr, pc, P, w, s, first_role)
                    : launch_upd_full_any<T, 1, 128>(dA, lda, n, pr, pc, P, w, s, first_role);
}

template int stage1_update_full<float>(float *, int64_t, int64_t, int, int, int, int, int, const Stage1Work &,
                                       cudaStream_t, int);

template int stage1_update_full<double>(double *, int64_t, int64_t, int, int, int, int, int, const Stage1Work &,
                                        cudaStream_t, int);

}  // namespace avs
