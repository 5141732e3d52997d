// Stage 2b: element bulge chase of a narrow band (width BW = 8, 16, 32) ->
// upper bidiagonal, with G consecutive sweeps per CTA in a shared-memory
// window.
//
// The ops are those of the element chase in stage2_chase.cu (the reference's
// bidiagonalize / block_bidiagonalize! with target width 1, KAbasedSVD/src/
// bulgechasing.jl:18-40): sweep j, step m, pivot column c0 = j + 1 + m BW,
// c1 = min(c0 + BW - 1, n - 1):
//   R op: a right reflector from row rho (= j for m = 0, c0 - BW after)
//     over columns c0..c1, applied to rows rho+1..c1;
//   L op: a left reflector from column c0 over rows c0..c1, applied to
//     columns c0+1..min(c0 + 2BW - 1, n - 1).
// Op k of sweep j touches nothing that ops >= k+4 of sweep j-1 touch, and shares
// with op k+3 one element: that op's pivot (its beta), which is element BW-1 of
// op k's last row (R op) or column (L op).
//
// Layout of the work.  A CTA owns the sweeps j0 .. j0+G-1 (groups handed out
// in order by a ticket); WPS compute warps run sweep j0+i, op t - 3i at tick t,
// and all the group's data stays in a window of W columns of the band in shared
// memory (column c in slot c mod W).  A tick has two barriers of the compute
// warps: before it, and between its phases.  Phase 1 reads the pivot, forms the
// reflector and all of the dot products but elements 0 and BW-1, and writes the
// new pivot; phase 2 reads element BW-1 (which may be the pivot that the sweep
// ahead wrote in this tick's phase 1) and applies.  That is what lets
// consecutive sweeps follow each other at three ops instead of four.
// A producer warp moves the band between the window and global memory: before
// tick t it has loaded (cp.async, 16-byte chunks, L2 only) every column the tick
// touches, and it prefetches the columns of tick t+3; a publisher warp writes
// back the columns that no sweep of the group touches again (those left of the
// trailing sweep's next pivot) and publishes the boundary in retired[g] (fence,
// release), off the ticks' critical path.  The next group's producer loads a
// column only once retired[g] has passed it, so it sees every update of this
// group, and this group never touches a column again once it is retired: the
// result is the sequential chase's, whatever the timing.  Compute warps touch
// only shared memory.  Every wait is bounded (kDevTimeout).
//
// What bounds it: the latency of one op times the ops on the critical path (3
// per sweep, plus 5 to 6 and the hand-off per group); the band stays in L2 and
// shared memory.  The op's chain is kept short: the reflector is used unscaled
// (u = x with u_0 = alpha - beta; the band comes scaled, band_scale.cuh), so the dot
// products do not wait for the norm;
// the norm's butterfly merges compensated pairs without renormalising; the
// scalars come from the hardware estimates with one residual each
// (reflect.cuh); full ops that do not wrap in the window have immediate
// addresses and no predicates.  H lanes share a row (column): with H = 2 a sweep
// runs on two warps, each forming the reflector itself.
// Measured (GB300, chase alone, before: one warp per sweep, scaled reflector,
// four ops of lag, generic double-float square root and divisions): band 16,
// double-float, n = 1024 12.3 -> 5.0 ms, n = 4096 50.4 -> 21.1 ms, n = 16384
// 204 -> 93 ms; band 32, n = 256 7.6 -> 2.5 ms.
//
// Band storage in global memory: the element chase's compact form, A(r, c) at
// AB[(r - c + 2BW - 1) + c * ldab], ldab = 3 BW.
#include <algorithm>
#include <type_traits>

#include "avs_common.cuh"
#include "chase_ar.cuh"

namespace avs {
namespace {

template <int BW, int G, int H>
struct WinCfg {
    static constexpr int KU = 2 * BW - 1;
    static constexpr int LAG = 3;               // ticks between consecutive sweeps of a group
    static constexpr int LDAB = 3 * BW;         // storage rows per column (global)
    static constexpr int LDW = 3 * BW + 2;      // window column stride (16-byte multiple; odd stride - 1)
    static constexpr int W = 2 * G * BW + 2 * BW;  // window columns (span of a group's ops + prefetch)
    static constexpr int RL = 32 / H;           // rows (R op) / columns (L op) per warp, H lanes each
    static constexpr int WPS = (2 * BW - 1 + RL - 1) / RL;  // warps per sweep
    static constexpr int SEG = BW / H;          // reflector elements per lane
    static constexpr int NC = 32 * G * WPS;     // compute threads
    static constexpr int D = 4;                 // ops of the mbarrier ring (producer lookahead)
    static constexpr int NT = NC + 64;          // + the producer and the publisher warps
    static constexpr int CHUNKS = LDAB * 8 / 16;  // 16-byte chunks per column
    static_assert(BW % 2 == 0 && BW <= 32 && SEG >= 4, "window chase band");
    static_assert(WPS == 1 || 3 + G <= 16, "named barriers");
    static constexpr size_t smem_bytes() { return 8 * (size_t)W * LDW; }
};

__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void bar_sync(int id, int cnt) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(cnt) : "memory"); }

// mbarriers of the tick ring: the producer's copies arrive on them
// (cp.async.mbarrier.arrive.noinc: when all of the lane's earlier copies have
// landed), the compute warps wait on the phase of their tick
__device__ __forceinline__ void mbar_init(unsigned long long *m, unsigned cnt) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(m)), "r"(cnt) : "memory");
}
__device__ __forceinline__ void mbar_inval(unsigned long long *m) {
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_addr(m)) : "memory");
}
__device__ __forceinline__ void cp_async_mbar_arrive(unsigned long long *m) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_addr(m)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long *m, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(m)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ int ld_volatile_shared(const int *p) { return *(const volatile int *)p; }
__device__ __forceinline__ void st_volatile_shared(int *p, int v) { *(volatile int *)p = v; }
__device__ __forceinline__ int ld_acquire_shared(const int *p) {
    int v;
    asm volatile("ld.acquire.cta.shared::cta.s32 %0, [%1];" : "=r"(v) : "r"(smem_addr(p)) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_shared(int *p, int v) {
    asm volatile("st.release.cta.shared::cta.s32 [%0], %1;" ::"r"(smem_addr(p)), "r"(v) : "memory");
}
__device__ __forceinline__ int ld_relaxed(const int *p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Bounded waits of the CTA's warps on one another: kWaitCycles of the SM clock
// (4 s at 2 GHz; reading it costs a few cycles, %globaltimer hundreds) and
// kSpinLimit polls.  A wait that runs out records kDevTimeout and raises *fail,
// on which every later wait of the CTA returns at once: the group runs to its
// end on whatever data it has.
constexpr long long kWaitCycles = 8000000000ll;
__device__ __forceinline__ bool wait_over(long long it, long long t0, int *fail, int *err) {
    if (ld_volatile_shared(fail)) return true;
    if (it > kSpinLimit || clock64() - t0 > kWaitCycles) {
        atomicCAS(err, kDevOk, kDevTimeout);
        st_volatile_shared(fail, 1);
        return true;
    }
    return false;
}
// a shared-memory counter written (release) by another warp of the CTA
__device__ __forceinline__ void wait_shared_geq(const int *p, int target, int *fail, int *err) {
    if (ld_acquire_shared(p) >= target) return;
    const long long t0 = clock64();
#pragma unroll 1
    for (long long it = 0; ld_acquire_shared(p) < target; ++it) {
        if ((it & 63) == 63 && wait_over(it, t0, fail, err)) return;
        if (it > 16) __nanosleep(20);
    }
}
// a phase of an mbarrier
__device__ __forceinline__ void mbar_wait(unsigned long long *m, unsigned parity, int *fail, int *err) {
    if (mbar_try_wait(m, parity)) return;
    const long long t0 = clock64();
#pragma unroll 1
    for (long long it = 0; !mbar_try_wait(m, parity); ++it)
        if ((it & 63) == 63 && wait_over(it, t0, fail, err)) return;
}

constexpr int kAllDone = 1 << 30;

// Per-sweep op geometry.
struct WOp {
    int c0, c1, hi;  // pivot column, last column of the reflector, last column touched
};
template <int BW>
__device__ __forceinline__ int wops(int64_t n, int j) { return 2 * ((int)((n - j - 2) / BW) + 1); }
template <int BW>
__device__ __forceinline__ WOp wop(int64_t n, int j, int k) {
    WOp o;
    o.c0 = j + 1 + (k >> 1) * BW;
    const int last = (int)(n - 1);
    o.c1 = min(o.c0 + BW - 1, last);
    o.hi = min(o.c0 + ((k & 1) ? 2 * BW - 1 : BW - 1), last);
    return o;
}

template <int BW, typename S, int G, int H>
__global__ void __launch_bounds__(WinCfg<BW, G, H>::NT, 1)
    chase_win_kernel(typename ChaseAr<S>::St *ab_base, int64_t n, int batch, int64_t sAB, int *ticket,
                     int *retired_base, int64_t sRet, int *err) {
    using Cfg = WinCfg<BW, G, H>;
    using Ar = ChaseAr<S>;
    using Wa = ChaseRefl<S>;
    using V = typename Ar::V;
    using St = typename Ar::St;
    static_assert(sizeof(St) == 8 && sizeof(V) == 8, "8-byte band elements");
    constexpr int KU = Cfg::KU, LDW = Cfg::LDW, W = Cfg::W, LDAB = Cfg::LDAB, LAG = Cfg::LAG;
    constexpr int CW = G * Cfg::WPS;  // compute warps; then the producer and the publisher
    extern __shared__ __align__(16) unsigned char smem_raw[];
    St *win = reinterpret_cast<St *>(smem_raw);  // [W][LDW]
    __shared__ int s_g;
    __shared__ int s_tick, s_wb, s_fail;  // ticks finished; columns below s_wb written back; a wait ran out
    __shared__ __align__(8) unsigned long long s_full[Cfg::D];  // tick t's columns are in: phase t / D of [t % D]
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    if (tid == 0)
        for (int d = 0; d < Cfg::D; ++d) mbar_init(&s_full[d], 32);
    const int nsweeps = (int)(n - 1);
    const int ngroups = (nsweeps + G - 1) / G;

    for (;;) {
        if (tid == 0) s_g = atomicAdd(ticket, 1);
        __syncthreads();
        const int tk = s_g;
        __syncthreads();
        // tickets are group-major over the batch: every matrix advances its own wavefront
        const int g = tk / batch, zb = tk % batch;
        if (g >= ngroups) return;
        St *ab = ab_base + (size_t)zb * sAB;
        int *retired = retired_base + (size_t)zb * sRet;
        const int j0 = g * G;
        if (tid == 0) {
            s_tick = 0;
            s_wb = j0 + 1;
            s_fail = 0;
        }
        __syncthreads();
        const int gs = min(G, nsweeps - j0);
        // the leading sweep's op t touches columns below need(t); every other sweep
        // of the group is left of it, and its last op reaches column n - 1
        const int ops0 = wops<BW>(n, j0);
        int nticks = 0;
        for (int i = 0; i < gs; ++i) nticks = max(nticks, LAG * i + wops<BW>(n, j0 + i));
        auto need_of = [&](int t) -> int { return t < ops0 ? wop<BW>(n, j0, t).hi + 1 : (int)n; };

        if (wid == CW) {
            // ---------------- producer warp: global -> window ----------------
            // The copies of each of the leading sweep's ops arrive on the op's mbarrier
            // as they land; the producer runs up to D - 1 ops ahead of that sweep.  The
            // other sweeps are left of it.
            int issued = j0 + 1;               // columns below are requested (cp.async)
            int rp = (g == 0) ? (int)n : 0;    // retired[g-1] as last observed
            int rp_next = rp;                  // lane 0: a relaxed read in flight, used at the next op
            // copies of the columns [from, to) into their slots (one column per step, lanes over chunks)
            auto copy_in = [&](int from, int to) {
                int sl = from % W;
                for (int c = from; c < to; ++c) {
                    for (int h = lane; h < Cfg::CHUNKS; h += 32)
                        cp_async16(win + (size_t)sl * LDW + 2 * h, ab + (size_t)c * LDAB + 2 * h);
                    if (++sl == W) sl = 0;
                }
            };
            for (int t = 0; t < nticks; ++t) {
                const int need = need_of(t);
                if (t >= Cfg::D) {  // the ring slot of tick t is free once tick t - D is done
                    if (lane == 0) wait_shared_geq(&s_tick, t - Cfg::D + 1, &s_fail, err);
                    __syncwarp();
                }
                if (issued < need) {
                    // not prefetched (the previous group was behind): load now
                    if (rp < need) {
                        if (lane == 0 && !wait_geq(retired + g - 1, need, err)) st_volatile_shared(&s_fail, 1);
                        __syncwarp();
                        rp = max(need, __shfl_sync(0xffffffffu, lane == 0 ? ld_acquire(retired + g - 1) : 0, 0));
                    }
                    if (need > ld_volatile_shared(&s_wb) + W) {  // free slots (bounded wait on the publisher)
                        if (lane == 0) wait_shared_geq(&s_wb, need - W, &s_fail, err);
                        __syncwarp();
                    }
                    copy_in(issued, need);
                    issued = need;
                }
                cp_async_mbar_arrive(&s_full[t % Cfg::D]);  // op t: when this lane's copies so far have landed
                // lane 0's read of the previous group's boundary, issued at the last op.  The
                // copies of the columns it releases are issued only once the value has
                // arrived (their range depends on it) and read L2, where the previous
                // group's writes were made visible before its release.
                rp = max(rp, __shfl_sync(0xffffffffu, rp_next, 0));
                if (g > 0 && rp < (int)n && lane == 0) rp_next = ld_relaxed(retired + g - 1);
                // prefetch the columns of the next three ops that the previous group
                // has retired and whose slots are free
                const int tgt = min(min(need_of(t + 3), rp), min(ld_volatile_shared(&s_wb) + W, (int)n));
                if (tgt > issued) {
                    copy_in(issued, tgt);
                    issued = tgt;
                }
            }
            cp_wait_all();
        } else if (wid == CW + 1) {
            // ---------------- publisher warp: window -> global, retired[g] ----------------
            // Follows the sweeps' progress: columns left of every sweep's current op
            // are final for this group; they are written back and the boundary is
            // released for the next group.
            int wb = j0 + 1;
            long long t0 = 0;
            for (long long it = 0;;) {
                int r = (int)n;
                if (lane < gs) {  // the lowest column this sweep's current and later ops touch
                    const int k = max(ld_acquire_shared(&s_tick) - LAG * lane, 0);
                    if (k < wops<BW>(n, j0 + lane)) r = wop<BW>(n, j0 + lane, k).c0;
                }
                r = __reduce_min_sync(0xffffffffu, r);
                __syncwarp();  // what each lane acquired is visible to the copying lanes
                if (r > wb) {
                    int sl = wb % W;
                    for (int c = wb; c < r; ++c) {
                        for (int h = lane; h < Cfg::CHUNKS; h += 32) {
                            const uint4 v = *reinterpret_cast<const uint4 *>(win + (size_t)sl * LDW + 2 * h);
                            *reinterpret_cast<uint4 *>(ab + (size_t)c * LDAB + 2 * h) = v;
                        }
                        if (++sl == W) sl = 0;
                    }
                    __syncwarp();
                    wb = r;
                    if (lane == 0) {
                        st_release_shared(&s_wb, wb);  // the slots may be refilled
                        __threadfence();
                        st_release(retired + g, wb);
                    }
                    it = 0;
                    if (r >= (int)n) break;
                } else {
                    if (it == 0) t0 = clock64();
                    int over = 0;
                    if (lane == 0 && (it & 63) == 63) over = wait_over(it, t0, &s_fail, err);
                    if (__shfl_sync(0xffffffffu, over, 0)) break;
                    ++it;
                    __nanosleep(20);
                }
            }
        } else {
            // ---------------- compute warps: WPS warps run sweep j0 + sw ----------------
            constexpr int SEG = Cfg::SEG, RL = Cfg::RL, WPS = Cfg::WPS;
            const int sw = wid / WPS, sub = wid % WPS;
            const int j = j0 + sw;
            const int ops = (sw < gs) ? wops<BW>(n, j) : 0;
            const int seg = lane / RL;                 // which SEG elements of the reflector
            const int rl = sub * RL + lane % RL;       // which row (R op) / column (L op)
            for (int t = 0; t < nticks; ++t) {
                bar_sync(1, Cfg::NC);  // every compute warp is done with tick t-1
                if (tid == 0) st_release_shared(&s_tick, t);
                mbar_wait(&s_full[t % Cfg::D], (unsigned)(t / Cfg::D) & 1u, &s_fail, err);  // tick t's columns are in
                const int k = t - LAG * sw;
                const bool run = k >= 0 && k < ops;
                const WOp o = wop<BW>(n, j, max(k, 0));
                const int L = o.c1 - o.c0 + 1;
                const bool act = run && L >= 2;
                const bool rop = (k & 1) == 0;
                // element i of the pivot (row rho of an R op, column c0 of an L op)
                // and of this lane's row / column at base + i * stride; an R op's
                // columns past the window's last slot continue at slot 0
                const int s0 = o.c0 % W;
                const int iw = W - s0;
                const bool fast = (L == BW) && (!rop || iw >= BW);
                const int rho = rop ? ((k == 0) ? j : o.c0 - BW) : o.c0;
                St *piv = win + (size_t)s0 * LDW + (rho - o.c0 + KU);
                St *row = piv;
                bool valid = false;
                if (act) {
                    if (rop) {
                        valid = rho + 1 + rl <= o.c1;
                        if (valid) row = piv + 1 + rl;
                    } else {
                        const int c = o.c0 + 1 + rl;
                        valid = c <= o.hi;
                        int sl = s0 + 1 + rl;
                        sl -= (sl >= W) ? W : 0;
                        if (valid) row = win + (size_t)sl * LDW + (o.c0 - c + KU);
                    }
                }
                // The op in two phases.  Phase 1 reads the pivot, forms the scalars and
                // all of the dot product but elements 0 and BW-1; the new pivot then goes
                // to the window and is posted.  Phase 2 reads element BW-1, which op k+2
                // of the previous sweep wrote, or which is the pivot of its op k+3 (the
                // only element that ops three apart share), and applies.
                V xr[SEG], xv[SEG];
                typename Ar::Acc a = Ar::acc_zero();
                V u0 = Ar::zero(), beta = Ar::zero(), rn = Ar::zero(), inv = Ar::zero();
                bool nz = false;
                V a0 = Ar::zero(), xl = Ar::zero();
                auto phase1 = [&](auto fast_c, auto rop_c) {
                    constexpr bool FAST = decltype(fast_c)::value, ROP = decltype(rop_c)::value;
                    constexpr int STR = ROP ? LDW - 1 : 1;
                    auto off = [&](int i) -> int { return i * STR - ((!FAST && ROP && i >= iw) ? W * LDW : 0); };
                    const V alpha = Ar::lds(piv);
#pragma unroll
                    for (int q = 0; q < SEG; ++q) {
                        const int i = seg * SEG + q;
                        xr[q] = (FAST || i < L) ? Ar::lds(piv + off(i)) : Ar::zero();
                    }
                    xl = (FAST || BW - 1 < L) ? Ar::lds(piv + off(BW - 1)) : Ar::zero();
                    a0 = Ar::lds(row);
#pragma unroll
                    for (int q = 0; q < SEG; ++q) {
                        const int i = seg * SEG + q;
                        const bool inner = q > 0 || seg > 0;  // element BW-1 only in phase 2
                        xv[q] = ((FAST || i < L) && inner && (q < SEG - 1 || seg < H - 1)) ? Ar::lds(row + off(i))
                                                                                          : Ar::zero();
                    }
                    // ||x||^2 without element 0, one element per lane and a butterfly (fewer
                    // instructions than summing it in every lane: 20.7 against 21.9 ms for
                    // the chase at n = 4096), and the dot product without elements 0 and
                    // BW-1 (their xv are zero here)
                    typename Ar::Acc s = Ar::acc_zero();
                    {
                        const int il = lane % BW;
                        const V xs = (il >= 1 && (FAST || il < L)) ? Ar::lds(piv + off(il)) : Ar::zero();
                        Ar::acc_add(s, xs, xs);
                    }
#pragma unroll
                    for (int sh = BW / 2; sh >= 1; sh >>= 1) s = Wa::merge_xor(s, sh);
#pragma unroll
                    for (int q = 0; q < SEG; ++q)
                        if ((q > 0 || H > 1) && (q < SEG - 1 || H > 1)) Ar::acc_add(a, xv[q], xr[q]);
#pragma unroll
                    for (int sh = RL; sh < 32; sh <<= 1) a = Wa::merge_xor(a, sh);
                    // H = I - u u^T / (||x|| (||x|| + |alpha|)), u = x with u_0 = alpha - beta,
                    // beta = -sign(alpha) ||x||: u needs no scaling, so the dot products do
                    // not wait for the norm
                    nz = Wa::positive(s);
                    beta = alpha;
                    if (nz) {
                        V nrm;
                        rsqrt_sqrt(Wa::norm2(s, alpha), rn, nrm);
                        const bool pos = Ar::ge0(alpha);
                        const V u = Ar::add(pos ? alpha : Ar::neg(alpha), nrm);
                        u0 = pos ? u : Ar::neg(u);
                        beta = pos ? Ar::neg(nrm) : nrm;
                    }
                };
                auto put_pivot = [&](auto fast_c, auto rop_c) {
                    constexpr bool FAST = decltype(fast_c)::value, ROP = decltype(rop_c)::value;
                    constexpr int STR = ROP ? LDW - 1 : 1;
                    if (lane < (FAST ? BW : L))
                        Ar::st(piv + lane * STR - ((!FAST && ROP && lane >= iw) ? W * LDW : 0),
                               lane == 0 ? beta : Ar::zero());
                };
                auto phase2 = [&](auto fast_c, auto rop_c) {
                    constexpr bool FAST = decltype(fast_c)::value, ROP = decltype(rop_c)::value;
                    constexpr int STR = ROP ? LDW - 1 : 1;
                    auto off = [&](int i) -> int { return i * STR - ((!FAST && ROP && i >= iw) ? W * LDW : 0); };
                    const V al = (FAST || BW - 1 < L) ? Ar::lds(row + off(BW - 1)) : Ar::zero();
                    Ar::acc_add(a, al, xl);
                    const V w = Ar::mul(Ar::mul(Ar::acc_value(a), rn), inv);
                    if (seg == 0) {
                        xv[0] = a0;
                        xr[0] = u0;
                    }
                    if (seg == H - 1) xv[SEG - 1] = al;
                    if (valid) {
#pragma unroll
                        for (int q = 0; q < SEG; ++q) {
                            const int i = seg * SEG + q;
                            if (FAST || i < L) Ar::st(row + off(i), Wa::sub_mul(xv[q], w, xr[q]));
                        }
                    }
                };
                auto dispatch = [&](auto f) {
                    if (fast) {
                        if (rop) f(std::true_type{}, std::true_type{});
                        else f(std::true_type{}, std::false_type{});
                    } else {
                        if (rop) f(std::false_type{}, std::true_type{});
                        else f(std::false_type{}, std::false_type{});
                    }
                };
                if (act) dispatch(phase1);
                if (WPS > 1) bar_sync(3 + sw, 32 * WPS);  // every warp of the sweep has read the pivot
                else __syncwarp();
                if (act && sub == 0) dispatch(put_pivot);
                if (act && nz) {
                    // the rest of the scalars and element 0's term, while the previous sweep
                    // reaches the pivot of its op k+3
                    inv = rcp_est(Ar::ge0(u0) ? u0 : Ar::neg(u0));
                    Ar::acc_add(a, a0, u0);
                }
                bar_sync(2, Cfg::NC);  // the tick's new pivots are in the window
                if (act && nz) dispatch(phase2);
            }
            bar_sync(1, Cfg::NC);
            if (tid == 0) st_release_shared(&s_tick, kAllDone);
        }
        __syncthreads();
        if (tid == 0) {  // fresh phases for the next group
            for (int d = 0; d < Cfg::D; ++d) {
                mbar_inval(&s_full[d]);
                mbar_init(&s_full[d], 32);
            }
        }
    }
}

template <int BW, typename S, int G, int H>
int launch_win(typename ChaseAr<S>::St *dAB, int64_t n, const Stage2Work &w, cudaStream_t s, int num_sms, int batch,
               int64_t sAB) {
    using Cfg = WinCfg<BW, G, H>;
    const size_t smem = Cfg::smem_bytes();
    auto kern = chase_win_kernel<BW, S, G, H>;
    AVS_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, Cfg::NT, smem) != cudaSuccess || per_sm < 1) {
        cudaGetLastError();
        per_sm = 1;
    }
    const int64_t ngroups = ((n - 1) + G - 1) / G;
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(ngroups * batch, (int64_t)num_sms * per_sm));
    kern<<<grid, Cfg::NT, smem, s>>>(dAB, n, batch, sAB, w.flags, w.flags + 1, n + 1, w.err);
    AVS_CUDA_TRY(cudaGetLastError());
    return AVS_SUCCESS;
}

}  // namespace

bool chase_window_supported(int bw) { return bw == 8 || bw == 16 || bw == 32; }

// The band (width bw, compact storage with ldab = 3 bw) -> bidiagonal, in
// place.  w.flags: n + 2 ints (zeroed here).
template <typename S>
static int chase_window(typename ChaseAr<S>::St *dAB, int64_t n, int bw, const Stage2Work &w, cudaStream_t s,
                        int num_sms, int batch, int64_t sAB) {
    if (n < 2 || batch < 1) return AVS_SUCCESS;
    if (n > ((int64_t)1 << 30) || (int64_t)batch * n > ((int64_t)1 << 31) - 64) return AVS_ERR_UNSUPPORTED;
    AVS_CUDA_TRY(cudaMemsetAsync(w.flags, 0, sizeof(int) * (size_t)((n + 1) * (int64_t)batch + 1), s));
    // Sweeps per CTA (G) and lanes per row (H), swept on GB300.  Double-float, band
    // 16: more sweeps share the hand-off between groups, but the tick is issue-bound
    // once a scheduler has four warps (G = 8, H = 2), and one warp per sweep (H = 1)
    // has twice the instructions on its path: G x H = 4 x 2 21.1 ms, 8 x 1 23.3, 4 x 1
    // 24.0, 2 x 2 25.8, 8 x 2 26.1 at n = 4096; batches agree within 10% (32 matrices
    // of order 1024: 10.3 ms of stage 2, 8 x 2 10.7, 8 x 1 11.9).  FP64 is bound by
    // the FP64 unit's issue (64 cycles a warp instruction): H = 1, which repeats no
    // reflector, and few sweeps per SM (n = 512, band 16: 4 x 1 6.3 ms, 8 x 1 7.8, 4 x 2
    // 7.6; band 32: 2 x 1 11.4, 3 x 1 11.5, 3 x 2 13.9).  The values do not depend on G
    // or, with one matrix or many, on the batch.
    constexpr bool df = std::is_same<S, df64>::value;
    switch (bw) {
        case 8: return launch_win<8, S, 8, 2>(dAB, n, w, s, num_sms, batch, sAB);
        case 16: return launch_win<16, S, 4, df ? 2 : 1>(dAB, n, w, s, num_sms, batch, sAB);
        case 32: return launch_win<32, S, df ? 3 : 2, df ? 2 : 1>(dAB, n, w, s, num_sms, batch, sAB);
        default: return AVS_ERR_UNSUPPORTED;
    }
}
int stage2_chase_window_df(float2 *dAB, int64_t n, int bw, const Stage2Work &w, cudaStream_t s, int num_sms,
                           int batch, int64_t sAB) {
    return chase_window<df64>(dAB, n, bw, w, s, num_sms, batch, sAB);
}
int stage2_chase_window_fp64(double *dAB, int64_t n, int bw, const Stage2Work &w, cudaStream_t s, int num_sms,
                             int batch, int64_t sAB) {
    return chase_window<double>(dAB, n, bw, w, s, num_sms, batch, sAB);
}

}  // namespace avs
