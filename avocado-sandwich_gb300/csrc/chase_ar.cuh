// Scalar arithmetic of the bulge chases (stage2_chase.cu, stage2_window.cu):
// FP64, or double-float pairs stored as float2 (df64.cuh).
#pragma once

#include <cuda_runtime.h>

#include "df64.cuh"
#include "reflect.cuh"

namespace avs {

// Scalar arithmetic of the chase: FP64, or double-float pairs stored as float2.
template <typename S>
struct ChaseAr;

template <>
struct ChaseAr<double> {
    using V = double;   // register value
    using St = double;  // storage element
    static __device__ __forceinline__ V zero() { return 0.0; }
    static __device__ __forceinline__ V one() { return 1.0; }
    static __device__ __forceinline__ V ld(const St *p) { return __ldcg(p); }
    static __device__ __forceinline__ V lds(const St *p) { return *p; }  // plain (shared memory) load
    static __device__ __forceinline__ void st(St *p, V v) { *p = v; }
    static __device__ __forceinline__ V add(V a, V b) { return a + b; }
    static __device__ __forceinline__ V sub(V a, V b) { return a - b; }
    static __device__ __forceinline__ V mul(V a, V b) { return a * b; }
    static __device__ __forceinline__ V fma(V a, V b, V c) { return ::fma(a, b, c); }
    static __device__ __forceinline__ V neg(V a) { return -a; }
    static __device__ __forceinline__ bool ge0(V a) { return a >= 0.0; }
    static __device__ __forceinline__ bool iszero(V a) { return a == 0.0; }
    static __device__ __forceinline__ V shfl(V a, int src) { return __shfl_sync(0xffffffffu, a, src); }
    static __device__ __forceinline__ St from_double(double a) { return a; }
    static __device__ __forceinline__ V v_from_double(double a) { return a; }
    // dot-product accumulator: plain FMA chain
    using Acc = double;
    static __device__ __forceinline__ Acc acc_zero() { return 0.0; }
    static __device__ __forceinline__ void acc_add(Acc &a, V x, V y) { a = ::fma(x, y, a); }
    static __device__ __forceinline__ V acc_value(Acc a) { return a; }
};

template <>
struct ChaseAr<df64> {
    using V = df64;
    using St = float2;
    static __device__ __forceinline__ V zero() { return df64{0.0f, 0.0f}; }
    static __device__ __forceinline__ V one() { return df64{1.0f, 0.0f}; }
    static __device__ __forceinline__ V ld(const St *p) {
        const float2 v = __ldcg(p);
        return df64{v.x, v.y};
    }
    static __device__ __forceinline__ V lds(const St *p) {
        const float2 v = *p;
        return df64{v.x, v.y};
    }
    static __device__ __forceinline__ void st(St *p, V v) { *p = make_float2(v.hi, v.lo); }
    static __device__ __forceinline__ V add(V a, V b) { return df_add(a, b); }
    static __device__ __forceinline__ V sub(V a, V b) { return df_sub(a, b); }
    static __device__ __forceinline__ V mul(V a, V b) { return df_mul(a, b); }
    static __device__ __forceinline__ V fma(V a, V b, V c) { return df_add(df_mul(a, b), c); }
    static __device__ __forceinline__ V neg(V a) { return df_neg(a); }
    static __device__ __forceinline__ bool ge0(V a) { return !df_lt0(a); }
    static __device__ __forceinline__ bool iszero(V a) { return a.hi == 0.0f && a.lo == 0.0f; }
    static __device__ __forceinline__ V shfl(V a, int src) {
        return df64{__shfl_sync(0xffffffffu, a.hi, src), __shfl_sync(0xffffffffu, a.lo, src)};
    }
    // Dot-product accumulator in compensated FP32 (Ogita, Rump & Oishi,
    // "Accurate sum and dot product", SIAM J. Sci. Comput. 26 (2005), Dot2):
    // s carries the running FP32 sum, c the exact rounding errors of the sums
    // and of the double-float products; the loop-carried chain is one add.
    struct Acc {
        float s, c;
    };
    static __device__ __forceinline__ Acc acc_zero() { return Acc{0.0f, 0.0f}; }
    static __device__ __forceinline__ void acc_add(Acc &a, V x, V y) {
        const float p = __fmul_rn(x.hi, y.hi);
        float ep = __fmaf_rn(x.hi, y.hi, -p);
        ep = __fmaf_rn(x.hi, y.lo, ep);
        ep = __fmaf_rn(x.lo, y.hi, ep);
        const float t = __fadd_rn(a.s, p);
        const float z = __fsub_rn(t, a.s);
        const float es = __fadd_rn(__fsub_rn(a.s, __fsub_rn(t, z)), __fsub_rn(p, z));
        a.s = t;
        a.c = __fadd_rn(a.c, __fadd_rn(es, ep));
    }
    static __device__ __forceinline__ V acc_value(Acc a) { return two_sum(a.s, a.c); }
    static __device__ __forceinline__ St from_double(double a) {
        const df64 v = df_from_double(a);
        return make_float2(v.hi, v.lo);
    }
    static __device__ __forceinline__ V v_from_double(double a) { return df_from_double(a); }
};

// The reflectors' arithmetic beyond ChaseAr: merging dot-product accumulators
// without renormalising between the levels of a butterfly, the squared norm, and
// a - w u with one renormalisation.
template <typename S>
struct ChaseRefl;
template <>
struct ChaseRefl<df64> {
    using Acc = ChaseAr<df64>::Acc;
    static __device__ __forceinline__ Acc merge_xor(Acc a, int o) {
        const df64 t = two_sum(a.s, __shfl_xor_sync(0xffffffffu, a.s, o));
        return Acc{t.hi, __fadd_rn(t.lo, __fadd_rn(a.c, __shfl_xor_sync(0xffffffffu, a.c, o)))};
    }
    static __device__ __forceinline__ bool positive(Acc s) {
        const df64 v = two_sum(s.s, s.c);
        return v.hi > 0.0f;
    }
    // s + alpha^2
    static __device__ __forceinline__ df64 norm2(Acc s, df64 al) {
        const float p = __fmul_rn(al.hi, al.hi);
        const float e = __fmaf_rn(2.0f * al.hi, al.lo, __fmaf_rn(al.hi, al.hi, -p));
        const df64 t = two_sum(p, s.s);
        return fast_two_sum(t.hi, __fadd_rn(t.lo, __fadd_rn(e, s.c)));
    }
    static __device__ __forceinline__ df64 sub_mul(df64 a, df64 w, df64 u) {
        const float p = __fmul_rn(w.hi, u.hi);
        const float e = __fmaf_rn(w.lo, u.hi, __fmaf_rn(w.hi, u.lo, __fmaf_rn(w.hi, u.hi, -p)));
        const df64 t = two_sum(a.hi, -p);
        return fast_two_sum(t.hi, __fadd_rn(t.lo, __fsub_rn(a.lo, e)));
    }
};
template <>
struct ChaseRefl<double> {
    using Acc = double;
    static __device__ __forceinline__ Acc merge_xor(Acc a, int o) { return a + __shfl_xor_sync(0xffffffffu, a, o); }
    static __device__ __forceinline__ bool positive(Acc s) { return s > 0.0; }
    static __device__ __forceinline__ double norm2(Acc s, double al) { return ::fma(al, al, s); }
    static __device__ __forceinline__ double sub_mul(double a, double w, double u) { return ::fma(-w, u, a); }
};

__device__ __forceinline__ double st_to_double(double v) { return v; }
__device__ __forceinline__ double st_to_double(float2 v) { return (double)v.x + (double)v.y; }

}  // namespace avs
