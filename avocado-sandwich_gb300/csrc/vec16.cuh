// Element types of the stage-1 kernels: 16-byte vectors (VN values of T from / to
// shared or global memory, 16-byte aligned) and sums of products.
#pragma once

#include <cuda_runtime.h>

#include "df64.cuh"

namespace avs {

template <typename T>
struct PVec;
template <>
struct PVec<float> {
    static constexpr int VN = 4;
    static __device__ __forceinline__ void ld(const float *p, float *v) {
        const float4 x = *reinterpret_cast<const float4 *>(p);
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    }
    static __device__ __forceinline__ void ldcg(const float *p, float *v) {
        const float4 x = __ldcg(reinterpret_cast<const float4 *>(p));
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    }
    static __device__ __forceinline__ void st(float *p, const float *v) {
        *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
    }
};
template <>
struct PVec<double> {
    static constexpr int VN = 2;
    static __device__ __forceinline__ void ld(const double *p, double *v) {
        const double2 x = *reinterpret_cast<const double2 *>(p);
        v[0] = x.x; v[1] = x.y;
    }
    static __device__ __forceinline__ void ldcg(const double *p, double *v) {
        const double2 x = __ldcg(reinterpret_cast<const double2 *>(p));
        v[0] = x.x; v[1] = x.y;
    }
    static __device__ __forceinline__ void st(double *p, const double *v) {
        *reinterpret_cast<double2 *>(p) = make_double2(v[0], v[1]);
    }
};
template <>
struct PVec<dfx> {
    static constexpr int VN = 2;
    static __device__ __forceinline__ void ld(const dfx *p, dfx *v) {
        const float4 x = *reinterpret_cast<const float4 *>(p);
        v[0] = dfx(df64{x.x, x.y}); v[1] = dfx(df64{x.z, x.w});
    }
    static __device__ __forceinline__ void st(dfx *p, const dfx *v) {
        *reinterpret_cast<float4 *>(p) = make_float4(v[0].v.hi, v[0].v.lo, v[1].v.hi, v[1].v.lo);
    }
};
// Sums of products: mac accumulates into Mac (double-float: the compensated dot
// product of Ogita, Rump and Oishi, an unnormalised pair), fin gives the value.
template <typename CT>
struct MacAr;
template <>
struct MacAr<float> {
    using Mac = float;
    static __device__ __forceinline__ Mac mac0() { return 0.0f; }
    static __device__ __forceinline__ Mac mac_from(float x) { return x; }
    static __device__ __forceinline__ void mac(Mac &a, float x, float y) { a = fmaf(x, y, a); }
    static __device__ __forceinline__ Mac mac_merge(Mac a, Mac b) { return a + b; }
    static __device__ __forceinline__ float fin(Mac a) { return a; }
};
template <>
struct MacAr<dfx> {
    using Mac = df64;
    static __device__ __forceinline__ Mac mac0() { return df64{0.0f, 0.0f}; }
    static __device__ __forceinline__ Mac mac_from(dfx x) { return x.v; }
    static __device__ __forceinline__ void mac(Mac &a, dfx x, dfx y) {
        const float p = __fmul_rn(x.v.hi, y.v.hi);
        float ep = __fmaf_rn(x.v.hi, y.v.hi, -p);
        ep = __fmaf_rn(x.v.hi, y.v.lo, ep);
        ep = __fmaf_rn(x.v.lo, y.v.hi, ep);
        const df64 t = two_sum(a.hi, p);
        a.hi = t.hi;
        a.lo = __fadd_rn(a.lo, __fadd_rn(t.lo, ep));
    }
    static __device__ __forceinline__ Mac mac_merge(Mac a, Mac b) {
        const df64 t = two_sum(a.hi, b.hi);
        return df64{t.hi, __fadd_rn(t.lo, __fadd_rn(a.lo, b.lo))};
    }
    static __device__ __forceinline__ dfx fin(Mac a) { return dfx(two_sum(a.hi, a.lo)); }
};
template <>
struct MacAr<double> {
    using Mac = double;
    static __device__ __forceinline__ Mac mac0() { return 0.0; }
    static __device__ __forceinline__ Mac mac_from(double x) { return x; }
    static __device__ __forceinline__ void mac(Mac &a, double x, double y) { a = fma(x, y, a); }
    static __device__ __forceinline__ Mac mac_merge(Mac a, Mac b) { return a + b; }
    static __device__ __forceinline__ double fin(Mac a) { return a; }
};

}  // namespace avs
