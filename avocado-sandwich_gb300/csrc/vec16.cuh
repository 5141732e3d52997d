// 16-byte vectors of the kernels' element types: VN values of T from / to shared
// or global memory (16-byte aligned).
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
}  // namespace avs
