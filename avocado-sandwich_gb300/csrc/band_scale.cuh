// Power-of-two scaling of a band for stage 2.  The chases and the block stage sum
// products of two entries (the chase's reflectors are unscaled, so its dot products
// are as large as twice the square of a norm): with entries of 1e18 they overflow in
// FP32 and double-float, with entries of 1e-16 the second words of a double-float
// product fall below the smallest FP32 number.  So a band whose largest entry is
// outside 2^-24 .. 2^25 is scaled to 1 by a power of two as it is copied in, and d and
// e are scaled back, in FP64, as they are copied out; bands inside keep their bits.
#pragma once

#include <cuda_runtime.h>

namespace avs {

// The biased FP64 exponent of |v| (0: zero; 2047: Inf or NaN), FP32 within the powers
// of two that FP32 holds.
__device__ __forceinline__ int exponent_code(float v) {
    const int m = __float_as_int(v) & 0x7fffffff;
    if (m == 0 || m >= 0x7f800000) return m == 0 ? 0 : 2047;
    return min(max((m >> 23) - 127, -126), 126) + 1023;
}
__device__ __forceinline__ int exponent_code(double v) { return (__double2hiint(v) >> 20) & 0x7ff; }

// The exponent k of the scaling by 2^-k, from the largest code (scale: one word per
// matrix)
__device__ __forceinline__ int band_exponent(const int *scale, int64_t zb) {
    const int code = scale[zb], k = code - 1023;
    if (code == 0 || code == 2047 || abs(k) <= 24) return 0;
    return min(max(k, -1022), 1022);
}
template <typename T>
__device__ __forceinline__ T pow2(int k);
template <>
__device__ __forceinline__ float pow2<float>(int k) { return __int_as_float((127 + k) << 23); }
template <>
__device__ __forceinline__ double pow2<double>(int k) { return __hiloint2double((1023 + k) << 20, 0); }

// The largest code of the band (entries a[r + c lda], 0 <= c - r <= bw) of each matrix
// (blockIdx.y, stride sA), a thread's loads all independent.
// scale: zeroed, or one block per matrix.
template <typename T, typename I>
__global__ void __launch_bounds__(1024) band_scale_kernel(const T *a, int64_t n, int64_t lda, int64_t sA, int bw,
                                                          int *scale) {
    __shared__ int sm[32];
    const T *az = a + blockIdx.y * sA;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const I len = (I)bw + 1, total = (I)n * len;
    int m = 0;
#pragma unroll 8
    for (I idx = blockIdx.x * (I)1024 + threadIdx.x; idx < total; idx += (I)gridDim.x * 1024) {
        const I c = idx / len, i = idx - c * len;  // row c - bw + i
        if (c + i >= (I)bw) m = max(m, exponent_code(az[(int64_t)(c + i) - bw + (int64_t)c * lda]));
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if (lane == 0) sm[wid] = m;
    __syncthreads();
    if (wid == 0) {
        m = __reduce_max_sync(0xffffffffu, sm[lane]);
        if (lane == 0) {
            if (gridDim.x == 1) scale[blockIdx.y] = m;
            else atomicMax(scale + blockIdx.y, m);
        }
    }
}

}  // namespace avs
