// Host versions of the device intrinsics that the arithmetic headers (df64.cuh,
// reflect.cuh) use, so that their source runs on the CPU.  Compile with
// -ffp-contract=off.  The hardware's estimates are approximated by the value with a
// relative error of up to 2^-21.5 drawn from the argument's bits.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>
#include <cuda_runtime.h>

static inline unsigned __float_as_uint(float f) { unsigned u; std::memcpy(&u, &f, 4); return u; }
static inline float __uint_as_float(unsigned u) { float f; std::memcpy(&f, &u, 4); return f; }
static inline int __float_as_int(float f) { return (int)__float_as_uint(f); }
static inline uint64_t bits_of(double d) { uint64_t u; std::memcpy(&u, &d, 8); return u; }
static inline int __double2hiint(double d) { return (int)(bits_of(d) >> 32); }
static inline int __double2loint(double d) { return (int)bits_of(d); }
static inline double __hiloint2double(int hi, int lo) {
    const uint64_t u = ((uint64_t)(unsigned)hi << 32) | (unsigned)lo;
    double d;
    std::memcpy(&d, &u, 8);
    return d;
}
static inline unsigned __funnelshift_r(unsigned lo, unsigned hi, unsigned s) {
    return (unsigned)(((((uint64_t)hi) << 32) | lo) >> (s & 31));
}
static inline int __float2int_rn(float f) { return (int)std::nearbyint(f); }
static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __fmaf_rn(float a, float b, float c) { return std::fmaf(a, b, c); }
static inline float __fsqrt_rn(float a) { return std::sqrt(a); }
static inline float __fdiv_rn(float a, float b) { return a / b; }
static inline float __frcp_rn(float a) { return 1.0f / a; }

static inline float estimate(double exact, float arg) {
    const uint32_t h = __float_as_uint(arg) * 2654435761u;
    return (float)(exact * (1.0 + ((double)h / 2147483648.0 - 1.0) * 0x1p-21 * 0.7071));
}
static inline float rsqrtf(float x) { return estimate(1.0 / std::sqrt((double)x), x); }
static inline float __fdividef(float a, float b) { return estimate((double)a / (double)b, b); }
