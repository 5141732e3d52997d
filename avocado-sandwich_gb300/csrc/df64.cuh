// Double-float ("df64") arithmetic: a value is the unevaluated sum hi + lo of
// two FP32 numbers (|lo| <= ulp(hi)/2), giving ~44-48 significant bits on the
// FP32 pipe.  GB300 issues FP64 at 1/64 of the FP32 rate, so the FP64-class
// stages (bulge chase, bisection) run their inner loops in this format.
//
// Error-free transformations: TwoSum (Knuth, TAOCP vol. 2), FastTwoSum
// (Dekker 1971), TwoProduct with a fused multiply-add; the composite
// operations follow Hida, Li & Bailey, "Library for double-double and
// quad-double arithmetic" (2007), "sloppy" variants.  The exponent range is
// FP32's: callers keep their data normalised.
#pragma once

#include <cuda_runtime.h>

namespace avs {

struct df64 {
    float hi, lo;
};

__device__ __forceinline__ df64 df_from_double(double x) {
    const float h = (float)x;
    return df64{h, (float)(x - (double)h)};
}
__device__ __forceinline__ double df_to_double(df64 a) { return (double)a.hi + (double)a.lo; }
// FP64 <-> double-float on the integer pipe: hi + lo rounded as (float)x and
// (float)(x - hi), and (double)hi + (double)lo, exactly (an exact tie of hi goes up
// instead of to even; hi + lo is the same).  The FP64 instructions for them, three
// either way, issue at 64 cycles per warp on GB300: with all warps converting they took
// as long as the products of a double-float trailing update.  Some 15 instructions,
// so a loss where few warps convert (the panels: FP64 tiles of 64 n = 1024 stage 1 14.9
// -> 15.8 ms).  Exponents within [-74, 126] and zeros, and normalised pairs; anything
// else takes the FP64 instructions.
__device__ __forceinline__ df64 df_from_double_int(double x) {
    const unsigned lo32 = (unsigned)__double2loint(x), hi32 = (unsigned)__double2hiint(x);
    const unsigned ahi = hi32 & 0x7fffffffu, sgn = hi32 & 0x80000000u;
    const unsigned ex = ahi >> 20;
    if (ex - (1023u - 74u) <= 200u) {
        const unsigned rl = lo32 + 0x10000000u, rh = ahi + (rl < lo32 ? 1u : 0u);  // + half a unit of hi
        const unsigned h = __funnelshift_r(rl, rh, 29) - ((1023u - 127u) << 23);
        const int rem = (int)(lo32 - (rl & 0xe0000000u));  // in units of 2^(ex - 1023 - 52)
        const float sc = __uint_as_float((ex - (1023u - 127u) - 52u) << 23);
        return df64{__uint_as_float(h | sgn), __uint_as_float(__float_as_uint(__fmul_rn((float)rem, sc)) ^ sgn)};
    }
    if ((ahi | lo32) == 0u) return df64{0.0f, 0.0f};
    return df_from_double(x);
}
__device__ __forceinline__ double df_to_double_int(df64 a) {
    const unsigned hb = __float_as_uint(a.hi), ah = hb & 0x7fffffffu, sgn = hb & 0x80000000u;
    const unsigned ex = ah >> 23;
    if (ex - (127u - 74u) <= 200u && fabsf(a.lo) <= __fmul_rn(fabsf(a.hi), 0x1p-24f)) {
        // hi + lo in units of 2^(ex - 127 - 52), half of that just below a power of two: a
        // normalised pair (|lo| <= 2^-24 |hi|) leaves hi's binade only there
        const float sl = __uint_as_float(__float_as_uint(a.lo) ^ sgn);  // lo relative to |hi|
        const unsigned half = ((ah & 0x7fffffu) == 0u && sl < 0.0f) ? 1u : 0u;
        const float sc = __uint_as_float((52u + 127u - (ex - 127u) + half) << 23);
        const int k = __float2int_rn(__fmul_rn(sl, sc));
        const unsigned l0 = ah << 29, h0 = (ah >> 3) + ((1023u - 127u) << 20);
        const unsigned l1 = l0 + (unsigned)k;
        const unsigned h1 = h0 + (unsigned)(k >> 31) + (l1 < l0 ? 1u : 0u);
        return __hiloint2double((int)(h1 | sgn), (int)l1);
    }
    return df_to_double(a);
}

// |a| >= |b| (or a == 0): s + e == a + b exactly
__device__ __forceinline__ df64 fast_two_sum(float a, float b) {
    const float s = __fadd_rn(a, b);
    const float e = __fsub_rn(b, __fsub_rn(s, a));
    return df64{s, e};
}
__device__ __forceinline__ df64 two_sum(float a, float b) {
    const float s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
    return df64{s, e};
}
__device__ __forceinline__ df64 two_prod(float a, float b) {
    const float p = __fmul_rn(a, b);
    return df64{p, __fmaf_rn(a, b, -p)};
}

__device__ __forceinline__ df64 df_add(df64 a, df64 b) {
    df64 s = two_sum(a.hi, b.hi);
    s.lo = __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo));
    return fast_two_sum(s.hi, s.lo);
}
__device__ __forceinline__ df64 df_neg(df64 a) { return df64{-a.hi, -a.lo}; }
__device__ __forceinline__ df64 df_sub(df64 a, df64 b) { return df_add(a, df_neg(b)); }

__device__ __forceinline__ df64 df_mul(df64 a, df64 b) {
    df64 p = two_prod(a.hi, b.hi);
    p.lo = __fmaf_rn(a.hi, b.lo, p.lo);
    p.lo = __fmaf_rn(a.lo, b.hi, p.lo);
    return fast_two_sum(p.hi, p.lo);
}

__device__ __forceinline__ bool df_lt0(df64 a) { return a.hi < 0.0f || (a.hi == 0.0f && a.lo < 0.0f); }

// A double-float value with arithmetic operators: the compute type of kernels
// templated on their element type when the data is stored in FP64 (converted
// on load, ~48 of the 53 significant bits kept, FP32's exponent range; rounded
// back to FP64 on store).
struct dfx {
    df64 v;
    __device__ __forceinline__ dfx() {}
    __device__ __forceinline__ dfx(int x) : v(df64{(float)x, 0.0f}) {}
    __device__ __forceinline__ explicit dfx(double x) : v(df_from_double(x)) {}
    __device__ __forceinline__ explicit dfx(df64 x) : v(x) {}
    __device__ __forceinline__ explicit operator double() const { return df_to_double(v); }
};
__device__ __forceinline__ dfx operator+(dfx a, dfx b) { return dfx(df_add(a.v, b.v)); }
__device__ __forceinline__ dfx operator-(dfx a, dfx b) { return dfx(df_sub(a.v, b.v)); }
__device__ __forceinline__ dfx operator*(dfx a, dfx b) { return dfx(df_mul(a.v, b.v)); }
__device__ __forceinline__ dfx operator-(dfx a) { return dfx(df_neg(a.v)); }
__device__ __forceinline__ dfx &operator+=(dfx &a, dfx b) { return a = a + b; }
__device__ __forceinline__ dfx &operator-=(dfx &a, dfx b) { return a = a - b; }
__device__ __forceinline__ bool operator==(dfx a, dfx b) { return a.v.hi == b.v.hi && a.v.lo == b.v.lo; }
__device__ __forceinline__ bool operator!=(dfx a, dfx b) { return !(a == b); }

}  // namespace avs
