"""The reflector scalars from hardware estimates (reflect.cuh), run on the CPU from the
header's own source with estimates wrong by up to 2^-21.5, against extended precision.
In FP32 and FP64 they are to be as accurate as the same expressions with a correctly
rounded square root and divisions: the largest error over the same arguments within 2%
of theirs.  Double-float: each result within 2^-45 (four roundings of at most 2^-47)."""
import os

import pytest

from test_df64_host import CSRC, run_host

PROGRAM = r"""
#include "intrinsics.h"
#include "reflect_host.cuh"
#include <cstdio>
#include <random>
using namespace avs;
typedef long double L;
static double ulp(float v) { return std::ldexp(1.0, std::ilogb(v) - 23); }
static double ulp(double v) { return std::ldexp(1.0, std::ilogb(v) - 52); }
template <typename T> static void worst(double &w, T got, L want) {
    const double e = (double)(std::fabs((L)got - want) / (L)ulp((T)want));
    if (!(e <= w)) w = e;
}
static L val(df64 v) { return (L)v.hi + (L)v.lo; }
static void worst_df(double &w, df64 got, L want) {
    const double e = (double)std::fabs((val(got) - want) / want) * 0x1p45;
    if (!(e <= w)) w = e;
}
int main() {
    std::mt19937_64 g(3);
    auto uni = [&]() { return (double)(g() >> 11) * 0x1p-53; };
    double fn = 0, ft = 0, fs = 0, dn = 0, dr = 0, di = 0, dt = 0, xn = 0, xr = 0, xi = 0;
    double Fn = 0, Ft = 0, Fs = 0, Dn = 0, Dr = 0, Di = 0, Dt = 0;  // correctly rounded operations
    for (int i = 0; i < 1000000; ++i) {
        const int e = (int)(g() % 60) - 30;
        const double al = std::ldexp(uni() * 2 - 1, e), s = std::ldexp(uni() + 1e-3, 2 * e);
        {
            const float alpha = (float)al, sf = (float)s;
            float tau, beta, scal;
            reflector_scalars(alpha, sf, tau, beta, scal);
            const float a2s = std::fmaf(alpha, alpha, sf);
            const L n = sqrtl((L)a2s);
            worst(fn, std::fabs(beta), n);
            worst(ft, tau, 1 + fabsl((L)alpha) / n);
            const L b = alpha >= 0 ? -n : n;
            worst(fs, scal, 1 / ((L)alpha - b));
            const float nf = std::sqrt(a2s), bf = alpha >= 0 ? -nf : nf;
            worst(Fn, nf, n);
            worst(Ft, std::fmaf(std::fabs(alpha), 1.0f / nf, 1.0f), 1 + fabsl((L)alpha) / n);
            worst(Fs, 1.0f / (alpha - bf), 1 / ((L)alpha - b));
        }
        {
            const double x = std::fma(al, al, s);
            double rn, n;
            rsqrt_sqrt(x, rn, n);
            worst(dn, n, sqrtl((L)x));
            worst(dr, rn, 1 / sqrtl((L)x));
            worst(di, rcp_est(al), 1 / (L)al);
            double tau, beta, scal;
            reflector_scalars(al, s, tau, beta, scal);
            worst(dt, tau, 1 + fabsl((L)al) / sqrtl((L)x));
            const double nd = std::sqrt(x), bd = al >= 0 ? -nd : nd;
            worst(Dn, nd, sqrtl((L)x));
            worst(Dr, 1.0 / nd, 1 / sqrtl((L)x));
            worst(Di, 1.0 / al, 1 / (L)al);
            worst(Dt, (bd - al) / bd, 1 + fabsl((L)al) / sqrtl((L)x));
        }
        {
            const df64 x = df_from_double(std::fma(al, al, s)), a = df_from_double(al);
            df64 rn, n;
            rsqrt_sqrt(x, rn, n);
            worst_df(xn, n, sqrtl(val(x)));
            worst_df(xr, rn, 1 / sqrtl(val(x)));
            worst_df(xi, rcp_est(a), 1 / val(a));
        }
    }
    printf("FP32 norm %.3f (%.3f) tau %.3f (%.3f) 1/(alpha - beta) %.3f (%.3f); FP64 norm %.3f (%.3f) 1/norm %.3f (%.3f) "
           "1/x %.3f (%.3f) tau %.3f (%.3f); double-float, of 2^-45: norm %.3f 1/norm %.3f 1/x %.3f\n", fn, Fn, ft, Ft, fs, Fs,
           dn, Dn, dr, Dr, di, Di, dt, Dt, xn, xr, xi);
    return !(fn <= 1.02 * Fn && ft <= 1.02 * Ft && fs <= 1.02 * Fs && dn <= 1.02 * Dn && dr <= 1.02 * Dr &&
             di <= 1.02 * Di && dt <= 1.02 * Dt && xn <= 1 && xr <= 1 && xi <= 1);
}
"""


def test_reflector_scalars(tmp_path):
    s = open(os.path.join(CSRC, "reflect.cuh")).read()
    for op, call in (("rsqrt", "rsqrtf(x)"), ("rcp", "__fdividef(1.0f, x)")):
        line = 'asm("%s.approx.ftz.f32 %%0, %%1;" : "=f"(r) : "f"(x));' % op
        assert s.count(line) == 1
        s = s.replace(line, "r = %s;" % call)
    (tmp_path / "reflect_host.cuh").write_text(s)
    out, rc = run_host(tmp_path, PROGRAM)
    print(out)
    assert rc == 0, out
