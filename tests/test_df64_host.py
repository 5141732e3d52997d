"""The conversions between FP64 and double-float on the integer pipe (df64.cuh), run on
the CPU from the header's own source: exact for every pair they take themselves, next
to powers of two above all, and every pair that is not normalised goes to the FP64
instructions."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "avocado-sandwich_gb300", "csrc")

PROGRAM = r"""
#include "intrinsics.h"
#include "df64.cuh"
#include <cstdio>
#include <random>
using namespace avs;
static long bad = 0, cases = 0;
// (double)hi + (double)lo, in the FP64 conversion's one rounding
static void pair(float hi, float lo) {
    ++cases;
    const double want = (double)hi + (double)lo, got = df_to_double_int(df64{hi, lo});
    if (std::fabs(got - want) > std::ldexp(std::fabs(want), -52)) {
        if (bad++ < 5) printf("hi %a lo %a: %a, not %a\n", hi, lo, got, want);
    }
}
static void value(double x) {
    ++cases;
    const df64 v = df_from_double_int(x), w = df_from_double(x);
    if ((double)v.hi + (double)v.lo != (double)w.hi + (double)w.lo || df_to_double_int(v) != df_to_double(w)) {
        if (bad++ < 5) printf("%a: %a + %a, not %a + %a\n", x, v.hi, v.lo, w.hi, w.lo);
    }
}
int main() {
    std::mt19937_64 g(1);
    for (int e = -72; e <= 124; ++e)
        for (int up = -3; up <= 3; ++up)
            for (int s = -1; s <= 1; s += 2) {
                // hi at a power of two and its neighbours; lo up to four times half an ulp
                float hi = std::ldexp(1.0f, e);
                for (int k = 0; k < std::abs(up); ++k) hi = std::nextafterf(hi, up > 0 ? INFINITY : 0.0f);
                for (int q = -16; q <= 16; ++q) {
                    const float lo = std::ldexp((float)q / 4.0f, e - 24);
                    pair(s * hi, lo);
                    pair(s * hi, std::nextafterf(lo, 1.0f));
                    pair(s * hi, std::nextafterf(lo, -1.0f));
                }
            }
    for (int i = 0; i < 2000000; ++i) {
        const double m = 1.0 + (double)(g() >> 12) * 0x1p-52, x = std::ldexp(g() & 1 ? m : -m, (int)(g() % 196) - 72);
        value(x);
        const df64 v = df_from_double(x);
        pair(v.hi, v.lo);
        pair(v.hi, v.lo * (float)(1 + g() % 8));  // pairs that are not normalised
    }
    value(0.0);
    value(-0.0);
    printf("%ld %ld\n", bad, cases);
    return bad != 0;
}
"""


def cuda_include():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    return inc if os.path.exists(os.path.join(inc, "cuda_runtime.h")) else None


def run_host(tmp_path, program):
    """Compiles `program` against the headers' sources and returns its output and status."""
    cxx, inc = shutil.which("g++"), cuda_include()
    if cxx is None or inc is None:
        pytest.skip("no g++ or no CUDA headers")
    src, exe = tmp_path / "host.cpp", str(tmp_path / "host")
    src.write_text(program)
    subprocess.check_call([cxx, "-std=c++17", "-O1", "-ffp-contract=off", "-I", os.path.join(HERE, "host"), "-I", CSRC,
                           "-I", inc, str(src), "-o", exe])
    r = subprocess.run([exe], text=True, capture_output=True)
    return r.stdout, r.returncode


def test_integer_conversions(tmp_path):
    out, rc = run_host(tmp_path, PROGRAM)
    assert rc == 0, out
