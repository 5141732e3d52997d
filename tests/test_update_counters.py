"""The counters of the full-T trailing update fit in the T-block buffer at every order
and for every part of a panel that a launch may have (out of core a slab may hold a
single tile: with the room counted by the launch's tiles, calls of more than about
131,000 columns were refused).  Compiles the header that the launch and the workspace
layouts share, and checks orders up to 2^24 on the CPU."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "avocado-sandwich_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "tblk.cuh"
using namespace avs;
int main() {
    long bad = 0, cases = 0;
    for (int b = 128; b <= 256; b *= 2)
        for (int elem = 4; elem <= 8; elem += 4)
            for (int narrow = 0; narrow <= (elem == 8); ++narrow)
                for (int64_t nt = 1; nt <= (1 << 24) / b; nt += 1 + nt / 64) {
                    const int64_t n = nt * b;
                    // the widest update of the call: every column right of the first panel
                    const int64_t c = upd_counters(n - b, b, elem, upd_strip(elem, narrow));
                    bad += 4 * (size_t)c > (size_t)elem * tblk_elems(n, b);
                    // and of a view of the last columns, on the same buffer
                    bad += upd_counters(b, b, elem, upd_strip(elem, narrow)) > c && nt > 1;
                    ++cases;
                }
    printf("%ld %ld\n", bad, cases);
    return bad != 0;
}
"""


def test_counters_fit_for_every_order(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    src = tmp_path / "counters.cpp"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "counters")
    subprocess.check_call([cxx, "-std=c++17", "-I", CSRC, str(src), "-o", exe])
    bad, cases = subprocess.check_output([exe], text=True).split()
    assert (int(bad), int(cases) > 1000) == (0, True)


def test_launch_and_layouts_share_the_header():
    read = lambda f: open(os.path.join(CSRC, f)).read()
    assert "upd_counters(" in read("stage1_wy.cu") and "AVS_ERR_INTERNAL" not in read("stage1_wy.cu")
    assert read("avs_api.cu").count("tblk_elems(n, b)") == 3 and read("avs_ooc.cu").count("tblk_elems(n, b)") == 2
