"""Host check of the one-launch network's layout (csrc/clb_net.cuh): the multiply-high divisions of every layout that is admitted are
exact over all their dividends, also of a single channel, and layouts for which one is not are refused."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include "clb_net.cuh"
using namespace clb;
static long check(const FastDiv &f, long long dividends)
{
    long wrong = 0;
    for (long long n = 0; n < dividends; ++n) wrong += f.div((int)n) != (int)(n / f.d);
    return wrong;
}
int main()
{
    long admitted = 0, refused = 0, wrong = 0;
    const int channels[] = {1, 2, 3, 64};
    for (int c : channels)
        for (int pad = 0; pad <= 2; ++pad)
            for (int side = 2; side <= 600; side += side < 40 ? 3 : side < 250 ? 37 : c == 1 ? 2 : 50) {
                NetStorage s = {};
                if (!s.lay_out(0, c, side, side + (side & 8), pad, pad)) {
                    ++refused;
                    continue;
                }
                ++admitted;
                if (!s.halo_units) continue; // then nothing is divided
                wrong += check(s.by_image, (long long)c * s.image) + check(s.by_W, s.image);
                wrong += check(s.by_channel, s.halo_units) + check(s.by_pitch, s.per_channel);
            }
    NetStorage s = {};
    printf("%ld %ld %ld", admitted, refused, wrong);
    printf(" %d", (int)s.lay_out(0, 1, 260, 260, 1, 1));       // 67599 / 67600 comes out as 1
    printf(" %d", (int)s.lay_out(0, 1, 2, 70000, 1, 1));       // one long row
    printf(" %d", (int)s.lay_out(0, 1, 28, 28, 1, 1));
    printf(" %d", (int)s.lay_out(0, 1, 1, 1 << 20, 0, 0));     // a flat layer's features
    printf(" %d\n", (int)s.lay_out(1 << 24, 1, 1, 1, 0, 0));   // beyond the units that 32 bits of bytes reach
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_divisions_of_admitted_layouts_are_exact(tmp_path):
    src, exe = tmp_path / "layout.cpp", tmp_path / "layout"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-D__host__=", "-D__device__=", "-D__forceinline__=inline", "-I", os.path.join(ROOT, "convlogic_b200", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    admitted, refused, wrong, side260, row, mnist, flat, beyond = map(int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert admitted > 300 and refused > 20
    assert wrong == 0
    assert (side260, row, mnist, flat, beyond) == (0, 0, 1, 1, 0)
