"""The second sinogram layout's index arithmetic (SinoLayout), compiled for the host:
every element of odd and even detectors has its own place, a row's successor is one
step away, a layout of another stride holds the same element, and what has no second
layout (one row or channel, 31 bits passed) keeps the raw data's order."""
import os
import subprocess

from ctbb_icd_b200 import build as B

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "gpu_internal.h"
#define REQUIRE(c) do { if (!(c)) { printf("line %d: %s (nr %d nch %d views %d)\n", __LINE__, #c, nr, nch, views); return 1; } } while (0)
int main() {
    const int sizes[][3] = {{2, 2, 1}, {2, 3, 7}, {3, 2, 8}, {5, 7, 9}, {64, 10, 17}, {7, 47, 33}};
    for (auto& z : sizes) {
        const int nr = z[0], nch = z[1], views = z[2];
        const SinoLayout l = SinoLayout::grouped(nch, nr, views), m = SinoLayout::grouped(nch, nr, views + 21);
        REQUIRE(!l.is_raw() && !(l == m) && l.stride % 8 == 0);
        std::vector<char> taken(l.size(), 0);
        for (int v = 0; v < views; ++v)
            for (int c = 0; c < nch; ++c)
                for (int r = 0; r < nr; ++r) {
                    const uint32_t a = l.from_raw((uint32_t)(r + nr * (c + nch * v)));
                    REQUIRE(a < l.size() && !taken[a]);
                    taken[a] = 1;
                    REQUIRE(a == l.at(v, c, r) && a == l.at(0, c, r) + 4u * v);
                    if (r + 1 < nr) REQUIRE(l.at(v, c, r + 1) == a + (a & 1 ? l.row_step() : 1u));
                    REQUIRE(l.restride(a, m) == m.at(v, c, r) && m.restride(m.at(v, c, r), l) == a);
                }
    }
    const int nr = 0, nch = 0, views = 0;
    REQUIRE(SinoLayout::raw().is_raw());
    REQUIRE(SinoLayout::grouped(736, 1, 1152).is_raw() && SinoLayout::grouped(1, 64, 1152).is_raw());
    REQUIRE(!SinoLayout::grouped(1024, 64, 32760).is_raw() && SinoLayout::grouped(1024, 64, 32761).is_raw());
    REQUIRE(SinoLayout::grouped(1024, 64, 65536).is_raw() && SinoLayout::raw().size() == 0);
    return 0;
}
"""


def test_second_layout(tmp_path):
    src, exe = str(tmp_path / "t.cpp"), str(tmp_path / "t")
    with open(src, "w") as f:
        f.write(PROGRAM)
    inc = os.path.join(os.path.dirname(B.HERE), "include")
    subprocess.run([B.HOSTCXX, "-std=c++17", "-O1", "-I", B.CSRC, "-I", inc, "-I", "/usr/local/cuda/include", src,
                    "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
