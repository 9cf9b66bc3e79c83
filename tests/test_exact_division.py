"""div_known and inv_sqrt_from (csrc/nd_rayprog.h) give the bits of a / b and of
1 / sqrt(s): the ray generation's 64-bit divisions and root in straight-line FMAs.
Compiled for the host; random operands of the ranges they serve, and the hard cases
(squares and their neighbours, roots whose significand is all ones), with the starting
reciprocal root an ulp off either way."""

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "numericdream_b200", "csrc")

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include "nd_rayprog.h"
int main() {
  std::mt19937_64 g(1);
  long bad_div = 0, bad_root = 0;
  for (long it = 0; it < 3000000; ++it) {
    // pixel coordinates: 2 (px + jitter) / width, jitter a multiple of 2^-24
    const int w = 1 + int((g() >> 33) % ((it & 1) ? 8192 : 2147483647ull));
    const double b = w, px = double(g() % uint64_t(w)), j = it % 3 == 0 ? 0.5 : double(g() >> 40) / 16777216.0;
    const double a = 2.0 * (px + j);
    bad_div += nd::div_known(a, b, 1.0 / b) != a / b;
    double s;
    const double m = 1.0 + double(g() >> 12) * 0x1p-52;
    switch (it % 5) {
      case 0: s = m * m; break;
      case 1: s = std::nextafter(m * m, (it & 8) ? 9.0 : 0.0); break;
      case 2: s = std::ldexp(m, int(g() % 400) - 200); break;
      case 3: s = std::nextafter(std::ldexp(4.0, int(g() % 60) - 30), (it & 8) ? 1e99 : 0.0); break;
      default: s = 1.0 + double(int(g() % 65) - 32) * 0x1p-53; break;
    }
    const double want = 1.0 / std::sqrt(s);
    for (double y : {want, std::nextafter(want, 0.0), std::nextafter(want, 1e300)}) bad_root += nd::inv_sqrt_from(s, y) != want;
  }
  std::printf("%ld %ld\n", bad_div, bad_root);
}
"""


def test_bits_of_division_and_root(tmp_path):
    (tmp_path / "m.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-mfma", "-ffp-contract=off", "-I", CSRC, str(tmp_path / "m.cpp"), "-o",
                    str(tmp_path / "m")], check=True)
    assert subprocess.run([str(tmp_path / "m")], check=True, capture_output=True, text=True).stdout.split() == ["0", "0"]
