"""inv_sqrt_from (csrc/nd_rayprog.h) on the arguments that are hardest to round: those whose
root lies beside the midpoint of two doubles, 2^-54 of an ulp from it and nearer, and the
powers of two, with the starting reciprocal root up to two ulps off."""

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "numericdream_b200", "csrc")

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include "nd_rayprog.h"
static long bad = 0, tried = 0;
static void check(double s) {
  const double want = 1.0 / std::sqrt(s);
  double y = std::nextafter(std::nextafter(want, 0.0), 0.0);
  for (int i = 0; i < 5; ++i, y = std::nextafter(y, 1e300)) {
    bad += nd::inv_sqrt_from(s, y) != want;
    ++tried;
  }
}
int main() {
  // (g + 1/2)^2 = g^2 + g + 1/4: g^2 + g = r modulo the spacing of the doubles there, solved
  // bit by bit (its derivative is odd), gives an s whose root is about r / 2g from g + 1/2
  for (long r = -60000; r <= 60000; r += 2)
    for (int root = 0; root < 2; ++root)
      for (int bits = 52; bits <= 53; ++bits) {
        unsigned long long x = (unsigned long long)root;
        for (int b = 1; b < bits; ++b)
          if (((x * x + x - (unsigned long long)r) >> b) & 1) x ^= 1ull << b;
        const unsigned long long g = bits == 52 ? x | (1ull << 52) : x;
        if (g < (1ull << 52) || g >= (1ull << 53)) continue;
        const __int128 s = (__int128)g * g + g - r;
        const double d = double((unsigned long long)(s >> 52));
        if ((__int128)d != (s >> 52) || (s & ((1ll << 52) - 1)) != 0) continue;  // not a double
        check(std::ldexp(d, -52));
        check(std::ldexp(d, -50));
        check(std::ldexp(d, -252));
      }
  for (double s : {0x1.d407bb3641da5p+0, 0x1.4eb5f85e783a9p+1, 0x1.5b95344972fe2p+1}) check(s);
  for (int e = -400; e <= 400; ++e)
    for (int k = -40; k <= 40; ++k) {
      double s = std::ldexp(1.0, e);
      for (int i = 0; i < (k < 0 ? -k : k); ++i) s = std::nextafter(s, k < 0 ? 0.0 : 1e300);
      check(s);
    }
  std::printf("%ld %ld\n", bad, tried);
}
"""


def test_hard_roots_are_correctly_rounded(tmp_path):
    (tmp_path / "m.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-mfma", "-ffp-contract=off", "-I", CSRC, str(tmp_path / "m.cpp"), "-o",
                    str(tmp_path / "m")], check=True)
    bad, tried = map(int, subprocess.run([str(tmp_path / "m")], check=True, capture_output=True, text=True).stdout.split())
    assert tried > 1000000 and bad == 0, (bad, tried)
