"""nd_atan2_poly on the host, which keeps subnormal operands (the device flushes them): the
angle of two subnormals is their own, and zeros give atan2's zeros."""

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "numericdream_b200", "csrc")

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include "nd_wgsl.h"
int main() {
  const float at[] = {0.0f, -0.0f, 1e-45f, -1e-45f, 3e-44f, -1e-42f, 1e-40f, -1e-40f, 7e-39f, 1.17549421e-38f, 1.17549435e-38f,
                      -1.2e-38f, 1e-37f, 1e-30f, -1.0f, 2.0f, 1e38f, INFINITY, -INFINITY};
  double worst = 0.0;
  int signs = 0;
  for (float y : at) for (float x : at) {
    const float got = ndw::nd_atan2_poly(y, x);
    const double e = std::fabs(double(got) - std::atan2(double(y), double(x)));
    if (!(e <= worst)) worst = e;
    signs += std::signbit(got) != std::signbit(y);
  }
  std::printf("%.9g %d\n", worst, signs);
}
"""


def test_angles_of_subnormals(tmp_path):
    (tmp_path / "m.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", CSRC, str(tmp_path / "m.cpp"), "-o",
                    str(tmp_path / "m")], check=True)
    worst, signs = subprocess.run([str(tmp_path / "m")], check=True, capture_output=True, text=True).stdout.split()
    # the polynomial's own bound on every other operand (5e-7), and atan2's sign
    assert float(worst) <= 5e-7 and int(signs) == 0, (worst, signs)
