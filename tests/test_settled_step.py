"""The `settled` form of a translated de_step: the iteration loop that stops at a step
which returned its own carry gives the bits of the loop that runs every iteration.  The
translated code is compiled for the host and both loops run on the same points."""

import os
import subprocess

import pytest

from numericdream_b200.translator import translate

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "numericdream_b200", "csrc")
BAILOUT = open(os.path.join(ROOT, "numericdream_b200", "formulas", "mandelbulb_bailout.wgsl")).read()
HEAD = "// @param A min=0 max=9 default=8\n// @param B min=0 max=9 default=2\n"
ITER = "fn de_iterations(p: Params) -> i32 { return 9; }\n"
FIN = "fn de_finalize(carry: IterCarry) -> f32 { return bulb_log_escape(carry); }\n"
STEP = "fn de_step(carry: IterCarry, pos: vec3f, p: Params) -> IterCarry {\n"
POWER = HEAD + ITER + STEP + "    return bulb_power_step(carry, pos, p[0]);\n}\n" + FIN
SHADOWED = HEAD + ITER + STEP + """    if (p[1] > 1.0) {
        let carry = IterCarry(pos * 0.5, 2.0);
        if (pos.x > 0.0) { return carry; }
    }
    if (length(carry.z) > p[1]) { return carry; }
    return IterCarry(carry.z * 1.5 + pos, carry.dr * 1.5);
}
""" + FIN
PLAIN = HEAD + ITER + STEP + "    return IterCarry(carry.z * 0.5 + pos, carry.dr);\n}\n" + FIN

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include "nd_helpers.h"
#include "f.inc"
template <class T> int differ(const float* prm) {
  int bad = 0;
  const double at[] = {0.0, -0.0, 1e-20, 0.3, -0.7, 1.1, 1.9999, 2.0, -2.0, 2.0001, 7.0, 1e20, INFINITY, NAN};
  for (double x : at) for (double y : at) for (double z : at) {
    const ndw::v3<T> pos{T(x), T(y), T(z)};
    for (int n = 0; n <= 9; ++n) {
      ndw::IterCarry<T> a{pos, T(1)}, b{pos, T(1)};
      for (int i = 0; i < n; ++i) a = NS::de_step<T, const float*>(a, pos, prm);
      for (int i = 0; i < n; ++i) {
        bool settled = false;
        b = NS::de_step<T, const float*>(b, pos, prm, settled);
        if (settled) break;
      }
      const T u[4] = {a.z.x, a.z.y, a.z.z, a.dr}, v[4] = {b.z.x, b.z.y, b.z.z, b.dr};
      for (int k = 0; k < 4; ++k) bad += !(u[k] != u[k] && v[k] != v[k]) && std::memcmp(&u[k], &v[k], sizeof(T)) != 0;
    }
  }
  return bad;
}
int main() {
  const float prm[16] = {8.0f, 2.0f, 2.0f}, odd[16] = {5.5f, 1.25f, 1.25f};
  std::printf("%d %d %d %d\n", differ<float>(prm), differ<float>(odd), differ<double>(prm), differ<double>(odd));
}
"""


@pytest.mark.parametrize("source", [BAILOUT, POWER, SHADOWED], ids=["early_return", "helper", "shadowed_name"])
def test_settled_loop_gives_the_same_carry(tmp_path, source):
    tf = translate(source, "f")
    assert tf.settles
    prog = PROGRAM.replace("NS::", tf.namespace + "::")
    (tmp_path / "f.inc").write_text(tf.cpp)
    (tmp_path / "m.cpp").write_text(prog)
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-I", CSRC, "-I", str(tmp_path),
                    str(tmp_path / "m.cpp"), "-o", str(tmp_path / "m")], check=True)
    out = subprocess.run([str(tmp_path / "m")], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["0", "0", "0", "0"]


def test_a_step_without_such_a_return_has_no_settled_form():
    tf = translate(PLAIN, "f")
    assert not tf.settles and "settled" not in tf.cpp
