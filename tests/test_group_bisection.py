"""The bisection that a formula group's march keeps (MarchLane's group form) against the
inline march (Lane), on the host: the same hit, distance, steps and evaluations, ray for ray,
over bisection budgets, exact hits and the edges of the limits, both DE precisions."""

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "numericdream_b200", "csrc")

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include "nd_rayprog.h"
#include "nd_view.h"
#include <vector>
// a bumpy sphere, an estimate that oversteps so that samples go below eps from far
template <class T> T de(ndw::v3<T> p) {
  const T r = ndw::length(p);
  return (r - T(1) + T(0.05) * ndw::sin(T(9) * p.x) * ndw::cos(T(7) * p.y)) * T(1.6);
}
static long bisected = 0;
template <class T> long differ(const nd::DevView& v) {
  long bad = 0;
  std::vector<float> depth(v.rays, 0.0f);
  nd_gbuffer g;
  memset(&g, 0, sizeof(g));
  g.depth = depth.data();
  for (int64_t it = 0; it < v.rays; ++it) {
    nd::Lane<T, true> a;
    a.start(v, int32_t(it), 0, true);
    a.evals = 0;
    a.hit = false;
    bool late = v.max_samples <= 0;
    for (int n = 0; !late && a.phase == nd::PH_MARCH && n < 100000; ++n) {
      nd::DEOut<T> o;
      o.d = de<T>(nd::to_t<T>(a.sample_pos(v)));
      a.advance(v, o, g, nullptr);
    }
    nd::MarchLane<T, true, true> b;
    b.start(v, int32_t(it), 0);
    for (int n = 0; b.mode != b.kDone && n < 100000; ++n) b.template advance<false>(v, de<T>(nd::to_t<T>(b.sample_pos(v))));
    const bool hit = !late && a.phase == nd::PH_NORMAL;
    bisected += b.hit && b.k > 1;
    bad += hit != b.hit || a.evals != b.evals(v) || (hit && (a.t != b.st || a.i != b.i));
  }
  return bad;
}
int main() {
  long bad = 0;
  for (int budget : {0, 1, 2, 4, 40})
    for (int exact : {0, 1})
      for (int steps : {0, 1, 3, 7, 200})
        for (int verify : {0, 1})
          for (float z : {-3.0f, -0.2f}) {
            nd_view_desc d;
            memset(&d, 0, sizeof(d));
            d.width = d.tile_w = 29;
            d.height = d.tile_h = 23;
            d.spp = 1;
            d.cam_pos[2] = z;
            d.fwd[2] = d.right[0] = d.up[1] = 1.0;
            d.max_steps = steps;
            d.max_dist = 24.0f;
            d.eps_coef = 1e-3f;
            d.eps_floor = 1e-4f;
            d.refine_budget = budget;
            d.march_verify = verify;
            d.step_safety = 1.0f;
            d.flags = exact ? ND_VIEW_EXACT_HIT : 0;
            const nd::DevView v = nd::make_dev_view(d, 0, 0, 0);
            bad += differ<float>(v) + differ<double>(v);
          }
  std::printf("%ld %ld\n", bad, bisected);
}
"""


def test_group_march_equals_the_inline_march(tmp_path):
    (tmp_path / "m.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-mfma", "-ffp-contract=off", "-I", CSRC, "-I", os.path.join(ROOT, "include"),
                    str(tmp_path / "m.cpp"), "-o", str(tmp_path / "m")], check=True)
    bad, bisected = map(int, subprocess.run([str(tmp_path / "m")], check=True, capture_output=True, text=True).stdout.split())
    assert bisected > 1000 and bad == 0
