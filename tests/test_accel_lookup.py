"""accel_skip's search (csrc/nd_rayprog.h) finds the finest cascade that holds a point, as
trying every cascade from the finest on does.  Compiled for the host; points around the
cascades' faces to a few ulps, far cameras, every grid size and depth, infinities, NaN."""

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "numericdream_b200", "csrc")

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>
#include "nd_view.h"
static float naive(const nd::DevView& v, float px, float py, float pz) {
  const float rf = float(v.accel_res);
  for (int l = 0; l < v.accel_levels; ++l) {
    const float inv = v.accel_inv[l];
    const float fx = floorf((px - v.accel_prm[l][0]) * inv), fy = floorf((py - v.accel_prm[l][1]) * inv),
                fz = floorf((pz - v.accel_prm[l][2]) * inv);
    if (!(fx >= 0.0f && fy >= 0.0f && fz >= 0.0f && fx < rf && fy < rf && fz < rf)) continue;
    const int r = v.accel_res;
    return v.accel_grid[((int64_t(l) * r + int(fz)) * r + int(fy)) * r + int(fx)];
  }
  return 0.0f;
}
int main() {
  std::mt19937_64 g(7);
  std::uniform_real_distribution<double> U(-1.0, 1.0);
  long bad = 0, found = 0;
  for (int res : {16, 20, 64, 160})
    for (int levels : {1, 2, 6, 8})
      for (double far : {0.0, 1.0, 37.0, 3000.0, 1e5}) {
        nd_view_desc d;
        memset(&d, 0, sizeof d);
        d.width = d.height = d.tile_w = d.tile_h = 8;
        d.spp = 1;
        d.max_dist = 24.0f;
        d.accel_res = res;
        d.accel_levels = levels;
        d.accel_safety = 1.0f;
        for (int a = 0; a < 3; ++a) d.cam_pos[a] = far * U(g);
        std::vector<float> grid(size_t(levels) * res * res * res);
        for (size_t i = 0; i < grid.size(); ++i) grid[i] = float(i % 16777213) + 1.0f;
        nd::DevView v = nd::make_dev_view(d, 0, 0, 0);
        nd::place_accel(v, d, grid.data());
        for (int it = 0; it < 40000; ++it) {
          float p[3];
          const int l = int(g() % levels), face = int(g() % 6);
          const float side = float(res) * v.accel_prm[l][3];
          for (int a = 0; a < 3; ++a) p[a] = v.accel_prm[l][a] + side * float(0.5 + 0.52 * U(g));
          if (it % 3) {  // on a face of cascade l, a few ulps or a fraction of a cell off
            float f = v.accel_prm[l][face % 3] + (face < 3 ? 0.0f : side);
            if (it % 3 == 1) for (int k = int(g() % 4); k > 0; --k) f = std::nextafterf(f, (g() & 1) ? 1e30f : -1e30f);
            else f += v.accel_prm[l][3] * float(1.5 * U(g));
            p[face % 3] = f;
          }
          if (it == 5) p[0] = NAN;
          if (it == 6) p[2] = INFINITY;
          if (it == 7) p[0] = p[1] = p[2] = NAN;
          if (it == 8) p[1] = -3e38f;
          const float a = nd::accel_skip(v, p[0], p[1], p[2]), b = naive(v, p[0], p[1], p[2]);
          bad += a != b;
          found += b != 0.0f;
        }
      }
  std::printf("%ld %ld\n", bad, found);
}
"""


def test_search_equals_trying_every_cascade(tmp_path):
    (tmp_path / "m.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", CSRC, str(tmp_path / "m.cpp"), "-o",
                    str(tmp_path / "m")], check=True)
    bad, found = map(int, subprocess.run([str(tmp_path / "m")], check=True, capture_output=True, text=True).stdout.split())
    assert bad == 0 and found > 1000000
