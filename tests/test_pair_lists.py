"""The pair lists' triangle test (pair_misses_tri, device_lists.cuh), compiled for
the host: it may drop a triangle only when no point of it lies within the
capsule's radius of the centroid segment.  Triangles here have an edge at a small
angle to the pair's direction, or are slivers: the computed axes of such edges
are mostly rounding."""
import subprocess

import pytest

from conftest import load_pkg

HARNESS = r"""
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>
#include "device_lists.cuh"
using namespace rvf;

int main() {
  std::mt19937_64 g(1);
  std::normal_distribution<double> nrm;
  std::uniform_real_distribution<double> U(0.0, 1.0);
  const double two_pi = 6.283185307179586;
  for (double angle : {0.0, 1e-7, 1e-6, 1e-4, 0.3})
    for (double size : {0.01, 0.05, 0.3})
      for (double height : {1.0, 1e-4, 1e-7}) {
        int dropped = 0, far = 0;
        for (int it = 0; it < 5000; ++it) {
          // the pair's direction d and a frame (x, y) across it
          double d[3], x[3], y[3], n = 0.0, q = 0.0;
          for (int k = 0; k < 3; ++k) n += (d[k] = nrm(g)) * d[k];
          for (int k = 0; k < 3; ++k) d[k] /= std::sqrt(n);
          for (int k = 0; k < 3; ++k) q += (x[k] = nrm(g)) * d[k];
          n = 0.0;
          for (int k = 0; k < 3; ++k) n += (x[k] -= q * d[k]) * x[k];
          for (int k = 0; k < 3; ++k) x[k] /= std::sqrt(n);
          for (int k = 0; k < 3; ++k) y[k] = d[(k + 1) % 3] * x[(k + 2) % 3] - d[(k + 2) % 3] * x[(k + 1) % 3];
          const double len = 0.5 + 0.5 * U(g), R = 0.02 + 0.05 * U(g);
          // a triangle with an edge along d, holding a point within 0.95 R of the segment
          // (odd turns: 100 R away, which some axis must see)
          const bool away = it & 1;
          const double t = U(g) * len, r = away ? 100.0 * R : 0.95 * R * U(g), ph = two_pi * U(g), al = two_pi * U(g),
                       s = U(g);
          double w1 = U(g), w2 = U(g), a[3], e1[3], e2[3], p[3], mx = 0.0;
          if (w1 + w2 > 1.0) w1 = 1.0 - w1, w2 = 1.0 - w2;
          for (int k = 0; k < 3; ++k) {
            a[k] = U(g);
            e1[k] = size * (d[k] + angle * x[k]);
            e2[k] = size * (s * d[k] + height * (std::cos(al) * x[k] + std::sin(al) * y[k]));
            p[k] = a[k] + t * d[k] + r * (std::cos(ph) * x[k] + std::sin(ph) * y[k]) - w1 * e1[k] - w2 * e2[k];
            mx = std::max({mx, std::fabs(a[k]), std::fabs(a[k] + len * d[k]), std::fabs(p[k]), std::fabs(p[k] + e1[k]),
                           std::fabs(p[k] + e2[k])});
          }
          float A[3], D[3];
          for (int k = 0; k < 3; ++k) {
            A[k] = (float)a[k];
            D[k] = (float)(a[k] + len * d[k]) - A[k];
          }
          const float4 p0 = make_float4((float)p[0], (float)p[1], (float)p[2], 0.0f);
          const float4 p1 = make_float4((float)(p[0] + e1[0]), (float)(p[1] + e1[1]), (float)(p[2] + e1[2]), 0.0f);
          const float4 p2 = make_float4((float)(p[0] + e2[0]), (float)(p[1] + e2[1]), (float)(p[2] + e2[2]), 0.0f);
          const float em = (float)std::ldexp(2.0 * std::sqrt(3.0) * (1.0 + mx), -16);
          const bool miss = pair_misses_tri(A, D, (float)R, em, p0, p1, p2);
          if (away) far += miss;
          else dropped += miss;
        }
        std::printf("%g %g %g %d %d\n", angle, size, height, dropped, far);
      }
}
"""


@pytest.fixture(scope="module")
def rows(tmp_path_factory):
    load_pkg()
    from rvf_b200 import build
    d = tmp_path_factory.mktemp("lists")
    (d / "h.cu").write_text(HARNESS)
    subprocess.run([build._nvcc(), *build.NVCC_FLAGS, "-o", str(d / "h"), str(d / "h.cu")], check=True,
                   capture_output=True, text=True)
    out = subprocess.run([str(d / "h")], check=True, capture_output=True, text=True).stdout
    return [tuple(map(float, line.split())) for line in out.splitlines()]


def test_keeps_what_a_ray_can_hit(rows):
    assert len(rows) == 45
    assert [r for r in rows if r[3] > 0] == []


def test_drops_what_is_far_from_the_pair(rows):
    """An edge at a clear angle to the direction, or a clear normal, separates."""
    for angle, size, height, _, far in rows:
        if angle == 0.3 and height == 1.0:
            assert far > 0.9 * 2500
