// device_lists.cuh -- certified geometric tests of the pair lists and of
// the tile classification: a pair's shadow rays all lie in its capsule (the
// centroid segment grown by R = max(rad_i, rad_j) plus a margin), and a box
// or triangle farther than the capsule's radius (plus the rounding margin of
// the reference's test) is never reached or hit by any of them.
#pragma once

#include "device_trace.cuh"

namespace rvf {

// True when no ray of the pair (segments within R of the centroid segment
// a -> a + d) can be a hit of the reference's test of the triangle
// with corners p0, p1, p2 (FP32) and rounding margin p0.w.  em = S 2^-16 (S: at least
// |d| and every edge) absorbs the FP32 rounding of the corners and of the
// projections (a few 2^-24 S |w|).
//
// An axis w = d x f of an edge f is taken to see the segment as the point 0 and the
// edge as one point, so that two corners' projections decide.  The computed w
// misses both directions by its own rounding, which does not shrink with |w| when
// f is nearly parallel to d: with u = 2^-24, |w - d x f| <= 2.5 u |d| |f|, and f is
// rounded by u |f|, so the segment spans up to 2.5 u |d|^2 |f| and the edge up to
// 3.5 u |d| |f|^2, together at most 6 u S |d| |f| = (6/256) em |d| |f|.  The gap is
// taken smaller by em/32 |d|_1 |f|_1.  The normal likewise: f1.n and f2.n are at most
// 3.5 u |f1| |f2| max(|f1|, |f2|).  (Without this, triangles with an edge along the pair's
// direction, and slivers, lost up to 16% of those a ray of the pair does hit.)
__host__ __device__ __forceinline__ bool pair_misses_tri(const float* a, const float* d, float R, float em,
                                                         const float4& p0, const float4& p1, const float4& p2) {
  const float rm = R + p0.w + em, rm2 = rm * rm;
  const float s0[3] = {p0.x - a[0], p0.y - a[1], p0.z - a[2]};
  const float s1[3] = {p1.x - a[0], p1.y - a[1], p1.z - a[2]};
  const float s2[3] = {p2.x - a[0], p2.y - a[1], p2.z - a[2]};
  const float c = -0.03125f * em, cd = c * (fabsf(d[0]) + fabsf(d[1]) + fabsf(d[2]));
  // w = d x (edge g - e): the segment at 0 (from a), the edge at g.w, the third corner at h.w
  auto edge = [&](const float4& e, const float4& g, const float* sg, const float* sh) {
    const float fx = g.x - e.x, fy = g.y - e.y, fz = g.z - e.z;
    const float wx = d[1] * fz - d[2] * fy, wy = d[2] * fx - d[0] * fz, wz = d[0] * fy - d[1] * fx;
    const float u = fmaf(sg[0], wx, fmaf(sg[1], wy, sg[2] * wz)), v = fmaf(sh[0], wx, fmaf(sh[1], wy, sh[2] * wz));
    const float gap = fmaf(cd, fabsf(fx) + fabsf(fy) + fabsf(fz), fmaxf(fminf(u, v), -fmaxf(u, v)));
    return gap > 0.0f && gap * gap > rm2 * fmaf(wx, wx, fmaf(wy, wy, wz * wz));
  };
  if (edge(p0, p1, s0, s2)) return true;
  if (edge(p0, p2, s0, s1)) return true;
  if (edge(p1, p2, s1, s0)) return true;
  // the triangle's normal: its plane at s0.n, the segment from 0 to d.n
  const float f1[3] = {p1.x - p0.x, p1.y - p0.y, p1.z - p0.z}, f2[3] = {p2.x - p0.x, p2.y - p0.y, p2.z - p0.z};
  const float nx = f1[1] * f2[2] - f1[2] * f2[1], ny = f1[2] * f2[0] - f1[0] * f2[2], nz = f1[0] * f2[1] - f1[1] * f2[0];
  const float u = fmaf(s0[0], nx, fmaf(s0[1], ny, s0[2] * nz)), e = fmaf(d[0], nx, fmaf(d[1], ny, d[2] * nz));
  const float gap = fmaf(c * (fabsf(f1[0]) + fabsf(f1[1]) + fabsf(f1[2])), fabsf(f2[0]) + fabsf(f2[1]) + fabsf(f2[2]),
                         fmaxf(u - fmaxf(e, 0.0f), fminf(e, 0.0f) - u));
  return gap > 0.0f && gap * gap > rm2 * fmaf(nx, nx, fmaf(ny, ny, nz * nz));
}

// The pair's capsule for the list walk, in FP32: the centroid segment's
// start A and direction reciprocals (from FP64, rounded once), and the radius
// grown by em.  A box test in FP32 (capsule_misses_box) then only reports a
// miss when the FP64 test with the ungrown radius would: every rounding of
// the test (the nodes' and A's FP32 copies, the subtraction, 1/d) moves a
// slab parameter by a few 2^-24 S |1/d|, the growth by em = 2^-16 S moves it
// by em |1/d|.  Components of d that are exactly zero use the containment
// test, as pair_misses_box does.
struct CapsuleF {
  float A[3], inv[3];
  bool zero[3];
  float R;
};

__device__ __forceinline__ bool capsule_misses_box(const CapsuleF& c, const NodeF& nd) {
  float te = 0.0f, tx = 1.0f;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float lo = nd.lo[k] - c.R, hi = nd.hi[k] + c.R;
    if (c.zero[k]) {
      if (c.A[k] < lo || c.A[k] > hi) return true;
      continue;
    }
    const float t1 = (lo - c.A[k]) * c.inv[k], t2 = (hi - c.A[k]) * c.inv[k];
    te = fmaxf(te, fminf(t1, t2));
    tx = fminf(tx, fmaxf(t1, t2));
  }
  return te > tx;
}

}  // namespace rvf
