// device_mixed.cuh -- FP32 shadow-ray primitives with certified decisions.
//
// Every FP32 slab or Moller-Trumbore decision comes with a forward error
// bound against the FP64 computation the reference performs (src/GPUBVH.jl:
// 219-269).  A decision is taken in FP32 only when the FP32 value clears its
// threshold by more than the bound; otherwise the lane is marked uncertain and
// its whole ray is traced again in FP64 with the reference's arithmetic.  The
// bounds are deliberately loose (relative terms 2^-16 .. 2^-18 against FP32
// rounding of ~2^-22 for these expressions): a loose bound only costs re-tests.
#pragma once

#include "device_common.cuh"

namespace rvf {

// relative error allowances
constexpr float kRho = 9.5367431640625e-07f;  // 2^-20: direction, 1/direction, segment length
constexpr float kE0 = 1.52587890625e-05f;     // 2^-16: Moller-Trumbore terms
constexpr float kMinDir = 1e-4f;              // smaller direction components go to FP64

struct RayF {
  float o[3];
  float d[3];
  float inv[3];
  float tmax;
  float k0;     // absolute slab-parameter error: 2 delta max|inv|
  float delta;  // absolute position error of origin / node / vertex coordinates
};

enum : int { kMiss = 0, kHit = 1, kUnsure = 2 };

// Approximate reciprocal (one MUFU op, at most 1 ulp = 2^-23 relative error):
// every quantity it feeds has an error allowance of 2^-20 or more.
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// FP32 ray from origin xo (absolute, rounded) along r = (rx,ry,rz), |r|^2 = r2.
// Returns false when a direction component is too small for a certified FP32
// traversal (the ray then goes to FP64).
__device__ __forceinline__ bool make_ray_f(const float* xo, float rx, float ry, float rz, float r2, float delta,
                                           RayF& R) {
  float ir = rsqrtf(r2);
  R.o[0] = xo[0]; R.o[1] = xo[1]; R.o[2] = xo[2];
  R.d[0] = rx * ir; R.d[1] = ry * ir; R.d[2] = rz * ir;
  R.tmax = r2 * ir;
  if (fabsf(R.d[0]) < kMinDir || fabsf(R.d[1]) < kMinDir || fabsf(R.d[2]) < kMinDir) return false;
  R.inv[0] = rcp_approx(R.d[0]); R.inv[1] = rcp_approx(R.d[1]); R.inv[2] = rcp_approx(R.d[2]);
  float mi = fmaxf(fmaxf(fabsf(R.inv[0]), fabsf(R.inv[1])), fabsf(R.inv[2]));
  R.delta = delta;
  R.k0 = 2.0f * delta * mi;
  return true;
}

// Slab test with a certified outcome (kHit / kMiss / kUnsure).
//
// The box is hit iff the four parameter intervals X, Y, Z (one per slab) and
// S = [0, t_max] share a point, i.e. (1-D Helly) iff every pair of different
// intervals overlaps: the comparison te <= tx of the reference.  An interval
// never needs a margin against itself -- in particular the two ends of a
// slab of zero thickness (lo == hi, as for the leaves of a flat face) are the
// same number in FP32 and in FP64 -- so each interval's end is compared with
// the largest start of the others, and the smallest such slack decides.
__device__ __forceinline__ int slab_f(const NodeF& nd, const RayF& R) {
  const float t1x = (nd.lo[0] - R.o[0]) * R.inv[0], t2x = (nd.hi[0] - R.o[0]) * R.inv[0];
  const float t1y = (nd.lo[1] - R.o[1]) * R.inv[1], t2y = (nd.hi[1] - R.o[1]) * R.inv[1];
  const float t1z = (nd.lo[2] - R.o[2]) * R.inv[2], t2z = (nd.hi[2] - R.o[2]) * R.inv[2];
  const float lx = fminf(t1x, t2x), hx = fmaxf(t1x, t2x);
  const float ly = fminf(t1y, t2y), hy = fmaxf(t1y, t2y);
  const float lz = fminf(t1z, t2z), hz = fmaxf(t1z, t2z);
  const float xy = fmaxf(lx, ly), zs = fmaxf(lz, 0.0f);
  const float te = fmaxf(xy, zs);
  const float tx = fminf(fminf(fminf(hx, hy), hz), R.tmax);
  const float m = R.k0 + 2.0f * kRho * (fabsf(te) + fabsf(tx) + R.tmax);
  const float slack = fminf(fminf(hx - fmaxf(ly, zs), hy - fmaxf(lx, zs)),
                            fminf(hz - fmaxf(xy, 0.0f), R.tmax - fmaxf(xy, lz)));
  return slack > m ? kHit : slack < -m ? kMiss : kUnsure;
}

// Allowances of mt_f: e0 relative (|o - v0| |e| or |e1| |e2|), d absolute, in
// units of the ray's delta = 2^-20 extent.
struct MtTol {
  float e0, d;
};
// kMtLoose: rays formed in FP32 as r = (c_j - c_i) + (o_q - o_p), with
// Q = |c_j - c_i| + rad_i + rad_j at most 33 |r| (kMinRay2; shorter ones go to FP64:
// elements can bulge far beyond their corners).  With u = 2^-24 and
// |c_j - c_i| + |o_p| + |o_q| <= Q, |o_q - o_p| <= Q + |r|, the direction is off by at
// most u (2 Q + 2 |r|) / |r| + 5 u <= 73 u in each component, so the largest of the
// terms below, a, by 1.73 (1.41 74 + 2) u n1 n2 = 184 u n1 n2, against 256 u.
constexpr MtTol kMtLoose{kE0, 2.0f};
constexpr float kMinRay2 = 1.0f / 1089.0f;  // |r|^2 / Q^2
// For rays whose direction is off by at most 7 2^-24 in each component: r formed
// in FP64 and rounded, or as above with |o_p| + |o_q| <= 0.6 D, D = |c_j - c_i|, so that
// |r| >= 0.4 D:
// 2^-24 (2.5 + 3 + 1), and the scaling's rounding.  With u = 2^-24, ns = |s|_1:
// h = d x e2 is within 13.4 u n2 a component, so U = s.h within
// (13.4 + 3 + 1) u ns n2 = 2^-19.9 ns n2, V within (1.73 4.5 + 12 + 5) u ns n1 =
// 2^-19.4 ns n1, T within 14.5 u ns n1 n2 and a within 30 u n1 n2 = 2^-19.1 n1 n2:
// 2^-18 is twice the largest.  Positions (origin 2^-23, vertex 2^-24 of the
// coordinates) move U by at most 4.5 2^-23 n2 = 2^-20.8 n2 and V by 2^-20.6 n1 per unit
// extent, against 2^-19.7 and 2^-18.7 here.
constexpr MtTol kMtTight{3.814697265625e-06f, 1.25f};

// Moller-Trumbore with certified outcome; the triangle stores |e1|, |e2|
// (rounded up) in n1, n2.  The reference's u, v, t are quotients U / a, V / a,
// T / a; with |a| certainly above its cut, each comparison is taken between
// the numerators and multiples of |a| (no division), the numerators within
//   |dU| <= (e0 ns + d2) n2,  |dV| <= (e0 ns + 2 d2) n1,  |dT| <= (e0 ns + 2 d2) n1 n2
// and |da| <= e0 n1 n2 of the reference's (ns bounds |o - v0|, d2 = d delta;
// the relative terms also cover its own FP64 rounding).
__device__ __forceinline__ int mt_f(const TriF& t, const RayF& R, MtTol tol = kMtLoose) {
  const float n1 = __int_as_float(t.pad0), n2 = __int_as_float(t.pad1);
  const float hx = fmaf(R.d[1], t.e2[2], -R.d[2] * t.e2[1]);
  const float hy = fmaf(R.d[2], t.e2[0], -R.d[0] * t.e2[2]);
  const float hz = fmaf(R.d[0], t.e2[1], -R.d[1] * t.e2[0]);
  const float a = fmaf(t.e1[0], hx, fmaf(t.e1[1], hy, t.e1[2] * hz));
  const float na = n1 * n2, Ea = tol.e0 * na;
  const float aa = fabsf(a), hi = aa + Ea, lo = aa - Ea;
  if (hi < 1e-10f) return kMiss;
  if (lo < 1e-10f) return kUnsure;
  const float sx = R.o[0] - t.v0[0], sy = R.o[1] - t.v0[1], sz = R.o[2] - t.v0[2];
  const float d2 = tol.d * R.delta;
  const float e = fmaf(tol.e0, fabsf(sx) + fabsf(sy) + fabsf(sz) + d2, d2), e2 = e + d2;
  const float u = copysignf(1.0f, a) * fmaf(sx, hx, fmaf(sy, hy, sz * hz));
  const float cu = e * n2;
  if (u < -cu || u > hi + cu) return kMiss;
  const float qx = fmaf(sy, t.e1[2], -sz * t.e1[1]);
  const float qy = fmaf(sz, t.e1[0], -sx * t.e1[2]);
  const float qz = fmaf(sx, t.e1[1], -sy * t.e1[0]);
  const float v = copysignf(1.0f, a) * fmaf(R.d[0], qx, fmaf(R.d[1], qy, R.d[2] * qz));
  const float cv = e2 * n1, cuv = cu + cv + 1e-6f * aa;
  if (v < -cv || u + v > hi + cuv) return kMiss;
  const float w = copysignf(1.0f, a) * fmaf(t.e2[0], qx, fmaf(t.e2[1], qy, t.e2[2] * qz));
  const float cw = e2 * na;
  const float eps = (float)kTEps, tm = 2.0f * kRho * R.tmax;
  if (w + cw < (1.0f - tol.e0) * eps * lo || w - cw > (R.tmax + tm) * hi) return kMiss;
  const bool inside = u > cu && u < lo - cu && v > cv && u + v < lo - cuv;
  return inside && w - cw > (1.0f + tol.e0) * eps * hi && w + cw < (R.tmax - tm) * lo ? kHit : kUnsure;
}

// Warp-coherent FP32 any-hit traversal (same walk as packet_any_hit) with
// certified decisions.  A lane leaves the walk at its first uncertain
// decision (unsure = true); its ray must then be traced in FP64.
template <typename LeafF>
__device__ __forceinline__ bool packet_any_hit_f(bool alive, const NodeF* __restrict__ nodes, int n_nodes,
                                                 const RayF& R, LeafF leaf, bool& unsure, TravCount& cnt) {
  bool hit = false;
  unsure = false;
  int wake = 0, node = 0;
  if (!__any_sync(kFull, alive)) return false;
  while (node < n_nodes) {
    const NodeF nd = nodes[node];
    const bool live = alive && !hit && !unsure;
    bool act = live && node >= wake;
    unsigned am = __ballot_sync(kFull, act);
    if (am == 0) {
      node = __reduce_min_sync(kFull, live ? wake : n_nodes);
      continue;
    }
    cnt.nodes += act ? 1 : 0;
    int s = act ? slab_f(nd, R) : kMiss;
    if (s == kUnsure) {
      unsure = true;
      ++cnt.unsure_slab;
    }
    bool sh = (s == kHit);
    unsigned hm = __ballot_sync(kFull, sh);
    const int cntp = nd.ab & 15, first = nd.ab >> 4;
    if (cntp > 0) {
      if (hm) {
        for (int k = first; k < first + cntp; ++k) {
          int r = leaf(k, sh && !hit && !unsure);
          if (r == kHit) hit = true;
          else if (r == kUnsure) {
            unsure = true;
            ++cnt.unsure_prim;
          }
        }
      }
      node = nd.miss;
    } else {
      if (hm) {
        if (act && s == kMiss) wake = nd.miss;
        node = node + 1;
      } else {
        node = nd.miss;
      }
    }
    if (!__any_sync(kFull, alive && !hit && !unsure)) break;
  }
  return hit;
}

}  // namespace rvf
