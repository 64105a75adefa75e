// device_hull.cuh -- the hull of a tile (the convex hull of the centroid boxes
// of its two element blocks) and certified tests of boxes and triangles
// against it: what is farther from the hull than the blocks' point radii no
// ray of the tile can reach.
#pragma once

#include "device_lists.cuh"

namespace rvf {

// Position of the n-th (from 0) set bit of m (n < popc(m)): binary search
// over halves by population count.
__device__ __forceinline__ int nth_set_bit(uint32_t m, int n) {
  int pos = 0;
#pragma unroll
  for (int s = 16; s >= 1; s >>= 1) {
    const int c = __popc(m & ((1u << s) - 1u));
    if (n >= c) {
      n -= c;
      m >>= s;
      pos += s;
    }
  }
  return pos;
}

// H = conv(B_1 u B_2) of two boxes (FP32 centres c and half extents h).
struct HullF {
  float c[2][3], h[2][3];
  float d[3];  // c[1] - c[0]
};

// The hull of a tile: the centroid boxes of its two blocks (lanes = elements
// of each block), rounded outwards to FP32; rmax / rj_max the largest point
// radius of both blocks / of the column block.  Warp-uniform results.
__device__ __forceinline__ void tile_hull(bool oki, bool okj, const double* ci, const double* cj, double ri, double rj,
                                          HullF& H, double& rmax, double& rj_max) {
  double lo[2][3], hi[2][3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    lo[0][c] = oki ? ci[c] : INFINITY;
    hi[0][c] = oki ? ci[c] : -INFINITY;
    lo[1][c] = okj ? cj[c] : INFINITY;
    hi[1][c] = okj ? cj[c] : -INFINITY;
  }
  rmax = fmax(ri, rj);
  rj_max = rj;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        lo[b][c] = fmin(lo[b][c], __shfl_xor_sync(kFull, lo[b][c], o));
        hi[b][c] = fmax(hi[b][c], __shfl_xor_sync(kFull, hi[b][c], o));
      }
    rmax = fmax(rmax, __shfl_xor_sync(kFull, rmax, o));
    rj_max = fmax(rj_max, __shfl_xor_sync(kFull, rj_max, o));
  }
#pragma unroll
  for (int b = 0; b < 2; ++b)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float l = __double2float_rd(lo[b][c]), h = __double2float_ru(hi[b][c]);
      H.c[b][c] = 0.5f * (l + h);
      H.h[b][c] = 0.5f * (h - l);
    }
#pragma unroll
  for (int c = 0; c < 3; ++c) H.d[c] = H.c[1][c] - H.c[0][c];
}

// Projection interval of the hull on w.
__device__ __forceinline__ void hull_proj(const HullF& H, float wx, float wy, float wz, float& lo, float& hi) {
  const float aw0 = fabsf(wx), aw1 = fabsf(wy), aw2 = fabsf(wz);
  const float m0 = fmaf(H.c[0][0], wx, fmaf(H.c[0][1], wy, H.c[0][2] * wz));
  const float r0 = fmaf(H.h[0][0], aw0, fmaf(H.h[0][1], aw1, H.h[0][2] * aw2));
  const float m1 = fmaf(H.c[1][0], wx, fmaf(H.c[1][1], wy, H.c[1][2] * wz));
  const float r1 = fmaf(H.h[1][0], aw0, fmaf(H.h[1][1], aw1, H.h[1][2] * aw2));
  lo = fminf(m0 - r0, m1 - r1);
  hi = fmaxf(m0 + r0, m1 + r1);
}

// True when the interval [qlo, qhi] lies farther than m |w| from the hull
// along w (squares avoid the square root; m > 0).
__device__ __forceinline__ bool hull_gap(const HullF& H, float wx, float wy, float wz, float qlo, float qhi,
                                         float m) {
  float lo, hi;
  hull_proj(H, wx, wy, wz, lo, hi);
  const float gap = fmaxf(qlo - hi, lo - qhi);
  return gap > 0.0f && gap * gap > m * m * fmaf(wx, wx, fmaf(wy, wy, wz * wz));
}

// True when every point of the box lies farther than m from the hull.
__device__ __forceinline__ bool hull_misses_box(const HullF& H, const NodeF& nd, float m) {
  // coordinate axes
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float lo = fminf(H.c[0][k] - H.h[0][k], H.c[1][k] - H.h[1][k]);
    const float hi = fmaxf(H.c[0][k] + H.h[0][k], H.c[1][k] + H.h[1][k]);
    if (nd.lo[k] - hi > m || lo - nd.hi[k] > m) return true;
  }
  // the centroid direction crossed with each coordinate axis
  const float bc[3] = {0.5f * (nd.lo[0] + nd.hi[0]), 0.5f * (nd.lo[1] + nd.hi[1]), 0.5f * (nd.lo[2] + nd.hi[2])};
  const float bh[3] = {0.5f * (nd.hi[0] - nd.lo[0]), 0.5f * (nd.hi[1] - nd.lo[1]), 0.5f * (nd.hi[2] - nd.lo[2])};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    float w[3] = {0.f, 0.f, 0.f};  // d x e_k
    w[(k + 1) % 3] = H.d[(k + 2) % 3];
    w[(k + 2) % 3] = -H.d[(k + 1) % 3];
    const float bm = fmaf(bc[0], w[0], fmaf(bc[1], w[1], bc[2] * w[2]));
    const float br = fmaf(bh[0], fabsf(w[0]), fmaf(bh[1], fabsf(w[1]), bh[2] * fabsf(w[2])));
    if (hull_gap(H, w[0], w[1], w[2], bm - br, bm + br, m)) return true;
  }
  return false;
}

__device__ __forceinline__ void tri_proj(const float4& p0, const float4& p1, const float4& p2, float wx, float wy,
                                         float wz, float& lo, float& hi) {
  const float q0 = fmaf(p0.x, wx, fmaf(p0.y, wy, p0.z * wz));
  const float q1 = fmaf(p1.x, wx, fmaf(p1.y, wy, p1.z * wz));
  const float q2 = fmaf(p2.x, wx, fmaf(p2.y, wy, p2.z * wz));
  lo = fminf(q0, fminf(q1, q2));
  hi = fmaxf(q0, fmaxf(q1, q2));
}

// True when the triangle lies farther than m from the hull.
__device__ __forceinline__ bool hull_misses_tri(const HullF& H, const float4& p0, const float4& p1, const float4& p2,
                                                float m) {
  float lo, hi;
  // coordinate axes
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float w[3] = {k == 0 ? 1.f : 0.f, k == 1 ? 1.f : 0.f, k == 2 ? 1.f : 0.f};
    tri_proj(p0, p1, p2, w[0], w[1], w[2], lo, hi);
    if (hull_gap(H, w[0], w[1], w[2], lo, hi, m)) return true;
  }
  const float e[3][3] = {{p1.x - p0.x, p1.y - p0.y, p1.z - p0.z},
                         {p2.x - p0.x, p2.y - p0.y, p2.z - p0.z},
                         {p2.x - p1.x, p2.y - p1.y, p2.z - p1.z}};
  // the normal
  {
    const float nx = e[0][1] * e[1][2] - e[0][2] * e[1][1];
    const float ny = e[0][2] * e[1][0] - e[0][0] * e[1][2];
    const float nz = e[0][0] * e[1][1] - e[0][1] * e[1][0];
    tri_proj(p0, p1, p2, nx, ny, nz, lo, hi);
    if (hull_gap(H, nx, ny, nz, lo, hi, m)) return true;
  }
  // the edges crossed with the centroid direction and with the coordinate axes
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float* f = e[a];
    {
      const float* d = H.d;
      const float wx = d[1] * f[2] - d[2] * f[1], wy = d[2] * f[0] - d[0] * f[2], wz = d[0] * f[1] - d[1] * f[0];
      tri_proj(p0, p1, p2, wx, wy, wz, lo, hi);
      if (hull_gap(H, wx, wy, wz, lo, hi, m)) return true;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      float w[3] = {0.f, 0.f, 0.f};  // e_k x f
      w[(k + 1) % 3] = -f[(k + 2) % 3];
      w[(k + 2) % 3] = f[(k + 1) % 3];
      tri_proj(p0, p1, p2, w[0], w[1], w[2], lo, hi);
      if (hull_gap(H, w[0], w[1], w[2], lo, hi, m)) return true;
    }
  }
  return false;
}

}  // namespace rvf
