// device_pairs.cuh -- pair-level building blocks shared by the generation
// (kernels_wave.cu) and the occlusion kernel (kernels_occ.cu): table access,
// the capsule-against-root test and the quadrature of pairs whose rays are all
// visible.
#pragma once

#include "device_lists.cuh"
#include "kernels.h"

namespace rvf {

// (element e, component c, point p) in a tile-blocked table
__device__ __forceinline__ int64_t tab_at(int64_t e, int c, int p, int pm) {
  return ((e >> 5) * kComp + c) * (int64_t)pm * kTile + (int64_t)p * kTile + (e & 31);
}

// True when every segment between a point of element i and a point of
// element j certainly misses the box: each such segment stays within
// R = max(rad_i, rad_j) of the centroid segment (convexity), so it suffices
// that the centroid segment misses the box grown by R plus a margin that
// dwarfs every rounding error of the reference's slab test.  2-D uses x, y.
template <bool DIM3>
__device__ __forceinline__ bool pair_misses_box(const double* ci, const double* cj, double R, const NodeD& nd) {
  double te = 0.0, tx = 1.0;
#pragma unroll
  for (int c = 0; c < (DIM3 ? 3 : 2); ++c) {
    const double lo = nd.lo[c] - R, hi = nd.hi[c] + R;
    const double d = cj[c] - ci[c];
    if (d == 0.0) {
      if (ci[c] < lo || ci[c] > hi) return true;
      continue;
    }
    const double inv = 1.0 / d;
    const double t1 = (lo - ci[c]) * inv, t2 = (hi - ci[c]) * inv;
    te = fmax(te, fmin(t1, t2));
    tx = fmin(tx, fmax(t1, t2));
  }
  return te > tx;
}

// request r of the launch with tile_base[r] <= t < tile_base[r+1]
__device__ __forceinline__ int find_req(const int64_t* tile_base, int n_req, int64_t t) {
  int lo = 0, hi = n_req - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (tile_base[mid] <= t) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// ---------------------------------------------------------------------------
// 1a. Generation of a tile without shadow-ray work (the tile classification
// found no pair whose rays may be blocked, or the mesh has no obstruction):
// the quadrature alone, register-blocked.  Lane l owns destination
// j = 32 bj + l and holds QB of its points in registers; the warp walks the
// source element's points p, read once per QB point pairs from the staged
// block in shared memory (broadcast), so each point pair costs the kernel's
// arithmetic and about 7/QB shared loads.  Sums run in the pipeline's order
// (over p inside, then w_q * inner over q), so an FP64 fast tile is bit for
// bit what the ray pipeline gives for pairs whose rays are all visible.
// Out of line: their registers are allocated apart from the ray pipeline's.
// ---------------------------------------------------------------------------
// FP64 arithmetic.  Per point pair the FP64 pipe runs r (3), r^2 (3), the two
// cosines' numerators (6), their product, r^4, the reciprocal (two steps) and
// the two multiply-adds into the sum: 19 instructions, 36 before, when r^2 was
// formed as the shadow rays form it, the reciprocal took two Newton steps and
// signs and grazing were compared on the FP64 pipe; 1 / pi is applied once per
// pair.  Signs and the grazing test read the high words as integers.  Bound by
// the FP64 pipe (about half of its cycles) and instruction issue.  Measured, one
// solve, before -> now: cylinder of 3,072 Quad8, nquad 5 (curved) 13.6 -> 8.6 ms;
// 800 Quad4, nquad 4 (a quarter of the point pairs graze) 0.53 -> 0.39 ms; the
// closed cube of 43,200 Tri3 (all plane) 163 -> 91 ms with its masked tiles' rest.
//
// 1 / x from rcp.approx.ftz.f64 (operand and result cut to 20 mantissa bits:
// relative error e0 below 2^-18.9): with e = 1 - x y, 1 / x = y (1 + e + e^2 + ...),
// cut after e^2 (e^3 < 2^-56).  x^-3/2 from rsqrt.approx.ftz.f64 likewise, with
// e = 1 - x y^2: y^3 (1 + 3/2 e + 15/8 e^2 + 35/16 e^3).
__device__ __forceinline__ double recip_scaled(double k, double x) {  // k / x
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0), k0 = k * y;
  return fma(k0, fma(e, e, e), k0);
}
__device__ __forceinline__ double recip32_scaled(double k, double x) {  // k x^-3/2
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double s = y * y, e = fma(-x, s, 1.0), k0 = k * (y * s);
  return fma(k0, e * fma(fma(2.1875, e, 1.875), e, 1.5), k0);
}

// s += w k when the sign bit of `both` is clear (di >= 0 and dj < 0), as one predicated instruction.
__device__ __forceinline__ void fma_if_facing(double& s, double w, double k, int both) {
  asm("{\n .reg .pred f;\n setp.ge.s32 f, %3, 0;\n @f fma.rn.f64 %0, %1, %2, %0;\n}" : "+d"(s) : "d"(w), "d"(k), "r"(both));
}

// Pairs of plane elements (one normal each) that are at least eight of their
// sizes apart: the cosine at a point depends on that point alone --
// n_i.(x_q - x_p) is the same for every p, up to the rounding of the element's
// points -- so a point pair costs r, r^2, 1 / r^4 and one multiply-add, 11
// FP64 instructions instead of 19, and no sign or grazing test.  A pair with a
// |cos| below 1e-3 (d^2 <= limit for some d; limit = 1e-6 of the largest
// possible r^2), or a point within 1e-4 M of the other element's plane (M: the
// mesh's largest coordinate), is left to the general loop.  A point of an element is
// rounded by up to 10 2^-53 M along the normal, for which the d of one point and of
// another differ: by 1.2e-11 of d at 1e-4 M, 2.4e-11 in the product of two, against the
// written 1e-10.  Cube of 588 Tri3 1e4 / 1e5 from the origin: off by 2.3e-12 /
// 1.3e-15, by 3.5e-11 / 3.5e-10 without the second bound.
struct FlatSum {
  double sum;  // pi times the pair's sum
  uint32_t cast;
  bool done;
};
template <int QB>
__device__ __noinline__ FlatSum flat_fp64_q(const double* S, const double* jb, int pm, int npi, int npj,
                                            double limit) {
  double ni[3], nj[3], xi0[3], xj0[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    xi0[c] = S[c];
    ni[c] = S[4 + c];
    xj0[c] = npj > 0 ? jb[c * pm * kTile] : 0.0;
    nj[c] = npj > 0 ? jb[(3 + c) * pm * kTile] : 0.0;
  }
  const int qmax = __reduce_max_sync(kFull, npj);
  double acc = 0.0;
  int pos_i = 0, pos_j = 0;
  bool ok = npj > 0;
  for (int q0 = 0; q0 < qmax; q0 += QB) {
    double x[QB][3], inner[QB];
#pragma unroll
    for (int u = 0; u < QB; ++u) {
      const int q = q0 + u < npj ? q0 + u : 0;  // past the element's points: the first again, not summed
#pragma unroll
      for (int c = 0; c < 3; ++c) x[u][c] = npj > 0 ? jb[(c * pm + q) * kTile] : 1.0;
      inner[u] = 0.0;
    }
    for (int p = 0; p < npi; ++p) {
      const double2 s0 = *reinterpret_cast<const double2*>(S + 8 * p), s1 = *reinterpret_cast<const double2*>(S + 8 * p + 2);
      const double x0 = s0.x, x1 = s0.y, x2 = s1.x;
      const double dj = fma(nj[0], x0 - xj0[0], fma(nj[1], x1 - xj0[1], nj[2] * (x2 - xj0[2])));
      const bool facing = __double2hiint(dj) >= 0;
      const double w = facing ? s1.y * dj : 0.0;
      if (q0 == 0) {
        ok = ok && dj * dj > limit;
        pos_j += facing ? 1 : 0;
      }
#pragma unroll
      for (int u = 0; u < QB; ++u) {
        const double rx = x[u][0] - x0, ry = x[u][1] - x1, rz = x[u][2] - x2;
        const double r2 = fma(rx, rx, fma(ry, ry, rz * rz)), r4 = r2 * r2;
        double y;
        asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(r4));
        const double e = fma(-r4, y, 1.0);
        inner[u] = fma(w, fma(y, fma(e, e, e), y), inner[u]);
      }
    }
#pragma unroll
    for (int u = 0; u < QB; ++u) {
      if (q0 + u < npj) {
        const double di = fma(ni[0], x[u][0] - xi0[0], fma(ni[1], x[u][1] - xi0[1], ni[2] * (x[u][2] - xi0[2])));
        ok = ok && di * di > limit;
        if (__double2hiint(di) >= 0) {
          acc = fma(jb[(6 * pm + q0 + u) * kTile] * di, inner[u], acc);
          ++pos_i;
        }
      }
    }
  }
  return FlatSum{acc, (uint32_t)(pos_i * pos_j), ok};
}
// The point block by the rule's size: no or few idle points (7: 7, 13 and 49
// points; 5: 5 and 25; 3: 3 and 9; 4: 4, 16, 36, 64, and the others).
__device__ __forceinline__ FlatSum flat_fp64(const double* S, const double* jb, int pm, int npi, int npj,
                                             double limit) {
  if (pm == 7 || pm == 13 || pm == 49) return flat_fp64_q<7>(S, jb, pm, npi, npj, limit);
  if (pm == 5 || pm == 25) return flat_fp64_q<5>(S, jb, pm, npi, npj, limit);
  if (pm == 3 || pm == 9) return flat_fp64_q<3>(S, jb, pm, npi, npj, limit);
  return flat_fp64_q<4>(S, jb, pm, npi, npj, limit);
}

// shared memory of a block's eight staged rows
__host__ __device__ __forceinline__ size_t stage_bytes(int pmax) { return (size_t)8 * 8 * pmax * sizeof(double); }

// The source element's points for the warp's loops: eight doubles a point (x, y,
// z, w, n) in shared memory, read by broadcast 16-byte loads from one address,
// where the table's component-major layout costs a load and an address per value.
__device__ __forceinline__ void stage_row(const double* ib, double* S, int pm) {
  const int lane = threadIdx.x & 31;
  const float per = 1.0f / (float)pm;  // v + 1/2 is at least 1/128 from a multiple of pm, v < 448
  __syncwarp();                        // the previous row's readers
  for (int v = lane; v < kComp * pm; v += 32) {
    const int c = (int)(((float)v + 0.5f) * per), p = v - c * pm;
    S[8 * p + (c < 3 ? c : c == 6 ? 3 : c + 1)] = ib[v * kTile];
  }
  __syncwarp();
}

// pi K (3-D) or 2 K (2-D) of one point pair, r2 as the shadow rays form it: the
// fast form, or the reference's cosines where one grazes (their product over the
// distance needs no correctly rounded quotient).
template <bool DIM3>
__device__ __forceinline__ double kernel_scaled(double rx, double ry, double rz, double r2, const double* ni,
                                                const double* nj) {
  if (r2 < 1e-30) return 0.0;
  const double di = fma(ni[0], rx, fma(ni[1], ry, ni[2] * rz));
  const double dj = -fma(nj[0], rx, fma(nj[1], ry, nj[2] * rz));
  const double thr = 1e-10 * r2;
  if (di * di <= thr || dj * dj <= thr) {
    double ci, cj, r;
    reference_cosines(rx, ry, rz, r2, ni, nj, ci, cj, r);
    return ci > 0.0 && cj > 0.0 ? recip_scaled(ci * cj, DIM3 ? r2 : r) : 0.0;
  }
  if (di <= 0.0 || dj <= 0.0) return 0.0;
  return DIM3 ? recip_scaled(di * dj, r2 * r2) : recip32_scaled(di * dj, r2);
}

// One column (point q of the lane's element, all points p of the source) with
// kernel_scaled, which takes the reference formula at grazing point pairs.
struct ColumnSum {
  double inner;  // scaled as the fast loop's
  uint32_t cast;
};
template <bool DIM3>
__device__ __noinline__ ColumnSum column_exact(const double* ib, const double* jq, int pm, int npi) {
  ColumnSum s{0.0, 0};
  double xj[3], nj[3];
  for (int c = 0; c < 3; ++c) {
    xj[c] = jq[c * pm * kTile];
    nj[c] = jq[(3 + c) * pm * kTile];
  }
#pragma unroll 2
  for (int p = 0; p < npi; ++p) {
    double xi[3], ni[3];
    for (int c = 0; c < 3; ++c) {
      xi[c] = ib[(c * pm + p) * kTile];
      ni[c] = ib[((3 + c) * pm + p) * kTile];
    }
    const double rx = xj[0] - xi[0], ry = xj[1] - xi[1], rz = xj[2] - xi[2];
    const double r2 = (rx * rx + ry * ry) + rz * rz;
    const double k = kernel_scaled<DIM3>(rx, ry, rz, r2, ni, nj);
    s.cast += k > 0.0 ? 1 : 0;
    s.inner = fma(ib[(6 * pm + p) * kTile], -k, s.inner);
  }
  return s;
}

// PLANE: pairs of plane elements by flat_fp64 first.
template <bool DIM3, bool OCC, int QB, bool PLANE = DIM3>
__device__ __forceinline__ void gen_fast_fp64_body(const PairArgs& a, const double* iblk, double* S, int64_t bi,
                                                   int64_t bj, int li0, int lane, uint32_t& n_pp, uint32_t& n_rays,
                                                   uint32_t skip = 0) {
  const int64_t N = a.N;
  const int pm = a.pmax;
  const int64_t j = bj * kTile + lane;
  const bool jok = j < N;
  const int64_t oj = jok ? (a.orig ? (int64_t)a.orig[j] : j) : 0;
  const int npj0 = jok ? a.np[j] : 0;
  const double* jb = a.tab + bj * kComp * pm * kTile + lane;
  // li0 < 8: the warp's rows li0, li0 + 8, ...; li0 >= 8: the single row li0 - 8
  const int r_last = li0 < 8 ? kTile / 8 : 1;
  for (int rr = 0; rr < r_last; ++rr) {
    const int li = li0 < 8 ? li0 + 8 * rr : li0 - 8;
    const int64_t i = bi * kTile + li;
    if (i >= N) break;  // warp-uniform; later rows are further out
    const bool valid = jok && i < j && !((skip >> lane) & 1u);
    const int64_t oi = a.orig ? (int64_t)a.orig[i] : i;
    const int npi = a.np[i];
    int npj = valid ? npj0 : 0;
    if (valid && a.flat[i] && a.flat[j] && a.nrm[3 * i] == a.nrm[3 * j] && a.nrm[3 * i + 1] == a.nrm[3 * j + 1] &&
        a.nrm[3 * i + 2] == a.nrm[3 * j + 2])
      npj = 0;
    // every distance of the pair's points lies within s of |c_j - c_i|
    double d2 = 0.0, s2 = 0.0;
    if (npj > 0) {
      const double dx = a.cen[3 * j] - a.cen[3 * i], dy = a.cen[3 * j + 1] - a.cen[3 * i + 1],
                   dz = a.cen[3 * j + 2] - a.cen[3 * i + 2];
      const double s = a.rad[i] + a.rad[j];
      d2 = dx * dx + dy * dy + dz * dz;
      s2 = s * s;
    }
    const double* ib = iblk + li;
    stage_row(ib, S, pm);
    double acc = 0.0;  // minus pi (3-D) or 2 (2-D) times the pair's sum
    n_pp += (uint32_t)(npi * npj);
    if constexpr (PLANE) {
      const int npf = npj > 0 && a.flat[i] && a.flat[j] && d2 > 64.0 * s2 ? npj : 0;
      if (__any_sync(kFull, npf > 0)) {
        const FlatSum f = flat_fp64(S, jb, pm, npi, npf, fmax(1.27e-6 * d2, a.plane_dist2));
        if (f.done) {
          acc = -f.sum;
          if (OCC) n_rays += f.cast;
          npj = 0;
        }
      }
    }
    // points of the pair may nearly coincide: every column with k_fast's own arithmetic
    const bool tiny = !(d2 > 1.0001 * s2 + 1e-28);
    // no |cos| is below 1e-5 when every |d| exceeds 1e-5 of the largest distance
    // (hi words, so the threshold is rounded up by one)
    const int graze = __double2hiint(1e-5 * sqrt(2.0 * (d2 + s2))) + 1;
    const int qmax = __reduce_max_sync(kFull, npj);
    for (int q0 = 0; q0 < qmax; q0 += QB) {
      double xq[QB][3], nq[QB][3];
#pragma unroll
      for (int u = 0; u < QB; ++u) {
        // past the element's points: the first one again (finite, not summed)
        const int q = q0 + u < npj ? q0 + u : 0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          xq[u][c] = jok ? jb[(c * pm + q) * kTile] : 0.0;
          nq[u][c] = jok ? jb[((3 + c) * pm + q) * kTile] : 0.0;
        }
      }
      double inner[QB];
      int least[QB];      // smallest hi|d| of the column
      uint32_t cast[QB];
#pragma unroll
      for (int u = 0; u < QB; ++u) {
        inner[u] = 0.0;
        least[u] = 0x7fffffff;
        cast[u] = 0;
      }
      for (int p = 0; p < npi; ++p) {
        const double2* s = reinterpret_cast<const double2*>(S + 8 * p);
        const double2 s0 = s[0], s1 = s[1], s2v = s[2];
        const double xi[3] = {s0.x, s0.y, s1.x}, ni[3] = {s2v.x, s2v.y, S[8 * p + 6]};
        const double wi = s1.y;
#pragma unroll
        for (int u = 0; u < QB; ++u) {
          const double rx = xq[u][0] - xi[0], ry = xq[u][1] - xi[1], rz = xq[u][2] - xi[2];
          const double r2 = fma(rx, rx, fma(ry, ry, rz * rz));
          const double di = fma(ni[0], rx, fma(ni[1], ry, ni[2] * rz));
          const double dj = fma(nq[u][0], rx, fma(nq[u][1], ry, nq[u][2] * rz));  // minus the reference's
          const int hi = __double2hiint(di), hj = __double2hiint(dj), both = hi | ~hj;
          least[u] = min(least[u], min(hi & 0x7fffffff, hj & 0x7fffffff));
          const double K = DIM3 ? recip_scaled(di * dj, r2 * r2) : recip32_scaled(di * dj, r2);
          fma_if_facing(inner[u], wi, K, both);
          if (OCC) cast[u] += (uint32_t)~both >> 31;
        }
      }
#pragma unroll
      for (int u = 0; u < QB; ++u) {
        // a column with a grazing point pair (a |cos| within 1e-5 of zero, where
        // the sign of the fast form could differ from the reference's) again
        const bool again = q0 + u < npj && (tiny || least[u] <= graze);
        if (__any_sync(kFull, again) && again) {
          const ColumnSum c = column_exact<DIM3>(ib, jb + (q0 + u) * kTile, pm, npi);
          inner[u] = c.inner;
          cast[u] = c.cast;
        }
        if (q0 + u < npj) {
          acc = fma(jb[(6 * pm + q0 + u) * kTile], inner[u], acc);
          if (OCC) n_rays += cast[u];
        }
      }
    }
    if (valid) {
      const double raw = fma(acc, DIM3 ? -1.0 / kPiD : -0.5, 0.0);  // (a sum of nothing is +0)
      a.F[oi + oj * N] = raw / a.area[i];
      a.F[oj + oi * N] = raw / a.area[j];
    } else if (j == i) {
      a.F[oi + oi * N] = 0.0 / a.area[i];
    }
  }
}

// a / b with y = 1 / b, rounded as the division
__device__ __forceinline__ double div_or(double a, double b, double y) {
  return div_by_ok(a) && div_by_ok(b) ? div_by(a, b, y) : a / b;
}

// The pairs of plane elements (flat_fp64) in the rows li0, li0 + 8, ... of a tile,
// for rules of at most QB points, in the kernel that only does this: the column's
// points are loaded once for the rows, which are staged together, and a row of pairs
// that are all done needs nothing else; the other rows run the general loop for what
// is left.  Same sums, bit for bit.  Bound by latency and FP64 issue.  Closed cube of
// 43,200 Tri3, 7 points, the tiles without ray work: 79 ms with flat_fp64 row by row
// (stalls on the column's points), 63 ms so.
constexpr int kFlatRows = kTile / 8;
template <bool OCC, int QB>
__device__ __forceinline__ void flat_rows(const PairArgs& a, const double* iblk, double* S, int64_t bi, int64_t bj,
                                          int li0, int lane, uint32_t& n_pp, uint32_t& n_rays) {
  const int64_t N = a.N;
  const int pm = a.pmax;
  const int64_t j = bj * kTile + lane, e = j < N ? j : bj * kTile;
  const bool jok = j < N;
  const int64_t oj = a.orig ? (int64_t)a.orig[e] : e;
  const int npj = jok ? a.np[j] : 0;
  const bool flat_j = a.flat[e];
  uint32_t left[kFlatRows] = {kFull, kFull, kFull, kFull};  // pairs the general loop takes
  if (__any_sync(kFull, flat_j)) {
    const double* jb = a.tab + bj * kComp * pm * kTile + (jok ? lane : 0);
    const double mj[3] = {a.nrm[3 * e], a.nrm[3 * e + 1], a.nrm[3 * e + 2]};
    const double cj[3] = {a.cen[3 * e], a.cen[3 * e + 1], a.cen[3 * e + 2]};
    const double rj = a.rad[e], aj = a.area[e], yj = 1.0 / aj;
    double x[QB][3], nj[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      nj[c] = jb[(3 + c) * pm * kTile];
#pragma unroll
      for (int u = 0; u < QB; ++u) x[u][c] = jb[(c * pm + (u < npj ? u : 0)) * kTile];  // past them: not summed
    }
    __syncwarp();
    for (int v = lane; v < kFlatRows * pm; v += 32) {
      const int rr = v / pm, q = v - rr * pm, li = li0 + 8 * rr;
      double* s = S + 8 * v;
      const double* ib = iblk + li + q * kTile;
#pragma unroll
      for (int c = 0; c < kComp; ++c) s[c < 3 ? c : c == 6 ? 3 : c + 1] = ib[c * pm * kTile];
    }
    __syncwarp();
#pragma unroll 1
    for (int rr = 0; rr < kFlatRows; ++rr) {
      const int li = li0 + 8 * rr;
      const int64_t i = bi * kTile + li;
      if (i >= N) continue;  // warp-uniform
      const double* Sr = S + 8 * rr * pm;
      const bool valid = jok && i < j;
      const double dx = cj[0] - a.cen[3 * i], dy = cj[1] - a.cen[3 * i + 1], dz = cj[2] - a.cen[3 * i + 2];
      const double s = a.rad[i] + rj, d2 = dx * dx + dy * dy + dz * dz;
      const bool flat_i = a.flat[i];
      const bool same =
          flat_i && flat_j && a.nrm[3 * i] == mj[0] && a.nrm[3 * i + 1] == mj[1] && a.nrm[3 * i + 2] == mj[2];
      bool ok = valid && flat_i && flat_j && npj > 0 && !same && d2 > 64.0 * (s * s);
      if (__any_sync(kFull, ok)) {
        const int npi = a.np[i];
        const double limit = fmax(1.27e-6 * d2, a.plane_dist2);
        double inner[QB];
#pragma unroll
        for (int u = 0; u < QB; ++u) inner[u] = 0.0;
        int pos_i = 0, pos_j = 0;
        for (int p = 0; p < npi; ++p) {
          const double2* sp = reinterpret_cast<const double2*>(Sr + 8 * p);
          const double2 s0 = sp[0], s1 = sp[1];
          const double x0 = s0.x, x1 = s0.y, x2 = s1.x;
          const double dj = fma(nj[0], x0 - x[0][0], fma(nj[1], x1 - x[0][1], nj[2] * (x2 - x[0][2])));
          const bool facing = __double2hiint(dj) >= 0;
          const double w = facing ? s1.y * dj : 0.0;
          ok = ok && dj * dj > limit;
          pos_j += facing ? 1 : 0;
#pragma unroll
          for (int u = 0; u < QB; ++u) {
            const double rx = x[u][0] - x0, ry = x[u][1] - x1, rz = x[u][2] - x2;
            const double r2 = fma(rx, rx, fma(ry, ry, rz * rz)), r4 = r2 * r2;
            double y;
            asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(r4));
            const double er = fma(-r4, y, 1.0);
            inner[u] = fma(w, fma(y, fma(er, er, er), y), inner[u]);
          }
        }
        double acc = 0.0;
        const double xi[3] = {Sr[0], Sr[1], Sr[2]}, ni[3] = {Sr[4], Sr[5], Sr[6]};
#pragma unroll
        for (int u = 0; u < QB; ++u) {
          if (u < npj) {
            const double di = fma(ni[0], x[u][0] - xi[0], fma(ni[1], x[u][1] - xi[1], ni[2] * (x[u][2] - xi[2])));
            ok = ok && di * di > limit;
            if (__double2hiint(di) >= 0) {
              acc = fma(jb[(6 * pm + u) * kTile] * di, inner[u], acc);
              ++pos_i;
            }
          }
        }
        if (ok) {
          n_pp += (uint32_t)(npi * npj);
          if (OCC) n_rays += (uint32_t)(pos_i * pos_j);
          const double raw = acc * (1.0 / kPiD), ai = a.area[i];
          const int64_t oi = a.orig ? (int64_t)a.orig[i] : i;
          a.F[oi + oj * N] = div_or(raw, ai, 1.0 / ai);
          a.F[oj + oi * N] = div_or(raw, aj, yj);
        }
      }
      const uint32_t m = __ballot_sync(kFull, jok && i <= j && !ok);
      left[0] = rr == 0 ? m : left[0];
      left[1] = rr == 1 ? m : left[1];
      left[2] = rr == 2 ? m : left[2];
      left[3] = rr == 3 ? m : left[3];
    }
  }
#pragma unroll 1
  for (int rr = 0; rr < kFlatRows; ++rr) {
    const uint32_t m = rr == 0 ? left[0] : rr == 1 ? left[1] : rr == 2 ? left[2] : left[3];
    const int li = li0 + 8 * rr;
    if (m && bi * kTile + li < N)
      gen_fast_fp64_body<true, OCC, (QB < 4 ? 3 : 4), false>(a, iblk, S, bi, bj, 8 + li, lane, n_pp, n_rays, ~m);
  }
}

// Mixed precision: the FP32 far-field arithmetic of k_gen_mixed (offsets
// from the element centroids, FP32 per-pair sums), for tiles with neither
// near-field nor nearly coincident pairs.  Grazing point pairs stay in FP32
// here: no ray depends on the sign of their K, and their FP32 error is that
// of any other far-field term.
template <bool OCC, int QB>
__device__ __forceinline__ void gen_fast_mixed_body(const MixedArgs& a, const float* iblk, int64_t bi, int64_t bj,
                                                    int li0, int lane, uint32_t& n_pp, uint32_t& n_rays, uint32_t skip = 0) {
  const int64_t N = a.N;
  const int pm = a.pmax;
  const int64_t j = bj * kTile + lane;
  const bool jok = j < N;
  const int64_t oj = jok ? (a.orig ? (int64_t)a.orig[j] : j) : 0;
  const int npj0 = jok ? a.np[j] : 0;
  const float* jbf = a.tabf + bj * kComp * pm * kTile + lane;
  const double cj0 = jok ? a.cen[3 * j] : 0.0, cj1 = jok ? a.cen[3 * j + 1] : 0.0, cj2 = jok ? a.cen[3 * j + 2] : 0.0;
  // li0 < 8: the warp's rows li0, li0 + 8, ...; li0 >= 8: the single row li0 - 8
  const int r_last = li0 < 8 ? kTile / 8 : 1;
  for (int rr = 0; rr < r_last; ++rr) {
    const int li = li0 < 8 ? li0 + 8 * rr : li0 - 8;
    const int64_t i = bi * kTile + li;
    if (i >= N) break;  // warp-uniform
    const bool valid = jok && i < j && !((skip >> lane) & 1u);
    const int64_t oi = a.orig ? (int64_t)a.orig[i] : i;
    const int npi = a.np[i];
    int npj = valid ? npj0 : 0;
    if (valid && a.flat[i] && a.flat[j] && a.nrm[3 * i] == a.nrm[3 * j] && a.nrm[3 * i + 1] == a.nrm[3 * j + 1] &&
        a.nrm[3 * i + 2] == a.nrm[3 * j + 2])
      npj = 0;
    const int qmax = __reduce_max_sync(kFull, npj);
    const float d0 = (float)(cj0 - a.cen[3 * i]), d1 = (float)(cj1 - a.cen[3 * i + 1]),
                d2 = (float)(cj2 - a.cen[3 * i + 2]);
    const float* ibf = iblk + li;
    float acc32 = 0.0f;
    uint32_t cast = 0;
    for (int q0 = 0; q0 < qmax; q0 += QB) {
      float oq[QB][3], nq[QB][3], wq[QB];
#pragma unroll
      for (int u = 0; u < QB; ++u) {
        const int q = q0 + u;
        const bool lq = q < npj;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          oq[u][c] = lq ? jbf[(c * pm + q) * kTile] : 0.0f;
          nq[u][c] = lq ? jbf[((3 + c) * pm + q) * kTile] : 0.0f;
        }
        wq[u] = lq ? jbf[(6 * pm + q) * kTile] : 0.0f;
      }
      float inner[QB];
#pragma unroll
      for (int u = 0; u < QB; ++u) inner[u] = 0.0f;
      for (int p = 0; p < npi; ++p) {
        const float op0 = ibf[(0 * pm + p) * kTile], op1 = ibf[(1 * pm + p) * kTile], op2 = ibf[(2 * pm + p) * kTile];
        const float np0 = ibf[(3 * pm + p) * kTile], np1 = ibf[(4 * pm + p) * kTile], np2 = ibf[(5 * pm + p) * kTile];
        const float wp = ibf[(6 * pm + p) * kTile];
        // straight-line over the block: a point q0 + u >= npj has zero
        // normal, so its dj is -0 and its K zero
#pragma unroll
        for (int u = 0; u < QB; ++u) {
          const float rx = d0 + (oq[u][0] - op0), ry = d1 + (oq[u][1] - op1), rz = d2 + (oq[u][2] - op2);
          const float r2 = fmaf(rx, rx, fmaf(ry, ry, rz * rz));
          const float di = fmaf(np0, rx, fmaf(np1, ry, np2 * rz));
          const float dj = -fmaf(nq[u][0], rx, fmaf(nq[u][1], ry, nq[u][2] * rz));
          const float K32 = (di > 0.0f && dj > 0.0f) ? (di * dj) * rcp_approx(3.14159265f * (r2 * r2)) : 0.0f;
          cast += K32 > 0.0f ? 1 : 0;
          inner[u] = fmaf(wp, K32, inner[u]);
        }
      }
#pragma unroll
      for (int u = 0; u < QB; ++u)
        if (q0 + u < npj) acc32 = fmaf(wq[u], inner[u], acc32);
    }
    if (OCC) n_rays += cast;
    n_pp += (uint32_t)(npi * npj);
    const double raw = 0.0 + (double)acc32;
    if (valid) {
      a.F[oi + oj * N] = raw / a.area[i];
      a.F[oj + oi * N] = raw / a.area[j];
    } else if (j == i) {
      a.F[oi + oi * N] = 0.0 / a.area[i];
    }
  }
}

// Two FP32 values in a register pair: one instruction does both operations, each
// rounded as the scalar one.
using F32x2 = unsigned long long;
__device__ __forceinline__ F32x2 f2_pack(float x, float y) {
  F32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ void f2_unpack(F32x2 a, float& x, float& y) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a));
}
__device__ __forceinline__ F32x2 f2_add(F32x2 a, F32x2 b) {
  F32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ F32x2 f2_mul(F32x2 a, F32x2 b) {
  F32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ F32x2 f2_fma(F32x2 a, F32x2 b, F32x2 c) {
  F32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// The same in the kernel that only does this:
// two of the column's points per instruction (packed FP32), the row's points in
// shared memory S with every value twice, so that an operand is a load, and the
// column's points kept in registers over the rows when one block holds them.  Every
// operation rounds as in gen_fast_mixed_body.  Bound by the FP32 pipes' non-packed
// operations (comparisons, selections, reciprocals).  Closed cube of 43,200 Tri3, 7
// points, the tiles without ray work: 56.1 ms with gen_fast_mixed_body, 55 with
// packed operations alone (long waits for the row's points from global memory), 44 ms
// so; single rows (k_occ_rest) gain nothing (+5 of 16 ms).
template <bool OCC, int QB>
__device__ __forceinline__ void fast_mixed_rows(const MixedArgs& a, const float* iblk, double* S, int64_t bi, int64_t bj,
                                                int li0, int lane, uint32_t& n_pp, uint32_t& n_rays) {
  const int64_t N = a.N;
  const int pm = a.pmax;
  const int64_t j = bj * kTile + lane;
  const bool jok = j < N;
  const int64_t oj = jok ? (a.orig ? (int64_t)a.orig[j] : j) : 0;
  const int npj0 = jok ? a.np[j] : 0;
  const float* jbf = a.tabf + bj * kComp * pm * kTile + lane;
  const double cj0 = jok ? a.cen[3 * j] : 0.0, cj1 = jok ? a.cen[3 * j + 1] : 0.0, cj2 = jok ? a.cen[3 * j + 2] : 0.0;
  // The column element's points in pairs, the last one alone when QB is odd;
  // normals negated (so is dj, exactly).  One block of points holds them all: loaded
  // once for the tile's rows.
  constexpr int P = QB / 2;
  F32x2 oq[P][3], nq[P][3];
  float wq[QB], oqs[3] = {0.0f, 0.0f, 0.0f}, nqs[3] = {0.0f, 0.0f, 0.0f};
  auto load = [&](int q0) {
    auto at = [&](int c, int u) { return q0 + u < npj0 ? jbf[(c * pm + q0 + u) * kTile] : 0.0f; };
#pragma unroll
    for (int c = 0; c < 3; ++c) {
#pragma unroll
      for (int u = 0; u < P; ++u) {
        oq[u][c] = f2_pack(at(c, 2 * u), at(c, 2 * u + 1));
        nq[u][c] = f2_pack(-at(3 + c, 2 * u), -at(3 + c, 2 * u + 1));
      }
      if (QB & 1) {
        oqs[c] = at(c, QB - 1);
        nqs[c] = -at(3 + c, QB - 1);
      }
    }
#pragma unroll
    for (int u = 0; u < QB; ++u) wq[u] = at(6, u);
  };
  if (pm <= QB) load(0);
  const F32x2 pi2 = f2_pack(3.14159265f, 3.14159265f);
  // li0 < 8: the warp's rows li0, li0 + 8, ...; li0 >= 8: the single row li0 - 8
  for (int li = li0 < 8 ? li0 : li0 - 8; li < kTile; li += li0 < 8 ? 8 : kTile) {
    const int64_t i = bi * kTile + li;
    if (i >= N) break;  // warp-uniform
    const bool valid = jok && i < j;
    const int64_t oi = a.orig ? (int64_t)a.orig[i] : i;
    const int npi = a.np[i];
    int npj = valid ? npj0 : 0;
    if (valid && a.flat[i] && a.flat[j] && a.nrm[3 * i] == a.nrm[3 * j] && a.nrm[3 * i + 1] == a.nrm[3 * j + 1] &&
        a.nrm[3 * i + 2] == a.nrm[3 * j + 2])
      npj = 0;
    const int qmax = __reduce_max_sync(kFull, npj);
    const float d0 = (float)(cj0 - a.cen[3 * i]), d1 = (float)(cj1 - a.cen[3 * i + 1]),
                d2 = (float)(cj2 - a.cen[3 * i + 2]);
    // the row's points, every value twice: -o0 | -o1 | -o2 | n0 | n1 | n2 | w
    const float* ibf = iblk + li;
    float4* Sf = reinterpret_cast<float4*>(S);
    __syncwarp();
    for (int p = lane; p < npi; p += 32) {
      float v[7];
#pragma unroll
      for (int c = 0; c < 7; ++c) v[c] = ibf[(c * pm + p) * kTile];
      Sf[4 * p] = make_float4(-v[0], -v[0], -v[1], -v[1]);
      Sf[4 * p + 1] = make_float4(-v[2], -v[2], v[3], v[3]);
      Sf[4 * p + 2] = make_float4(v[4], v[4], v[5], v[5]);
      Sf[4 * p + 3] = make_float4(v[6], v[6], 0.0f, 0.0f);
    }
    __syncwarp();
    float acc32 = 0.0f;
    uint32_t cast = 0;
    const F32x2 d02 = f2_pack(d0, d0), d12 = f2_pack(d1, d1), d22 = f2_pack(d2, d2);
    for (int q0 = 0; q0 < qmax; q0 += QB) {
      if (pm > QB) load(q0);
      F32x2 inner2[P];
      float inners = 0.0f;
#pragma unroll
      for (int u = 0; u < P; ++u) inner2[u] = f2_pack(0.0f, 0.0f);
      for (int p = 0; p < npi; ++p) {
        const ulonglong2* sp = reinterpret_cast<const ulonglong2*>(S) + 4 * p;
        const ulonglong2 s0 = sp[0], s1 = sp[1], s2 = sp[2];
        const F32x2 o0 = s0.x, o1 = s0.y, o2 = s1.x, n0 = s1.y, n1 = s2.x, n2 = s2.y, w2 = sp[3].x;
        // straight-line over the block: a point q0 + u >= npj has zero
        // normal, so its dj is 0 and its K zero
#pragma unroll
        for (int u = 0; u < P; ++u) {
          const F32x2 rx = f2_add(d02, f2_add(oq[u][0], o0)), ry = f2_add(d12, f2_add(oq[u][1], o1)),
                      rz = f2_add(d22, f2_add(oq[u][2], o2));
          const F32x2 r2 = f2_fma(rx, rx, f2_fma(ry, ry, f2_mul(rz, rz)));
          const F32x2 di = f2_fma(n0, rx, f2_fma(n1, ry, f2_mul(n2, rz)));
          const F32x2 dj = f2_fma(nq[u][0], rx, f2_fma(nq[u][1], ry, f2_mul(nq[u][2], rz)));
          float b0, b1, k0, k1, i0, i1, j0, j1;
          f2_unpack(f2_mul(pi2, f2_mul(r2, r2)), b0, b1);
          f2_unpack(f2_mul(f2_mul(di, dj), f2_pack(rcp_approx(b0), rcp_approx(b1))), k0, k1);
          f2_unpack(di, i0, i1);
          f2_unpack(dj, j0, j1);
          k0 = i0 > 0.0f && j0 > 0.0f ? k0 : 0.0f;
          k1 = i1 > 0.0f && j1 > 0.0f ? k1 : 0.0f;
          cast += k0 > 0.0f ? 1 : 0;
          cast += k1 > 0.0f ? 1 : 0;
          inner2[u] = f2_fma(w2, f2_pack(k0, k1), inner2[u]);
        }
        if (QB & 1) {
          float op0, op1, op2, np0, np1, np2, wp, skip2;
          f2_unpack(o0, op0, skip2);
          f2_unpack(o1, op1, skip2);
          f2_unpack(o2, op2, skip2);
          f2_unpack(n0, np0, skip2);
          f2_unpack(n1, np1, skip2);
          f2_unpack(n2, np2, skip2);
          f2_unpack(w2, wp, skip2);
          const float rx = d0 + (oqs[0] + op0), ry = d1 + (oqs[1] + op1), rz = d2 + (oqs[2] + op2);
          const float r2 = fmaf(rx, rx, fmaf(ry, ry, rz * rz));
          const float di = fmaf(np0, rx, fmaf(np1, ry, np2 * rz));
          const float dj = fmaf(nqs[0], rx, fmaf(nqs[1], ry, nqs[2] * rz));
          const float K32 = (di > 0.0f && dj > 0.0f) ? (di * dj) * rcp_approx(3.14159265f * (r2 * r2)) : 0.0f;
          cast += K32 > 0.0f ? 1 : 0;
          inners = fmaf(wp, K32, inners);
        }
      }
#pragma unroll
      for (int u = 0; u < QB; ++u) {
        float v = inners, x, y;
        if (u < 2 * P) {
          f2_unpack(inner2[u / 2], x, y);
          v = u & 1 ? y : x;
        }
        if (q0 + u < npj) acc32 = fmaf(wq[u], v, acc32);
      }
    }
    if (OCC) n_rays += npj > 0 ? cast : 0u;
    n_pp += (uint32_t)(npi * npj);
    const double raw = 0.0 + (double)acc32;
    if (valid) {
      a.F[oi + oj * N] = raw / a.area[i];
      a.F[oj + oi * N] = raw / a.area[j];
    } else if (j == i) {
      a.F[oi + oi * N] = 0.0 / a.area[i];
    }
  }
}

// Out of line inside the chunked generation kernels, whose own registers are
// allocated for the ray pipeline.
template <bool DIM3, bool OCC, int QB>
__device__ __noinline__ void gen_fast_fp64(const PairArgs& a, const double* iblk, double* S, int64_t bi, int64_t bj,
                                           int li0, int lane, uint32_t& n_pp, uint32_t& n_rays, uint32_t skip) {
  gen_fast_fp64_body<DIM3, OCC, QB>(a, iblk, S, bi, bj, li0, lane, n_pp, n_rays, skip);
}
template <bool OCC, int QB>
__device__ __noinline__ void gen_fast_mixed(const MixedArgs& a, const float* iblk, int64_t bi, int64_t bj, int li0,
                                            int lane, uint32_t& n_pp, uint32_t& n_rays, uint32_t skip) {
  gen_fast_mixed_body<OCC, QB>(a, iblk, bi, bj, li0, lane, n_pp, n_rays, skip);
}

// The fast loop with the point block for the rule's size (li0 as there).
template <bool DIM3, bool OCC>
__device__ __forceinline__ void fast_fp64(const PairArgs& a, const double* iblk, double* S, int64_t bi, int64_t bj,
                                          int li0, int lane, uint32_t& n_pp, uint32_t& n_rays, uint32_t skip = 0) {
  if (a.pmax <= 3) gen_fast_fp64<DIM3, OCC, 3>(a, iblk, S, bi, bj, li0, lane, n_pp, n_rays, skip);
  else gen_fast_fp64<DIM3, OCC, 4>(a, iblk, S, bi, bj, li0, lane, n_pp, n_rays, skip);
}
template <bool OCC>
__device__ __forceinline__ void fast_mixed(const MixedArgs& a, const float* iblk, int64_t bi, int64_t bj, int li0,
                                           int lane, uint32_t& n_pp, uint32_t& n_rays, uint32_t skip = 0) {
  const int pm = a.pmax;
  if (pm == 7 || pm == 13 || pm == 49) gen_fast_mixed<OCC, 7>(a, iblk, bi, bj, li0, lane, n_pp, n_rays, skip);
  else if (pm == 5 || pm == 25) gen_fast_mixed<OCC, 5>(a, iblk, bi, bj, li0, lane, n_pp, n_rays, skip);
  else if (pm == 3 || pm == 9) gen_fast_mixed<OCC, 3>(a, iblk, bi, bj, li0, lane, n_pp, n_rays, skip);
  else gen_fast_mixed<OCC, 8>(a, iblk, bi, bj, li0, lane, n_pp, n_rays, skip);
}

}  // namespace rvf
