// kernels_mc.cu -- stratified Monte Carlo pair kernel (src/GPUMCKernels.jl:146-281).
//
// Every pair keeps the reference's own random stream: splitmix64 of
// seed + ((i-1) N + j) * golden (1-based caller indices, i < j), then
// xorshift64 draws u = (s >> 11) / (2^53 - 1), four per sample (u1,u2 for
// element i, u3,u4 for element j), s = floor(sqrt(n)) strata per axis with the
// same stratum on both elements, uniform remainder samples.  Geometry, kernel
// and rays use the reference's FP64 arithmetic bit for bit, and K_sum is
// accumulated in sample order, so raw values equal the reference's exactly.
//
// Areas follow a fixed rule where the reference races (src/GPUMCKernels.jl:
// 258-259): A_i is the estimate of pair (i, i+1) in the i-role, A_N that of
// pair (N-1, N) in the j-role.
//
// Curve meshes (the reference GPU path rejects them): element i is sampled at
// xi = 2*((si+u1)/s) - 1, element j at xi = 2*((sj+u3)/s) - 1 (u2, u4 drawn and
// unused), remainder samples at 2*u1-1 and 2*u3-1, reference measure 2,
// kernel cos*cos/(2r), occlusion by the 2-D segment test.
//
// Surfaces run in two kernels: k_mc_rows, a lane per pair, for the pairs whose
// rays the tile classification (kernels_cull.cu) proves visible, and k_mc_queue, a
// lane per sample, for the others.  Curves run in k_mc_curves with per-row segment
// lists.  Element nodes are staged in shared memory; quotients by a common divisor
// take one division and a corrected product each (div_by).
//
// Measured on a B200, 64 samples a pair.  Closed cube of 2,166 Quad4 with a box:
// rows 4.4 ms, blockable pairs (7% of all) 5.0 ms, classification 1.6 ms; one kernel
// with a tree walk in every masked row took 46 ms (2.6 of a row's 32 pairs masked,
// eight warps at a barrier per tile).  Rows are bound by FP64 issue (66% of the
// pipe), blockable pairs by the walks' issue and latency.  Cavity of 4,000 Line3 with
// four circles: 15.5 ms; 33 ms with a tree walk per ray, 24 ms with a lane per
// pair testing its own list (lists differ in length between the lanes).
// Measured and not kept: the blockable pairs a lane each (52 ms: a walk's 32 rays
// share few nodes); per-pair triangle lists in place of the walks (9.4 to 11.0 ms
// for both kernels by the longest list allowed, against 9.8: a whole element's
// capsule reaches as many leaves as a walk visits nodes); two blocks a
// multiprocessor (17.2 ms for the curves).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "device_mixed.cuh"
#include "device_segs.cuh"
#include "kernels.h"

namespace rvf {

namespace {

__device__ __forceinline__ uint64_t init_rng(uint64_t seed, uint64_t tid) {  // src/GPUMCKernels.jl:44-50
  uint64_t z = seed + tid * 0x9E3779B97F4A7C15ULL;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
  return z ^ (z >> 31);
}

__device__ __forceinline__ double xorshift64(uint64_t& s) {  // src/GPUMCKernels.jl:37-42
  s ^= s << 13;
  s ^= s >> 7;
  s ^= s << 17;
  // v / (2^53 - 1) for an integer v < 2^53.  x = v 2^-53 is exact, and the
  // quotient is x + x 2^-53 (1 + 2^-53 + ...): above x by more than half and at
  // most one unit of x's last place, so it rounds to the next number above x.
  // v becomes a double from its halves (exact sums).
  const uint64_t v = s >> 11;
  const double d = (__hiloint2double(0x45300000, (int)(v >> 32)) - (0x1p84 + 0x1p52)) +
                   __hiloint2double(0x43300000, (int)(uint32_t)v);
  const long long b = __double_as_longlong(d) + (1ll - (53ll << 52));
  return __longlong_as_double(v ? b : 0ll);
}

__device__ __forceinline__ double ref_measure(int f) { return is_quad_fam(f) ? 4.0 : (is_line_fam(f) ? 2.0 : 0.5); }

// sample of one element at (u, v) in [0,1]^2 (src/GPUMCKernels.jl:266-281)
// or, for curves, at reference coordinate u (already mapped to [-1,1]).
// A curve mesh holds line elements only, a surface mesh surface elements
// only: each kernel compiles its own families.
// Surfaces: out of line, so that the six families' geometry does not
// hold the pair kernel's registers.
__device__ __noinline__ void mc_surface(const double* coords, const int32_t* en, int f, double u, double v, double* x,
                                        double* n, double* dA) {
  if (is_quad_fam(f)) {
    eval_surface(coords, en, f, 2.0 * u - 1.0, 2.0 * v - 1.0, x, n, dA);
  } else {
    double xi = u, eta = v;
    if (xi + eta > 1.0) {
      xi = 1.0 - xi;
      eta = 1.0 - eta;
    }
    eval_surface(coords, en, f, xi, eta, x, n, dA);
  }
}

template <bool DIM3>
__device__ __forceinline__ void mc_point(const McArgs& a, const int32_t* en, int f, double u, double v, double* x,
                                         double* n, double* dA) {
  if (!DIM3) {
    eval_line(a.coords, en, f, u, x, n, dA);
  } else {
    mc_surface(a.coords, en, f, u, v, x, n, dA);
  }
}

// A pair's stream: its samples in order.
struct McStream {
  uint64_t st;
  double s, inv_s, si, sj;  // strata per axis, the next sample's stratum
  int left;                 // stratified samples left
  bool pow2;                // s a power of two: the strata's quotients are products
  __device__ __forceinline__ McStream(uint64_t state, int strata)
      : st(state), s(strata), inv_s(1.0 / strata), si(0.0), sj(0.0), left(strata * strata),
        pow2((strata & (strata - 1)) == 0) {}
  __device__ __forceinline__ double in_stratum(double a) const {  // a / s: a is 0 or at least 2^-53
    return pow2 ? a * inv_s : div_by(a, s, inv_s);
  }
  // to sample k, the state being that before it
  __device__ __forceinline__ void skip(int k) {
    if (k >= left) {
      left = 0;
    } else {
      left -= k;
      const int n = (int)s;
      si = (double)(k / n);
      sj = (double)(k % n);
    }
  }
  // the two elements' reference coordinates of the next sample
  template <bool DIM3>
  __device__ __forceinline__ void next(double* ci, double* cj) {
    double u1 = xorshift64(st), u2 = xorshift64(st), u3 = xorshift64(st), u4 = xorshift64(st);
    if (left > 0) {
      --left;
      u1 = in_stratum(si + u1);
      u3 = in_stratum((DIM3 ? si : sj) + u3);
      if (DIM3) {
        u2 = in_stratum(sj + u2);
        u4 = in_stratum(sj + u4);
      }
      sj += 1.0;
      if (sj == s) {
        sj = 0.0;
        si += 1.0;
      }
    }
    if (DIM3) {
      ci[0] = u1; ci[1] = u2; cj[0] = u3; cj[1] = u4;
    } else {
      ci[0] = 2.0 * u1 - 1.0; ci[1] = 0.0; cj[0] = 2.0 * u3 - 1.0; cj[1] = 0.0;
    }
  }
};

// ---------------------------------------------------------------------------
// Curves with occlusion: per-pair candidate segments.
//
// The reference walks the whole segment tree for every sample ray, testing a
// node when the ray's bounding box overlaps it (src/BVH.jl:285-322).  A
// segment blocks a ray only if the computed test puts their intersection
// inside both, which (rounding included) needs the segment within
// cand_margin of the ray; and every ray of pair (i, j) lies within
// R = max(r_i, r_j) of the segment between the elements' centres (each
// element's points lie within r of its centre).  So a block lists the segments
// within reach of its tile, a lane per pair those within reach of its capsule
// (device_segs.cuh), and each sample tests only these with the reference's own
// segment test, a hit counting when the overlap test of its leaf passes too (the
// leaf box lies inside every ancestor's, so the test passing there means the
// reference's walk reaches it).  Decisions are identical to the full walk's.  Rows
// with more than kRowItems tests, and tiles whose list overflows, walk the tree for
// every sample.
// ---------------------------------------------------------------------------

// Centre and radius of a Line3 / Line2 element: the quadratic curve lies in
// the triangle of its end nodes and its Bezier middle control point
// 2 x_mid - (x_a + x_b) / 2; a Line2 between its ends.
__device__ __forceinline__ void line_bounds(const double* coords, const int32_t* en, int f, double* c, double& r) {
  const double* a = coords + 3 * (int64_t)en[0];
  const double* b = coords + 3 * (int64_t)en[1];
  double p[3][2];
  int n = 2;
  p[0][0] = a[0]; p[0][1] = a[1];
  p[1][0] = b[0]; p[1][1] = b[1];
  if (f == 4) {
    const double* m = coords + 3 * (int64_t)en[2];
    p[2][0] = 2.0 * m[0] - 0.5 * (a[0] + b[0]);
    p[2][1] = 2.0 * m[1] - 0.5 * (a[1] + b[1]);
    n = 3;
  }
  c[0] = c[1] = 0.0;
  for (int k = 0; k < n; ++k) {
    c[0] += p[k][0] / n;
    c[1] += p[k][1] / n;
  }
  r = 0.0;
  for (int k = 0; k < n; ++k) r = fmax(r, hypot(p[k][0] - c[0], p[k][1] - c[1]));
  r *= 1.0 + 1e-12;
}

}  // namespace

// Area rule: one thread per caller-order element.
// A point of a surface element: with each mid-side node written as its
// edge's midpoint plus a deviation, x_m = (x_a + x_b) / 2 + delta_m, the
// quadratic families reproduce their linear / bilinear interpolant, so
//   x(xi) = sum_c L_c(xi) x_c + sum_m N_m(xi) delta_m
// with L_c >= 0 summing to 1 (the corners' linear or bilinear functions) and
// N_m >= 0 the mid-side functions, whose sum peaks at 2 (Quad8, at the
// centre) and 4/3 (Tri6, at the centroid).  Hence |x - c| <= max_c |x_c - c|
// + (2 or 4/3) max_m |delta_m| for the corners' centroid c.  Node order as
// shape_surface: Quad8 mid-sides 4..7 on edges 0-1, 1-2, 2-3, 3-0; Tri6 3..5
// on edges 0-1, 1-2, 0-2.  The radius is rounded up by a relative 1e-9: a
// Monte Carlo sample point, evaluated in FP64 from the same nodes, lies
// inside it.
__global__ void k_mc_bounds(McBoundsArgs a) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= a.N) return;
  const int f = a.fam[e];
  const int nc = (f == 0 || f == 2) ? 4 : 3;
  const int32_t* en = a.enodes + 8 * e;
  auto X = [&](int k) { return a.coords + 3 * (int64_t)en[k]; };
  double c[3] = {0.0, 0.0, 0.0};
  for (int k = 0; k < nc; ++k)
    for (int d = 0; d < 3; ++d) c[d] += X(k)[d];
  for (int d = 0; d < 3; ++d) c[d] /= nc;
  double r2 = 0.0;
  for (int k = 0; k < nc; ++k) {
    const double* x = X(k);
    const double dx = x[0] - c[0], dy = x[1] - c[1], dz = x[2] - c[2];
    r2 = fmax(r2, dx * dx + dy * dy + dz * dz);
  }
  double dev2 = 0.0, lam = 0.0;
  if (f == 0 || f == 1) {
    static constexpr int q8[4][3] = {{4, 0, 1}, {5, 1, 2}, {6, 2, 3}, {7, 3, 0}};
    static constexpr int t6[3][3] = {{3, 0, 1}, {4, 1, 2}, {5, 0, 2}};
    const int nm = f == 0 ? 4 : 3;
    lam = f == 0 ? 2.0 : 4.0 / 3.0;
    for (int m = 0; m < nm; ++m) {
      const int* mb = f == 0 ? q8[m] : t6[m];
      const double *xm = X(mb[0]), *xa = X(mb[1]), *xb = X(mb[2]);
      double q = 0.0;
      for (int d = 0; d < 3; ++d) {
        const double dd = xm[d] - 0.5 * (xa[d] + xb[d]);
        q += dd * dd;
      }
      dev2 = fmax(dev2, q);
    }
  }
  for (int d = 0; d < 3; ++d) a.cen[3 * e + d] = c[d];
  a.rad[e] = (sqrt(r2) + lam * sqrt(dev2)) * (1.0 + 1e-9);
}

__global__ void k_mc_area(McArgs a) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t N = a.N;
  if (e >= N) return;
  if (N < 2) {
    a.area_orig[e] = 0.0;
    return;
  }
  const bool first = e + 1 < N;
  const int64_t lo = first ? e : e - 1, hi = first ? e + 1 : e;
  McStream q(init_rng(a.seed, (uint64_t)(lo * N + hi + 1)), (int)floor(sqrt((double)a.n_samples)));
  const int64_t ie = a.inv[e];
  const int f = a.fam[ie];
  const int32_t* en = a.enodes + 8 * ie;
  double A = 0.0;
  for (int k = 0; k < a.n_samples; ++k) {
    double ci[2], cj[2];
    if (a.dim3) q.next<true>(ci, cj);
    else q.next<false>(ci, cj);
    const double* c = first ? ci : cj;
    double x[3], n[3], dA;
    if (a.dim3) mc_point<true>(a, en, f, c[0], c[1], x, n, &dA);
    else mc_point<false>(a, en, f, c[0], c[1], x, n, &dA);
    A += dA;
  }
  a.area_orig[e] = (A * ref_measure(f)) / (double)a.n_samples;
}

// Element evaluation from node coordinates staged in shared memory (value 3 k + c
// at X[(3 k + c) stride]), eval_surface's arithmetic operation for operation.
struct McPoint {
  double x[3], n[3], dA;
};
template <int F>
__device__ __forceinline__ void mc_eval_family(const double* X, int stride, double xi, double eta, McPoint& r) {
  constexpr int nn = F == 0 ? 8 : F == 1 ? 6 : F == 2 ? 4 : 3;
  double N[8], dX[8], dE[8];
  shape_surface(F, xi, eta, N, dX, dE);
  double p[3] = {0.0, 0.0, 0.0}, a[3] = {0.0, 0.0, 0.0}, b[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int k = 0; k < nn; ++k)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double v = X[(3 * k + c) * stride];
      p[c] = p[c] + N[k] * v;
      a[c] = a[c] + dX[k] * v;
      b[c] = b[c] + dE[k] * v;
    }
  const double c[3] = {a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]};
  r.dA = sqrt((c[0] * c[0] + c[1] * c[1]) + c[2] * c[2]);
  div_all(c, r.dA, r.n);
#pragma unroll
  for (int k = 0; k < 3; ++k) r.x[k] = p[k];
}
// The normal and dA of a Tri3 or Line2 are the same at every point (their
// derivatives are constants): computed once per pair, the samples then need the
// point alone.
__device__ __forceinline__ void mc_const_normal(int f, const double* X, int stride, McPoint& r) {
  if (f == 3) mc_eval_family<3>(X, stride, 0.0, 0.0, r);
}
__device__ __forceinline__ void mc_eval(int f, const double* X, int stride, double u, double v, McPoint& r) {
  if (is_quad_fam(f)) {
    u = 2.0 * u - 1.0;
    v = 2.0 * v - 1.0;
    if (f == 0) mc_eval_family<0>(X, stride, u, v, r);
    else mc_eval_family<2>(X, stride, u, v, r);
    return;
  }
  if (u + v > 1.0) {
    u = 1.0 - u;
    v = 1.0 - v;
  }
  if (f == 1) {
    mc_eval_family<1>(X, stride, u, v, r);
    return;
  }
  const double N[3] = {(1.0 - u) - v, u, v};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    double p = 0.0;
#pragma unroll
    for (int k = 0; k < 3; ++k) p = p + N[k] * X[(3 * k + c) * stride];
    r.x[c] = p;
  }
}
// Line3 / Line2 (eval_line).  FLAT: every node's z is zero, and so are the
// point's z and the tangent's (sums of products with zeros).
template <bool FLAT>
__device__ __forceinline__ void mc_tangent(const double* t, McPoint& r) {
  r.dA = FLAT ? sqrt(t[0] * t[0] + t[1] * t[1]) : sqrt((t[0] * t[0] + t[1] * t[1]) + t[2] * t[2]);
  const double tt[2] = {t[0], t[1]};
  double q[2];
  div_all(tt, r.dA, q);
  r.n[0] = -q[1];
  r.n[1] = q[0];
  r.n[2] = 0.0;
}
template <bool FLAT>
__device__ __forceinline__ void mc_eval_line(int f, const double* X, int stride, double xi, McPoint& r) {
  constexpr int C = FLAT ? 2 : 3;
  r.x[2] = 0.0;
  if (f == 4) {
    const double N[3] = {((-0.5) * xi) * (1.0 - xi), (0.5 * xi) * (1.0 + xi), 1.0 - xi * xi};
    const double dN[3] = {-0.5 + xi, 0.5 + xi, -2.0 * xi};
    double t[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int c = 0; c < C; ++c) {
      double p = 0.0;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        p = p + N[k] * X[(3 * k + c) * stride];
        t[c] = t[c] + dN[k] * X[(3 * k + c) * stride];
      }
      r.x[c] = p;
    }
    mc_tangent<FLAT>(t, r);
  } else {
    const double N[2] = {0.5 * (1.0 - xi), 0.5 * (1.0 + xi)};
#pragma unroll
    for (int c = 0; c < C; ++c) {
      double p = 0.0;
#pragma unroll
      for (int k = 0; k < 2; ++k) p = p + N[k] * X[(3 * k + c) * stride];
      r.x[c] = p;
    }
  }
}
__device__ __forceinline__ void mc_const_tangent(int f, const double* X, int stride, McPoint& r) {
  if (f != 5) return;
  double t[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) t[c] = (0.0 + (-0.5) * X[c * stride]) + 0.5 * X[(3 + c) * stride];
  mc_tangent<false>(t, r);
}
// cos cos / (2 r) of a curve pair (k_reference_inl): one reciprocal of r serves
// the direction and, halved (exact), the last quotient.  Symmetric in the two
// points bit for bit, as is k_reference_inl.
template <bool FLAT>
__device__ __forceinline__ double mc_kernel_2d(double rx, double ry, double rz, double r2, const double* ni,
                                               const double* nj) {
  const double r = sqrt(r2);
  const double rv[3] = {rx, ry, rz};
  const bool ok = div_by_ok(r) && div_by_ok(rx) && div_by_ok(ry) && (FLAT || div_by_ok(rz));
  const double y = 1.0 / r;
  double h[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int c = 0; c < (FLAT ? 2 : 3); ++c) h[c] = div_by(rv[c], r, y);
  if (!ok)
    for (int c = 0; c < 3; ++c) h[c] = rv[c] / r;
  double ci = ni[0] * h[0] + ni[1] * h[1], cj = nj[0] * (-h[0]) + nj[1] * (-h[1]);
  if constexpr (!FLAT) {
    ci = ci + ni[2] * h[2];
    cj = cj + nj[2] * (-h[2]);
  }
  if (ci <= 0.0 || cj <= 0.0) return 0.0;
  const double c = ci * cj, b = 2.0 * r;
  return ok && div_by_ok(c) ? div_by(c, b, 0.5 * y) : c / b;
}

// One pair a lane: identity, stream and what its result needs.
struct McPair {
  int64_t oi, oj;  // caller indices of the row's and the lane's element
  bool sw;         // the reference's pair is (lane's, row's)
  uint8_t* log;
  __device__ __forceinline__ McPair(const McArgs& a, int64_t i, int64_t j, bool valid)
      : oi(a.orig[i]), oj(valid ? (int64_t)a.orig[j] : 0), sw(valid && oi > oj), log(nullptr) {
    if (a.ray_log && valid) log = a.ray_log + ((uint64_t)lo() * a.N + hi()) * a.n_samples;
  }
  // the reference's pair (lo, hi): lo samples with u1,u2 and casts the ray
  __device__ __forceinline__ int64_t lo() const { return sw ? oj : oi; }
  __device__ __forceinline__ int64_t hi() const { return sw ? oi : oj; }
  __device__ __forceinline__ uint64_t seed(const McArgs& a) const {
    return init_rng(a.seed, (uint64_t)(lo() * a.N + hi() + 1));
  }
  __device__ __forceinline__ void finish(const McArgs& a, double Ks, int f_i, int f_j) const {
    const int f_lo = sw ? f_j : f_i, f_hi = sw ? f_i : f_j;
    const double raw = ((Ks * ref_measure(f_lo)) * ref_measure(f_hi)) / (double)a.n_samples;
    a.F[oi + oj * a.N] = raw / a.area_orig[oi];
    a.F[oj + oi * a.N] = raw / a.area_orig[oj];
  }
};

// The pairs of row li of tile t whose sample rays may be blocked.
__device__ __forceinline__ uint32_t mc_row_mask(const McArgs& a, int64_t t, int li) {
  if (!a.tcls) return kFull;
  return (a.tcls[t] & kClsSlow) ? a.tmask[t * kTile + li] : 0u;
}
// node coordinates of element e (or zeros) at X[(3 k + c) stride]
__device__ __forceinline__ void mc_stage(const McArgs& a, int64_t e, bool ok, double* X, int stride) {
  const int nn = ok ? fam_nodes(a.fam[e]) : 0;
#pragma unroll
  for (int k = 0; k < 8; ++k)
    if (k < nn) {
      const double* p = a.coords + 3 * (int64_t)a.enodes[8 * e + k];
#pragma unroll
      for (int c = 0; c < 3; ++c) X[(3 * k + c) * stride] = p[c];
    } else {
#pragma unroll
      for (int c = 0; c < 3; ++c) X[(3 * k + c) * stride] = 0.0;
    }
}

// A sample of a surface pair: the points and K.  The kernel is symmetric in the
// two elements bit for bit (the cosines swap and every difference changes sign
// exactly), so the row's element stays the source whatever the reference's order
// of the pair; only the draws, the product's order and the ray's direction follow it.
__device__ __forceinline__ double mc_sample_3d(McStream& q, bool sw, bool mine, int f_i, const double* Xi, int f_j,
                                               const double* Xj, int stride_i, int stride_j, McPoint& pi, McPoint& pj,
                                               double* r, double& r2) {
  double ulo[2], uhi[2];
  q.next<true>(ulo, uhi);
  mc_eval(f_i, Xi, stride_i, sw ? uhi[0] : ulo[0], sw ? uhi[1] : ulo[1], pi);
  mc_eval(f_j, Xj, stride_j, sw ? ulo[0] : uhi[0], sw ? ulo[1] : uhi[1], pj);
#pragma unroll
  for (int c = 0; c < 3; ++c) r[c] = pj.x[c] - pi.x[c];
  r2 = (r[0] * r[0] + r[1] * r[1]) + r[2] * r[2];
  return mine && !(r2 < 1e-30) ? k_reference_inl<true>(r[0], r[1], r[2], r2, pi.n, pj.n) : 0.0;
}
// make_ray's cast rule
__device__ __forceinline__ bool mc_cast(double K, double r2) { return K > 0.0 && (r2 > 2e-30 || sqrt(r2) > 1e-15); }

__device__ __forceinline__ void mc_count(const McArgs& a, uint64_t n_pp, uint64_t n_rays, const TravCount& tc) {
  const uint64_t v[4] = {n_pp, n_rays, tc.nodes, tc.prims};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const uint64_t s = warp_sum_u64(v[k]);
    if ((threadIdx.x & 31) == 0 && a.counters && s) atomicAdd(a.counters + k, (unsigned long long)s);
  }
}

// Surfaces, pairs without a blockable ray: a warp per claimed rows of a tile, a
// lane a pair; the elements' nodes staged in the warp's shared memory.
struct McRow {
  double xj[24 * 32];  // column elements', value v of lane l at 32 v + l
  double xi[24];
};
template <bool OCC>
__global__ void __launch_bounds__(256, 3) k_mc_rows(McArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  McRow& W = reinterpret_cast<McRow*>(smem)[warp];
  const int64_t N = a.N;
  const int s = (int)floor(sqrt((double)a.n_samples));
  const int per_tile = kTile / a.rows;
  uint64_t n_rays = 0, n_pp = 0;
  for (;;) {
    unsigned long long k = 0;
    if (lane == 0) k = atomicAdd(a.tile_counter, 1ull);
    k = __shfl_sync(kFull, k, 0);
    const int64_t tl = (int64_t)(k / (unsigned)per_tile);
    if (tl >= a.tile_count) break;
    const int64_t t = a.tile0 + tl;
    int64_t bi, bj;
    tile_coords(t, a.nT, bi, bj);
    const int row0 = (int)(k - (unsigned long long)tl * (unsigned)per_tile) * a.rows;
    const int64_t j = bj * kTile + lane;
    const bool okj = j < N;
    const int f_j = a.fam[okj ? j : bj * kTile];
    __syncwarp();
    mc_stage(a, j, okj, W.xj + lane, 32);
    for (int li = row0; li < row0 + a.rows; ++li) {
      const int64_t i = bi * kTile + li;
      if (i >= N) break;
      const bool mine = okj && i < j && !(OCC && ((mc_row_mask(a, t, li) >> lane) & 1u));
      const int f_i = a.fam[i];
      const McPair P(a, i, j, mine);
      if (j == i) a.F[P.oi + P.oi * N] = 0.0 / a.area_orig[P.oi];
      if (!__any_sync(kFull, mine)) continue;
      __syncwarp();
      if (lane < 8) {
        const bool in = lane < fam_nodes(f_i);
        const double* p = a.coords + 3 * (int64_t)(in ? a.enodes[8 * i + lane] : 0);
#pragma unroll
        for (int c = 0; c < 3; ++c) W.xi[3 * lane + c] = in ? p[c] : 0.0;
      }
      __syncwarp();
      McStream q(P.seed(a), s);
      McPoint pi, pj;
      mc_const_normal(f_i, W.xi, 1, pi);
      mc_const_normal(f_j, W.xj + lane, 32, pj);
      double Ks = 0.0;
      for (int smp = 0; smp < a.n_samples; ++smp) {
        double r[3], r2;
        const double K = mc_sample_3d(q, P.sw, mine, f_i, W.xi, f_j, W.xj + lane, 1, 32, pi, pj, r, r2);
        if (OCC) {
          const bool cast = mc_cast(K, r2);
          n_rays += cast ? 1 : 0;
          if (P.log) P.log[smp] = cast ? 1 : 0;
        }
        Ks += (K * (P.sw ? pj.dA : pi.dA)) * (P.sw ? pi.dA : pj.dA);
      }
      if (mine) {
        n_pp += (uint64_t)a.n_samples;
        P.finish(a, Ks, f_i, f_j);
      }
    }
  }
  mc_count(a, n_pp, n_rays, TravCount{});
}

// Surfaces, pairs whose rays may be blocked: a warp takes 8 of them from the masks
// of kMcBundle consecutive tiles.  A lane per pair runs the pair's stream ahead
// and leaves the state before each sample; a lane per sample then draws it,
// evaluates the pair there and walks the tree, so that a walk's 32 rays are one
// pair's: in FP32 with certified decisions (device_mixed.cuh), the uncertain rays
// again in FP64 with the reference's arithmetic.  The lane of the pair adds its
// terms in sample order.
constexpr int kMcBundle = 4;   // tiles whose pairs are put together
constexpr int kMcShare = 32;   // warps that share a bundle's groups of pairs
constexpr int kMcPairs = 8;    // pairs of a group
constexpr int kMcChunk = 32;   // samples of each between two sums
struct McQueue {
  double xi[24 * kMcPairs], xj[24 * kMcPairs];  // value v of pair p at 8 v + p
  union {
    uint64_t state;
    double term;
  } smp[kMcPairs * (kMcChunk + 1)];  // sample k of pair p at 33 p + k
  int64_t i[kMcPairs], j[kMcPairs];
  int first[kMcBundle * kTile];      // pairs before each row's
};
__global__ void __launch_bounds__(128, 4) k_mc_queue(const __grid_constant__ McArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  McQueue& W = reinterpret_cast<McQueue*>(smem)[warp];
  const int64_t N = a.N;
  const int s = (int)floor(sqrt((double)a.n_samples));
  uint64_t n_rays = 0, n_pp = 0;
  TravCount tc;
  for (;;) {
    unsigned long long k = 0;
    if (lane == 0) k = atomicAdd(a.tile_counter + 1, 1ull);
    k = __shfl_sync(kFull, k, 0);
    const int64_t b0 = (int64_t)(k / kMcShare) * kMcBundle;
    if (b0 >= a.tile_count) break;
    __syncwarp();
    int total = 0;
    uint32_t rows[kMcBundle];  // of tile u: row `lane`'s pairs
#pragma unroll
    for (int u = 0; u < kMcBundle; ++u) {
      rows[u] = 0;
      if (b0 + u < a.tile_count) {
        int64_t bi, bj;
        tile_coords(a.tile0 + b0 + u, a.nT, bi, bj);
        const int64_t i = bi * kTile + lane, j0 = bj * kTile;
        const uint32_t in = N - j0 >= 32 ? kFull : (1u << (int)(N - j0)) - 1u;  // j < N
        const uint32_t up = bi < bj ? kFull : (kFull << lane) & ~(1u << lane);  // i < j
        if (i < N) rows[u] = mc_row_mask(a, a.tile0 + b0 + u, lane) & in & up;
      }
      const int n = __popc(rows[u]);
      int incl = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += v;
      }
      W.first[u * kTile + lane] = total + incl - n;
      total += __shfl_sync(kFull, incl, 31);
    }
    __syncwarp();
    for (int g = (int)(k % kMcShare) * kMcPairs; g < total; g += kMcPairs * kMcShare) {
      const int cnt = min(kMcPairs, total - g);
      // lane l < cnt: pair g + l, in the last row that begins at or before it
      const int at = g + min(lane, cnt - 1);
      int row = 0;
#pragma unroll
      for (int o = kMcBundle * kTile / 2; o > 0; o >>= 1)
        if (W.first[row + o] <= at) row += o;
      const int u = row / kTile, li = row % kTile;
      uint32_t m = 0;
#pragma unroll
      for (int v = 0; v < kMcBundle; ++v) {
        const uint32_t x = __shfl_sync(kFull, rows[v], li);
        if (u == v) m = x;
      }
      int64_t bi, bj;
      tile_coords(a.tile0 + b0 + u, a.nT, bi, bj);
      const int64_t i = bi * kTile + li, j = bj * kTile + nth_set_bit(m, at - W.first[row]);
      const McPair P(a, i, j, true);
      if (lane < kMcPairs) {
        W.i[lane] = i;
        W.j[lane] = j;
        mc_stage(a, i, true, W.xi + lane, kMcPairs);
        mc_stage(a, j, true, W.xj + lane, kMcPairs);
      }
      uint64_t st = P.seed(a);
      double Ks = 0.0;
      for (int k0 = 0; k0 < a.n_samples; k0 += kMcChunk) {
        const int S = min(kMcChunk, a.n_samples - k0);
        if (lane < cnt)
          for (int e = 0; e < S; ++e) {
            W.smp[lane * (kMcChunk + 1) + e].state = st;
#pragma unroll
            for (int d = 0; d < 4; ++d) xorshift64(st);
          }
        __syncwarp();
        for (int e0 = 0; e0 < cnt * S; e0 += 32) {
          const bool in = e0 + lane < cnt * S;
          const int p = in ? (e0 + lane) / S : 0, e = in ? e0 + lane - p * S : 0;
          auto& slot = W.smp[p * (kMcChunk + 1) + e];
          const int64_t ip = W.i[p], jp = W.j[p];
          const McPair Q(a, ip, jp, true);
          const int f_i = a.fam[ip], f_j = a.fam[jp];
          const int32_t gx = a.exclude ? a.group[ip] : 0, gy = a.exclude ? a.group[jp] : 0;
          McStream q(slot.state, s);
          q.skip(k0 + e);
          McPoint pi, pj;
          mc_const_normal(f_i, W.xi + p, kMcPairs, pi);
          mc_const_normal(f_j, W.xj + p, kMcPairs, pj);
          double r[3], r2;
          double K = mc_sample_3d(q, Q.sw, in, f_i, W.xi + p, f_j, W.xj + p, kMcPairs, kMcPairs, pi, pj, r, r2);
          const bool cast = mc_cast(K, r2);
          n_rays += cast ? 1 : 0;
          if (__any_sync(kFull, cast)) {
            bool blocked = false, again = cast;
            if (a.trisf) {
              const double* o = Q.sw ? pj.x : pi.x;
              const float of[3] = {(float)o[0], (float)o[1], (float)o[2]};
              const float sg = Q.sw ? -1.0f : 1.0f;
              const float rx = sg * (float)r[0], ry = sg * (float)r[1], rz = sg * (float)r[2];
              const float r2f = fmaf(rx, rx, fmaf(ry, ry, rz * rz));
              RayF R;
              const bool usable = cast && r2f > 1e-18f && make_ray_f(of, rx, ry, rz, r2f, a.delta, R);
              bool unsure = false;
              blocked = packet_any_hit_f(
                  usable, a.nodesf, a.n_nodes, R,
                  [&](int kk, bool test) -> int {
                    const TriF tr = a.trisf[kk];
                    if (!test || tr.group == gx || tr.group == gy) return kMiss;
                    ++tc.prims;
                    return mt_f(tr, R, kMtTight);
                  },
                  unsure, tc);
              again = cast && (unsure || !usable);
            }
            if (__any_sync(kFull, again)) {
              RayD R;
              if (again) {
                if (Q.sw) make_ray(pj.x, -r[0], -r[1], -r[2], r2, R);
                else make_ray(pi.x, r[0], r[1], r[2], r2, R);
              }
              const bool b64 = packet_any_hit(
                  again, a.nodes, a.n_nodes, [&](const NodeD& nd) { return slab_d(nd, R); },
                  [&](int kk, bool test) {
                    const TriD tr = a.tris[kk];
                    if (!test || tr.group == gx || tr.group == gy) return false;
                    ++tc.prims;
                    return mt_d(tr, R);
                  },
                  tc);
              if (again) blocked = b64;
            }
            if (blocked) K = 0.0;
            if (Q.log && cast) Q.log[k0 + e] = blocked ? 2 : 1;
          }
          if (in) slot.term = (K * (Q.sw ? pj.dA : pi.dA)) * (Q.sw ? pi.dA : pj.dA);
        }
        __syncwarp();
        if (lane < cnt)
          for (int e = 0; e < S; ++e) Ks += W.smp[lane * (kMcChunk + 1) + e].term;
      }
      if (lane < cnt) {
        n_pp += (uint64_t)a.n_samples;
        P.finish(a, Ks, a.fam[i], a.fam[j]);
      }
      __syncwarp();
    }
  }
  mc_count(a, n_pp, n_rays, tc);
}

// Curves: a block claims a tile or a part of its rows, a warp takes rows, a lane a
// pair; the elements' nodes in shared memory.
template <bool OCC, bool FLAT>
__device__ __forceinline__ void mc_curve_row(const McArgs& a, const SegScene& sc, SegTile& T, int warp, int ncand,
                                             const McPair& P, bool valid, int f_i, int f_j, int32_t gi, int32_t gj,
                                             int s, const double* Xi, const double* Xj, uint64_t& n_rays,
                                             TravCount& tc) {
  const int lane = threadIdx.x & 31;
  McStream q(P.seed(a), s);
  McPoint pi, pj;
  mc_const_tangent(f_i, Xi, 1, pi);
  mc_const_tangent(f_j, Xj, 32, pj);
  double Ks = 0.0;
  for (int k = 0; k < a.n_samples; ++k) {
    double ulo[2], uhi[2];
    q.next<false>(ulo, uhi);
    mc_eval_line<FLAT>(f_i, Xi, 1, P.sw ? uhi[0] : ulo[0], pi);
    mc_eval_line<FLAT>(f_j, Xj, 32, P.sw ? ulo[0] : uhi[0], pj);
    const double rx = pj.x[0] - pi.x[0], ry = pj.x[1] - pi.x[1], rz = FLAT ? 0.0 : pj.x[2] - pi.x[2];
    const double r2 = FLAT ? rx * rx + ry * ry : (rx * rx + ry * ry) + rz * rz;
    double K = 0.0;
    if (valid && !(r2 < 1e-30)) K = mc_kernel_2d<FLAT>(rx, ry, rz, r2, pi.n, pj.n);
    if (OCC) {
      const bool cast = K > 0.0;
      n_rays += cast ? 1 : 0;
      bool blocked = false;
      const uint32_t casts = ncand != 0 ? __ballot_sync(kFull, cast) : 0u;
      if (casts) {
        const double from[2] = {P.sw ? pj.x[0] : pi.x[0], P.sw ? pj.x[1] : pi.x[1]};
        const double to[2] = {P.sw ? pi.x[0] : pj.x[0], P.sw ? pi.x[1] : pj.x[1]};
        if (ncand > 0) {
          blocked = (items_block(sc, T, warp, ncand, casts, from, to, tc.nodes, tc.prims) >> lane) & 1u;
        } else {
          const double lx = fmin(from[0], to[0]), hx = fmax(from[0], to[0]);
          const double ly = fmin(from[1], to[1]), hy = fmax(from[1], to[1]);
          blocked = packet_any_hit(
              cast, a.nodes, a.n_nodes,
              [&](const NodeD& nd) { return !(nd.lo[0] > hx || nd.hi[0] < lx || nd.lo[1] > hy || nd.hi[1] < ly); },
              [&](int kk, bool test) {
                const SegD sg = a.segs[kk];
                if (!test || sg.group == gi || sg.group == gj) return false;
                ++tc.prims;
                return seg_blocks(sg, from, to);
              },
              tc);
        }
      }
      if (P.log) P.log[k] = cast ? (blocked ? 2 : 1) : 0;
      if (blocked) K = 0.0;
    }
    Ks += (K * (P.sw ? pj.dA : pi.dA)) * (P.sw ? pi.dA : pj.dA);
  }
  if (valid) P.finish(a, Ks, f_i, f_j);
}
template <bool OCC>
__global__ void __launch_bounds__(256, 3) k_mc_curves(McArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  SegTile& T = *reinterpret_cast<SegTile*>(smem);  // with occlusion
  __shared__ int64_t s_tile;
  __shared__ int s_row, s_end, s_segs;
  __shared__ double s_xj[9 * 32], s_xi[8][9];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t N = a.N;
  const int s = (int)floor(sqrt((double)a.n_samples));
  const int per_tile = kTile / a.rows;
  uint64_t n_rays = 0, n_pp = 0;
  TravCount tc;
  for (;;) {
    if (threadIdx.x == 0) {
      const unsigned long long k = atomicAdd(a.tile_counter, 1ull);
      const int64_t tl = (int64_t)(k / (unsigned)per_tile);
      const int part = (int)(k - (unsigned long long)tl * (unsigned)per_tile);
      s_tile = tl < a.tile_count ? a.tile0 + tl : -1;
      s_row = part * a.rows;
      s_end = s_row + a.rows;
    }
    __syncthreads();
    const int64_t t = s_tile;
    if (t < 0) break;
    int64_t bi, bj;
    tile_coords(t, a.nT, bi, bj);
    const int64_t j = bj * kTile + lane;
    const bool okj = j < N;
    const int64_t ej = okj ? j : bj * kTile;
    const int f_j = a.fam[ej];
    const int32_t gj = a.group[ej];
    if (warp < 3) {  // node `warp` of the tile's column elements
      const bool in = warp < fam_nodes(f_j);
      const double* p = a.coords + 3 * (int64_t)a.enodes[8 * ej + (in ? warp : 0)];
#pragma unroll
      for (int c = 0; c < 3; ++c) s_xj[(3 * warp + c) * 32 + lane] = in ? p[c] : 0.0;
    }
    __syncthreads();
    const double* Xj = s_xj + lane;
    HullF H;
    double cj[3] = {0.0, 0.0, 0.0}, rj = 0.0, rj_max = 0.0;
    int nseg = 0;
    SegScene sc{};
    if constexpr (OCC) {
      sc = SegScene{a.nodes, a.nodesf, a.n_nodes, a.segs, a.frontier, a.n_frontier, a.cand_margin, a.seg_slack};
      const int64_t ei = bi * kTile + lane;
      const bool oki = ei < N;
      double cc[3] = {0.0, 0.0, 0.0}, ri = 0.0, rmax;
      if (oki) line_bounds(a.coords, a.enodes + 8 * ei, a.fam[ei], cc, ri);
      if (okj) line_bounds(a.coords, a.enodes + 8 * j, f_j, cj, rj);
      tile_hull(oki, okj, cc, cj, ri, rj, H, rmax, rj_max);
      const int32_t g_i = oki ? a.group[ei] : 0, gi0 = __shfl_sync(kFull, g_i, 0), gj0 = __shfl_sync(kFull, gj, 0);
      const bool g_same = __all_sync(kFull, (!oki || g_i == gi0) && (!okj || gj == gj0));
      if (warp == 0) {
        const int n = tile_segments(sc, H, rmax, g_same, gi0, gj0, T);
        if (lane == 0) s_segs = n;
      }
      __syncthreads();
      nseg = s_segs;
    }
    for (;;) {  // rows, as the warps get to them
      int li = 0;
      if (lane == 0) li = atomicAdd(&s_row, 1);
      li = __shfl_sync(kFull, li, 0);
      if (li >= s_end) break;
      const int64_t i = bi * kTile + li;
      if (i >= N) break;
      const bool valid = okj && i < j;
      const McPair P(a, i, j, valid);
      if (j == i) a.F[P.oi + P.oi * N] = 0.0 / a.area_orig[P.oi];
      if (!__any_sync(kFull, valid)) continue;
      const int f_i = a.fam[i];
      const int32_t gi = a.group[i];
      double* Xi = s_xi[warp];
      if (lane < 3) {
        const bool in = lane < fam_nodes(f_i);
        const double* p = a.coords + 3 * (int64_t)a.enodes[8 * i + (in ? lane : 0)];
#pragma unroll
        for (int c = 0; c < 3; ++c) Xi[3 * lane + c] = in ? p[c] : 0.0;
      }
      __syncwarp();
      int ncand = 0;
      if constexpr (OCC) {
        double A[3] = {0.0, 0.0, 0.0}, ri;
        line_bounds(a.coords, a.enodes + 8 * i, f_i, A, ri);
        uint32_t some;
        ncand = row_segments(sc, H, T, nseg, warp, A, cj, ri, rj, rj_max, valid, true, gi, gj, some);
      }
      bool flat = true;
#pragma unroll
      for (int k = 0; k < 3; ++k) flat = flat && Xi[3 * k + 2] == 0.0 && Xj[(3 * k + 2) * 32] == 0.0;
      n_pp += valid ? (uint64_t)a.n_samples : 0;
      if (__all_sync(kFull, flat))
        mc_curve_row<OCC, true>(a, sc, T, warp, ncand, P, valid, f_i, f_j, gi, gj, s, Xi, Xj, n_rays, tc);
      else mc_curve_row<OCC, false>(a, sc, T, warp, ncand, P, valid, f_i, f_j, gi, gj, s, Xi, Xj, n_rays, tc);
      __syncwarp();
    }
    __syncthreads();
  }
  mc_count(a, n_pp, n_rays, tc);
}

template <class K>
static cudaError_t mc_shape(K kernel, int threads, size_t smem, int& per_sm) {
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  per_sm = 1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess || per_sm < 1)
    per_sm = 1;
  return e;
}
static cudaError_t mc_pairs_shape(const McArgs& a, int& per_sm) {
  const bool occ = a.n_nodes > 0;
  if (a.dim3) return occ ? mc_shape(k_mc_rows<true>, 256, 8 * sizeof(McRow), per_sm)
                         : mc_shape(k_mc_rows<false>, 256, 8 * sizeof(McRow), per_sm);
  return occ ? mc_shape(k_mc_curves<true>, 256, sizeof(SegTile), per_sm) : mc_shape(k_mc_curves<false>, 256, 0, per_sm);
}

int mc_resident_blocks(const McArgs& a, int sm_count) {
  int per_sm = 1;
  mc_pairs_shape(a, per_sm);
  return sm_count * per_sm;
}

cudaError_t launch_mc_bounds(const McBoundsArgs& a, cudaStream_t st) {
  if (a.N <= 0) return cudaSuccess;
  k_mc_bounds<<<(unsigned)((a.N + 127) / 128), 128, 0, st>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_mc(const McArgs& a, int sm_count, cudaStream_t st) {
  if (a.N == 0) return cudaSuccess;
  if (a.area_pass) {
    k_mc_area<<<(unsigned)((a.N + 127) / 128), 128, 0, st>>>(a);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  if (a.tile_count <= 0) return cudaSuccess;
  // persistent blocks, as many as are resident at once; a claim is a tile's 32
  // rows for the blocks of a curve mesh, four for the warps of a surface mesh,
  // and fewer rows while that leaves a block or warp less than eight claims
  const bool occ = a.n_nodes > 0;
  int per_sm = 1;
  cudaError_t e = mc_pairs_shape(a, per_sm);
  if (e != cudaSuccess) return e;
  McArgs b = a;
  const int64_t blocks = (int64_t)sm_count * per_sm, workers = a.dim3 ? 8 * blocks : blocks;
  b.rows = a.dim3 ? 4 : kTile;
  const int least = a.dim3 ? 1 : 8;
  // Curves among more segments than a tile's list holds: the rows that walk the tree take
  // hundreds of times as long as the others, so a claim is a row for each warp.  Cavities
  // of 3,016 / 3,800 Line3 with 3,000 segments, 16 samples: 70 / 80 to 90 ms with whole tiles,
  // 21 / 30 ms so (58 / 61 ms with a tree walk for each pair, before there were lists).
  const bool uneven = !a.dim3 && occ && a.n_segs > kSegs;
  while (b.rows > least && (uneven || a.tile_count * (kTile / b.rows) < 8 * workers)) b.rows /= 2;
  const int64_t tasks = a.tile_count * (kTile / b.rows), per_block = a.dim3 ? 8 : 1;
  const unsigned grid = (unsigned)std::min<int64_t>(blocks, (tasks + per_block - 1) / per_block);
  if (!a.dim3) {
    if (occ) k_mc_curves<true><<<grid, 256, sizeof(SegTile), st>>>(b);
    else k_mc_curves<false><<<grid, 256, 0, st>>>(b);
    return cudaGetLastError();
  }
  if (occ) {
    // the blockable pairs first: their warps' work is the more uneven
    int q_sm = 1;
    if ((e = mc_shape(k_mc_queue, 128, 4 * sizeof(McQueue), q_sm)) != cudaSuccess) return e;
    const int64_t q_tasks = (a.tile_count + kMcBundle - 1) / kMcBundle * kMcShare;
    k_mc_queue<<<(unsigned)std::min<int64_t>((int64_t)sm_count * q_sm, (q_tasks + 3) / 4), 128, 4 * sizeof(McQueue), st>>>(b);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    k_mc_rows<true><<<grid, 256, 8 * sizeof(McRow), st>>>(b);
  } else {
    k_mc_rows<false><<<grid, 256, 8 * sizeof(McRow), st>>>(b);
  }
  return cudaGetLastError();
}

}  // namespace rvf
