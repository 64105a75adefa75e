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
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

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
  // v / (2^53 - 1): v < 2^53 put together from its halves (exact), the division by div_by
  const uint64_t v = s >> 11;
  constexpr double kMax = 9007199254740991.0;
  const double d = (__hiloint2double(0x45300000, (int)(v >> 32)) - (0x1p84 + 0x1p52)) +
                   __hiloint2double(0x43300000, (int)(uint32_t)v);
  return div_by(d, kMax, 1.0 / kMax);
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

// sample k of a pair's stream: the two reference coordinates
__device__ __forceinline__ void mc_coords(bool dim3, int k, int s, double inv_s, uint64_t& st, double* ci,
                                          double* cj) {
  const double u1 = xorshift64(st), u2 = xorshift64(st), u3 = xorshift64(st), u4 = xorshift64(st);
  if (k < s * s) {
    const int si = k / s, sj = k - si * s;
    // (si + u) / s with inv_s = 1 / s (the numerators are 0 or at least 2^-53)
    if (dim3) {
      ci[0] = div_by(si + u1, s, inv_s); ci[1] = div_by(sj + u2, s, inv_s);
      cj[0] = div_by(si + u3, s, inv_s); cj[1] = div_by(sj + u4, s, inv_s);
    } else {
      ci[0] = 2.0 * div_by(si + u1, s, inv_s) - 1.0; ci[1] = 0.0;
      cj[0] = 2.0 * div_by(sj + u3, s, inv_s) - 1.0; cj[1] = 0.0;
    }
  } else if (dim3) {
    ci[0] = u1; ci[1] = u2; cj[0] = u3; cj[1] = u4;
  } else {
    ci[0] = 2.0 * u1 - 1.0; ci[1] = 0.0; cj[0] = 2.0 * u3 - 1.0; cj[1] = 0.0;
  }
}

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
// (device_segs.cuh), and each sample tests only these, each behind the overlap
// test of its own leaf (the walk's test at that leaf: the leaf box lies inside
// every ancestor's, so the test passing there means the reference's walk
// reaches it), with the reference's own segment test.  Decisions are identical
// to the full walk's.  Pairs with more than kPairSegs segments, and tiles whose
// list overflows, walk the tree for every sample.
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
  uint64_t st = init_rng(a.seed, (uint64_t)(lo * N + hi + 1));
  const int64_t ie = a.inv[e];
  const int f = a.fam[ie];
  const int32_t* en = a.enodes + 8 * ie;
  const int s = (int)floor(sqrt((double)a.n_samples));
  double A = 0.0;
  for (int k = 0; k < a.n_samples; ++k) {
    double ci[2], cj[2];
    mc_coords(a.dim3, k, s, 1.0 / s, st, ci, cj);
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
// Out of line: the families' geometry does not hold the pair kernel's registers.
struct McPoint {
  double x[3], n[3], dA;
};
template <int F>
__device__ __forceinline__ McPoint mc_eval_family(const double* X, int stride, double xi, double eta) {
  constexpr int nn = F == 0 ? 8 : F == 1 ? 6 : F == 2 ? 4 : 3;
  double N[8], dX[8], dE[8];
  shape_surface(F, xi, eta, N, dX, dE);
  McPoint r;
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
  return r;
}
__device__ __noinline__ McPoint mc_eval(int f, const double* X, int stride, double u, double v) {
  if (is_quad_fam(f)) {
    u = 2.0 * u - 1.0;
    v = 2.0 * v - 1.0;
    return f == 0 ? mc_eval_family<0>(X, stride, u, v) : mc_eval_family<2>(X, stride, u, v);
  }
  if (u + v > 1.0) {
    u = 1.0 - u;
    v = 1.0 - v;
  }
  return f == 1 ? mc_eval_family<1>(X, stride, u, v) : mc_eval_family<3>(X, stride, u, v);
}
// Line3 / Line2 (eval_line): three or two nodes.
__device__ __forceinline__ McPoint mc_eval_line(int f, const double (&X)[9], double xi) {
  double N[3], dN[3];
  if (f == 4) {
    N[0] = ((-0.5) * xi) * (1.0 - xi); N[1] = (0.5 * xi) * (1.0 + xi); N[2] = 1.0 - xi * xi;
    dN[0] = -0.5 + xi; dN[1] = 0.5 + xi; dN[2] = -2.0 * xi;
  } else {
    N[0] = 0.5 * (1.0 - xi); N[1] = 0.5 * (1.0 + xi); N[2] = 0.0;
    dN[0] = -0.5; dN[1] = 0.5; dN[2] = 0.0;
  }
  double p[3] = {0.0, 0.0, 0.0}, t[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int k = 0; k < 3; ++k)
    if (k < 2 || f == 4) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        p[c] = p[c] + N[k] * X[3 * k + c];
        t[c] = t[c] + dN[k] * X[3 * k + c];
      }
    }
  McPoint r;
  r.dA = sqrt((t[0] * t[0] + t[1] * t[1]) + t[2] * t[2]);
  const double tt[2] = {t[0], t[1]};
  double q[2];
  div_all(tt, r.dA, q);
#pragma unroll
  for (int c = 0; c < 3; ++c) r.x[c] = p[c];
  r.n[0] = -q[1];
  r.n[1] = q[0];
  r.n[2] = 0.0;
  return r;
}

struct McTile {
  double xi[32 * 24];  // row elements' node coordinates, 24 a row element
  double xj[24 * 32];  // column elements', value v of lane l at 32 v + l
};

// A block claims a tile (or a part of its rows); warps take rows, a lane a
// pair.  Both elements' node coordinates are staged in shared memory per tile:
// the samples' evaluations were gathers of indices and coordinates.  The kernel
// is symmetric in the two elements bit for bit (the cosines swap and every
// difference changes sign exactly), so a row keeps one source element whatever
// the reference's order of the pair; only the draws, the product's order and the
// ray's direction follow it.  Bound by FP64 issue: about 500 FP64 instructions a
// sample pair, a division and a square root per normalisation and for the
// kernel, the other quotients by div_by.
template <bool DIM3, bool OCC>
__global__ void __launch_bounds__(256, 2) k_pairs_mc(McArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  McTile& T = *reinterpret_cast<McTile*>(smem);
  SegTile& ST = *reinterpret_cast<SegTile*>(smem + sizeof(McTile));  // curves with occlusion
  __shared__ int64_t s_tile;
  __shared__ int s_row, s_end, s_segs;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t N = a.N;
  const int s = (int)floor(sqrt((double)a.n_samples));
  const double inv_s = 1.0 / s;
  uint64_t n_rays = 0, n_pp = 0;
  TravCount tc;
  for (;;) {
    if (threadIdx.x == 0) {
      const unsigned long long k = atomicAdd(a.tile_counter, 1ull);
      const int64_t tl = (int64_t)(k / (unsigned)a.groups);
      const int part = (int)(k - (unsigned long long)tl * (unsigned)a.groups);
      s_tile = tl < a.tile_count ? a.tile0 + tl : -1;
      s_row = part * (kTile / a.groups);
      s_end = s_row + kTile / a.groups;
    }
    __syncthreads();
    const int64_t t = s_tile;
    if (t < 0) break;
    int64_t bi, bj;
    tile_coords(t, a.nT, bi, bj);
    for (int v = threadIdx.x; v < 32 * 8; v += 256) {
      const int el = v & 31, k = v >> 5;  // element of the block, node
      const int64_t ei = bi * kTile + el, ej = bj * kTile + el;
      const bool oki = ei < N && k < fam_nodes(a.fam[ei < N ? ei : 0]), okj = ej < N && k < fam_nodes(a.fam[ej < N ? ej : 0]);
      const double* pi = a.coords + 3 * (int64_t)(oki ? a.enodes[8 * ei + k] : 0);
      const double* pj = a.coords + 3 * (int64_t)(okj ? a.enodes[8 * ej + k] : 0);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        T.xi[24 * el + 3 * k + c] = oki ? pi[c] : 0.0;
        T.xj[32 * (3 * k + c) + el] = okj ? pj[c] : 0.0;
      }
    }
    __syncthreads();
    const int64_t j = bj * kTile + lane;
    const bool okj = j < N;
    const int64_t oj = okj ? (int64_t)a.orig[j] : 0;
    const int f_j = okj ? a.fam[j] : a.fam[bj * kTile];
    const int32_t g_j = okj ? a.group[j] : 0;
    const double* Xj = T.xj + lane;
    // surfaces: the tile's class; a pair outside its row's mask has no
    // sample ray that can be blocked (its rays skip the traversal)
    const uint8_t tcl = (DIM3 && OCC && a.tcls) ? a.tcls[t] : (uint8_t)kClsSlow;
    // curves: the segments within reach of the tile
    HullF H;
    double cj[3] = {0.0, 0.0, 0.0}, rj = 0.0, rj_max = 0.0;
    int nseg = 0;
    SegScene sc;
    if constexpr (!DIM3 && OCC) {
      sc = SegScene{a.nodes, a.nodesf, a.n_nodes, a.segs, a.frontier, a.n_frontier, a.cand_margin, a.seg_slack};
      const int64_t ei = bi * kTile + lane;
      double cc[3] = {0.0, 0.0, 0.0}, ri = 0.0, rmax;
      if (ei < N) line_bounds(a.coords, a.enodes + 8 * ei, a.fam[ei], cc, ri);
      if (okj) line_bounds(a.coords, a.enodes + 8 * j, f_j, cj, rj);
      tile_hull(ei < N, okj, cc, cj, ri, rj, H, rmax, rj_max);
      const int32_t g_i = ei < N ? a.group[ei] : 0, gi0 = __shfl_sync(kFull, g_i, 0), gj0 = __shfl_sync(kFull, g_j, 0);
      const bool g_same = a.exclude && __all_sync(kFull, (ei >= N || g_i == gi0) && (!okj || g_j == gj0));
      if (warp == 0) {
        const int n = tile_segments(sc, H, rmax, g_same, gi0, gj0, ST);
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
      const bool may_block =
          !(DIM3 && OCC && a.tcls) || ((tcl & kClsSlow) && ((a.tmask[t * kTile + li] >> lane) & 1u));
      const bool valid = okj && i < j;
      const int64_t oi = a.orig[i];
      const bool sw = valid && oi > oj;
      // the reference's pair (lo, hi): lo samples with u1,u2 and casts the ray
      const int64_t o_lo = sw ? oj : oi, o_hi = sw ? oi : oj;
      const int f_i = a.fam[i];
      const int32_t gi = a.group[i];
      const int32_t gx = a.exclude ? gi : 0, gy = a.exclude ? g_j : 0;
      uint64_t st = init_rng(a.seed, (uint64_t)(o_lo * N + o_hi + 1));
      uint8_t* logp = (a.ray_log && valid) ? a.ray_log + ((uint64_t)o_lo * N + o_hi) * a.n_samples : nullptr;
      const double* Xi = T.xi + 24 * li;
      int ncand = 0;
      double Li[9], Lj[9];
      if constexpr (!DIM3) {
#pragma unroll
        for (int k = 0; k < 9; ++k) {
          Li[k] = Xi[k];
          Lj[k] = Xj[32 * k];
        }
        if constexpr (OCC) {
          double A[3] = {0.0, 0.0, 0.0}, ri;
          line_bounds(a.coords, a.enodes + 8 * i, f_i, A, ri);
          ncand = pair_segments(sc, H, ST, nseg, warp, A, cj, ri, rj, rj_max, valid, a.exclude, gi, g_j);
        }
      }
      double Ks = 0.0;
      for (int k = 0; k < a.n_samples; ++k) {
        double ulo[2], uhi[2];
        mc_coords(DIM3, k, s, inv_s, st, ulo, uhi);
        McPoint pi, pj;
        if constexpr (DIM3) {
          pi = mc_eval(f_i, Xi, 1, sw ? uhi[0] : ulo[0], sw ? uhi[1] : ulo[1]);
          pj = mc_eval(f_j, Xj, 32, sw ? ulo[0] : uhi[0], sw ? ulo[1] : uhi[1]);
        } else {
          pi = mc_eval_line(f_i, Li, sw ? uhi[0] : ulo[0]);
          pj = mc_eval_line(f_j, Lj, sw ? ulo[0] : uhi[0]);
        }
        const double rx = pj.x[0] - pi.x[0], ry = pj.x[1] - pi.x[1], rz = pj.x[2] - pi.x[2];
        const double r2 = (rx * rx + ry * ry) + rz * rz;
        double K = 0.0;
        if (valid && !(r2 < 1e-30)) K = k_reference_inl<DIM3>(rx, ry, rz, r2, pi.n, pj.n);
        n_pp += valid ? 1 : 0;
        if (OCC) {
          uint8_t lg = 0;
          if constexpr (DIM3) {
            RayD R;
            const bool cast = K > 0.0 && (r2 > 2e-30 || sqrt(r2) > 1e-15);  // make_ray's cast rule
            n_rays += cast ? 1 : 0;
            bool blocked = false;
            if (__any_sync(kFull, cast && may_block)) {
              if (cast && may_block) {
                if (sw) make_ray(pj.x, -rx, -ry, -rz, r2, R);
                else make_ray(pi.x, rx, ry, rz, r2, R);
              }
              blocked = packet_any_hit(
                  cast && may_block, a.nodes, a.n_nodes, [&](const NodeD& nd) { return slab_d(nd, R); },
                  [&](int kk, bool test) {
                    const TriD tr = a.tris[kk];
                    if (!test || tr.group == gx || tr.group == gy) return false;
                    ++tc.prims;
                    return mt_d(tr, R);
                  },
                  tc);
            }
            if (cast) lg = blocked ? 2 : 1;
            if (blocked) K = 0.0;
          } else {
            const bool cast = K > 0.0;
            n_rays += cast ? 1 : 0;
            const double from[2] = {sw ? pj.x[0] : pi.x[0], sw ? pj.x[1] : pi.x[1]};
            const double to[2] = {sw ? pi.x[0] : pj.x[0], sw ? pi.x[1] : pj.x[1]};
            const double lx = fmin(from[0], to[0]), hx = fmax(from[0], to[0]);
            const double ly = fmin(from[1], to[1]), hy = fmax(from[1], to[1]);
            bool blocked = false;
            if (cast && ncand > 0)
              blocked = list_blocks(sc, ST, warp, ncand, lx, hx, ly, hy, from, to, tc.nodes, tc.prims);
            const bool walk = cast && ncand < 0;
            if (__any_sync(kFull, walk)) {
              const bool bw = packet_any_hit(
                  walk, a.nodes, a.n_nodes,
                  [&](const NodeD& nd) {
                    return !(nd.lo[0] > hx || nd.hi[0] < lx || nd.lo[1] > hy || nd.hi[1] < ly);
                  },
                  [&](int kk, bool test) {
                    const SegD sg = a.segs[kk];
                    if (!test || sg.group == gx || sg.group == gy) return false;
                    ++tc.prims;
                    return seg_blocks(sg, from, to);
                  },
                  tc);
              if (walk) blocked = bw;
            }
            if (cast) lg = blocked ? 2 : 1;
            if (blocked) K = 0.0;
          }
          if (logp) logp[k] = lg;
        }
        Ks += (K * (sw ? pj.dA : pi.dA)) * (sw ? pi.dA : pj.dA);
      }
      if (valid) {
        const int f_lo = sw ? f_j : f_i, f_hi = sw ? f_i : f_j;
        const double raw = ((Ks * ref_measure(f_lo)) * ref_measure(f_hi)) / (double)a.n_samples;
        a.F[oi + oj * N] = raw / a.area_orig[oi];
        a.F[oj + oi * N] = raw / a.area_orig[oj];
      } else if (j == i) {
        a.F[oi + oi * N] = 0.0 / a.area_orig[oi];
      }
      __syncwarp();
    }
    __syncthreads();
  }
  n_rays = warp_sum_u64(n_rays);
  n_pp = warp_sum_u64(n_pp);
  const uint64_t s_nodes = warp_sum_u64(tc.nodes), s_prims = warp_sum_u64(tc.prims);
  if (lane == 0 && a.counters) {
    atomicAdd(a.counters + 0, n_pp);
    atomicAdd(a.counters + 1, n_rays);
    atomicAdd(a.counters + 2, s_nodes);
    atomicAdd(a.counters + 3, s_prims);
  }
}

template <bool D3, bool O>
static cudaError_t mc_shape(int& per_sm, size_t& smem) {
  smem = sizeof(McTile) + (!D3 && O ? sizeof(SegTile) : 0);
  const cudaError_t e = cudaFuncSetAttribute(k_pairs_mc<D3, O>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  per_sm = 1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pairs_mc<D3, O>, 256, smem) != cudaSuccess || per_sm < 1)
    per_sm = 1;
  return e;
}

template <bool D3, bool O>
static cudaError_t launch_mc_t(McArgs a, int sm_count, cudaStream_t st) {
  // persistent blocks: as many as are resident at once; small launches split
  // tiles into parts of their rows, so that the blocks have eight tasks each
  int per_sm = 1;
  size_t smem = 0;
  const cudaError_t e = mc_shape<D3, O>(per_sm, smem);
  if (e != cudaSuccess) return e;
  int64_t grid = (int64_t)sm_count * per_sm;
  a.groups = a.tile_count >= 8 * grid ? 1 : 2 * a.tile_count >= 8 * grid ? 2 : 4;
  grid = std::min<int64_t>(grid, a.tile_count * a.groups);
  k_pairs_mc<D3, O><<<(unsigned)grid, 256, smem, st>>>(a);
  return cudaGetLastError();
}

int mc_resident_blocks(const McArgs& a, int sm_count) {
  const bool occ = a.n_nodes > 0;
  int per_sm = 1;
  size_t smem = 0;
  if (a.dim3) occ ? mc_shape<true, true>(per_sm, smem) : mc_shape<true, false>(per_sm, smem);
  else occ ? mc_shape<false, true>(per_sm, smem) : mc_shape<false, false>(per_sm, smem);
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
  const bool occ = a.n_nodes > 0;
  if (a.dim3) return occ ? launch_mc_t<true, true>(a, sm_count, st) : launch_mc_t<true, false>(a, sm_count, st);
  return occ ? launch_mc_t<false, true>(a, sm_count, st) : launch_mc_t<false, false>(a, sm_count, st);
}

}  // namespace rvf
