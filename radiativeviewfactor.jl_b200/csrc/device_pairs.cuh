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
template <bool DIM3, bool OCC, int QB>
__device__ __forceinline__ void gen_fast_fp64_body(const PairArgs& a, const double* iblk, int64_t bi, int64_t bj,
                                                   int li0, int lane, uint32_t& n_pp, uint32_t& n_rays, uint32_t skip = 0) {
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
    const int qmax = __reduce_max_sync(kFull, npj);
    const double* ib = iblk + li;
    double acc = 0.0;
    for (int q0 = 0; q0 < qmax; q0 += QB) {
      double xq[QB][3], nq[QB][3], wq[QB];
#pragma unroll
      for (int u = 0; u < QB; ++u) {
        const int q = q0 + u;
        const bool lq = q < npj;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          xq[u][c] = lq ? jb[(c * pm + q) * kTile] : 0.0;
          nq[u][c] = lq ? jb[((3 + c) * pm + q) * kTile] : 0.0;
        }
        wq[u] = lq ? jb[(6 * pm + q) * kTile] : 0.0;
      }
      double inner[QB];
#pragma unroll
      for (int u = 0; u < QB; ++u) inner[u] = 0.0;
      // k_fast with its grazing branch taken out of the loop: a lane that
      // meets a grazing point pair (either |cos| within 1e-5 of zero) forms
      // the chunk again below with k_fast's own arithmetic
      bool graze = false;
      uint32_t cast = 0;
      const int ulim = npj - q0;
      for (int p = 0; p < npi; ++p) {
        double xi[3], ni[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          xi[c] = ib[(c * pm + p) * kTile];
          ni[c] = ib[((3 + c) * pm + p) * kTile];
        }
        const double wi = ib[(6 * pm + p) * kTile];
        // straight-line over the block: a point q0 + u >= npj has zero
        // normal and weight, so its dj is -0 and its K zero (it only must not
        // ask for the grazing redo)
#pragma unroll
        for (int u = 0; u < QB; ++u) {
          const double rx = xq[u][0] - xi[0], ry = xq[u][1] - xi[1], rz = xq[u][2] - xi[2];
          const double r2 = (rx * rx + ry * ry) + rz * rz;
          const double di = fma(ni[0], rx, fma(ni[1], ry, ni[2] * rz));
          const double dj = -fma(nq[u][0], rx, fma(nq[u][1], ry, nq[u][2] * rz));
          const double thr = 1e-10 * r2;
          const bool big = !(r2 < 1e-30);
          graze = graze || (u < ulim && big && (di * di <= thr || dj * dj <= thr));
          double K = 0.0;
          if (big && di > 0.0 && dj > 0.0)
            K = DIM3 ? (di * dj) * rcp_nr(kPiD * (r2 * r2)) : (di * dj) * rcp_nr(2.0 * (r2 * sqrt(r2)));
          cast += K > 0.0 ? 1 : 0;
          inner[u] = fma(wi, K, inner[u]);
        }
      }
      if (__any_sync(kFull, graze) && graze) {  // rare: the chunk again, exactly as the ray pipeline forms it
        cast = 0;
#pragma unroll
        for (int u = 0; u < QB; ++u) inner[u] = 0.0;
        for (int p = 0; p < npi; ++p) {
          double xi[3], ni[3];
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            xi[c] = ib[(c * pm + p) * kTile];
            ni[c] = ib[((3 + c) * pm + p) * kTile];
          }
          const double wi = ib[(6 * pm + p) * kTile];
#pragma unroll
          for (int u = 0; u < QB; ++u) {
            if (q0 + u < npj) {
              const double rx = xq[u][0] - xi[0], ry = xq[u][1] - xi[1], rz = xq[u][2] - xi[2];
              const double r2 = (rx * rx + ry * ry) + rz * rz;
              // k_fast, with the reference formula in line
              double K = 0.0;
              if (!(r2 < 1e-30)) {
                const double di = fma(ni[0], rx, fma(ni[1], ry, ni[2] * rz));
                const double dj = -fma(nq[u][0], rx, fma(nq[u][1], ry, nq[u][2] * rz));
                const double thr = 1e-10 * r2;
                if (di * di <= thr || dj * dj <= thr) K = k_reference_inl<DIM3>(rx, ry, rz, r2, ni, nq[u]);
                else if (di > 0.0 && dj > 0.0)
                  K = DIM3 ? (di * dj) * rcp_nr(kPiD * (r2 * r2)) : (di * dj) * rcp_nr(2.0 * (r2 * sqrt(r2)));
              }
              cast += K > 0.0 ? 1 : 0;
              inner[u] = fma(wi, K, inner[u]);
            }
          }
        }
      }
      if (OCC) n_rays += cast;
#pragma unroll
      for (int u = 0; u < QB; ++u)
        if (q0 + u < npj) acc = fma(wq[u], inner[u], acc);
    }
    n_pp += (uint32_t)(npi * npj);
    if (valid) {
      a.F[oi + oj * N] = acc / a.area[i];
      a.F[oj + oi * N] = acc / a.area[j];
    } else if (j == i) {
      a.F[oi + oi * N] = 0.0 / a.area[i];
    }
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

// Out of line inside the chunked generation kernels, whose own registers are
// allocated for the ray pipeline.
template <bool DIM3, bool OCC, int QB>
__device__ __noinline__ void gen_fast_fp64(const PairArgs& a, const double* iblk, int64_t bi, int64_t bj, int li0, int lane, uint32_t& n_pp,
    uint32_t& n_rays, uint32_t skip = 0) {
  gen_fast_fp64_body<DIM3, OCC, QB>(a, iblk, bi, bj, li0, lane, n_pp, n_rays, skip);
}
template <bool OCC, int QB>
__device__ __noinline__ void gen_fast_mixed(const MixedArgs& a, const float* iblk, int64_t bi, int64_t bj, int li0, int lane, uint32_t& n_pp,
    uint32_t& n_rays, uint32_t skip = 0) {
  gen_fast_mixed_body<OCC, QB>(a, iblk, bi, bj, li0, lane, n_pp, n_rays, skip);
}

// The fast loop with the point block for the rule's size (li0 as there).
template <bool DIM3, bool OCC>
__device__ __forceinline__ void fast_fp64(const PairArgs& a, const double* iblk, int64_t bi, int64_t bj, int li0, int lane, uint32_t& n_pp,
    uint32_t& n_rays, uint32_t skip = 0) {
  if (a.pmax <= 3) gen_fast_fp64<DIM3, OCC, 3>(a, iblk, bi, bj, li0, lane, n_pp, n_rays, skip);
  else gen_fast_fp64<DIM3, OCC, 4>(a, iblk, bi, bj, li0, lane, n_pp, n_rays, skip);
}
template <bool OCC>
__device__ __forceinline__ void fast_mixed(const MixedArgs& a, const float* iblk, int64_t bi, int64_t bj, int li0, int lane, uint32_t& n_pp,
    uint32_t& n_rays, uint32_t skip = 0) {
  const int pm = a.pmax;
  if (pm == 7 || pm == 13 || pm == 49) gen_fast_mixed<OCC, 7>(a, iblk, bi, bj, li0, lane, n_pp, n_rays, skip);
  else if (pm == 5 || pm == 25) gen_fast_mixed<OCC, 5>(a, iblk, bi, bj, li0, lane, n_pp, n_rays, skip);
  else if (pm == 3 || pm == 9) gen_fast_mixed<OCC, 3>(a, iblk, bi, bj, li0, lane, n_pp, n_rays, skip);
  else gen_fast_mixed<OCC, 8>(a, iblk, bi, bj, li0, lane, n_pp, n_rays, skip);
}

}  // namespace rvf
