// kernels_occ2d.cu -- curve meshes with obstructions: quadrature, shadow
// segments and F of a tile in one kernel.
//
// Replaces _vf_pair_kernel! (src/GPUKernels.jl:226-323) for curves, whose rays
// the reference walks through the whole segment tree (src/BVH.jl:265-322).  A
// block claims a tile and collects the segments within reach of the tile's
// hull; row by row, a lane per pair lists those within reach of its own capsule
// (the segment between the elements' centroids grown by their
// point radius and by cand_margin, which bounds how far from a ray a computed
// hit of the segment test can lie).  Pairs with an empty list have visible rays
// only and run the quadrature-only loop; the others test each ray against their
// listed segments, each behind the overlap test of its own leaf (the leaf box
// lies in every ancestor's, so the reference's walk reaches it exactly when it
// passes), with the reference's segment test: the decisions are the walk's.  A
// tile with more than kSegs segments within reach, or a pair with more than
// kPairSegs, walks the tree for every ray.
//
// Measured on a B200, 2-D cavity of 4,000 Line3 with four circles of 200 as
// obstruction, nquad 4: 4.8 ms a solve; walking the tree for every ray took
// 47 ms (39 segment and 16 box tests a ray, from shared memory at 79% of its
// bandwidth).  Bound by FP64 issue.
#include <cuda_runtime.h>

#include <cstdint>

#include "device_hull.cuh"
#include "device_pairs.cuh"

namespace rvf {

namespace {

constexpr int kSegs = 2048;  // segments of a tile's list
constexpr int kPairSegs = 24;  // of a pair's (more: its rays walk the tree)
constexpr int kFront = kTileFront;

struct SegTile {
  int seg[kSegs];    // segment
  int leaf[kSegs];   // its leaf node
  union {
    struct {
      int front[2 * kFront];
      int leaves[kTileLeaves];
    } walk;
    uint16_t list[8][kPairSegs][32];  // per warp: the row's pairs' lists (positions in the tile's)
  };
};

// True when the hull (of two boxes of FP32 centres and half extents, x and y)
// is farther than m from the box [lo, hi].
__device__ __forceinline__ bool hull2_misses(const HullF& H, float lx, float ly, float hx, float hy, float m) {
  const float ax = fminf(H.c[0][0] - H.h[0][0], H.c[1][0] - H.h[1][0]), bx = fmaxf(H.c[0][0] + H.h[0][0], H.c[1][0] + H.h[1][0]);
  const float ay = fminf(H.c[0][1] - H.h[0][1], H.c[1][1] - H.h[1][1]), by = fmaxf(H.c[0][1] + H.h[0][1], H.c[1][1] + H.h[1][1]);
  if (lx - bx > m || ax - hx > m || ly - by > m || ay - hy > m) return true;
  // the normal of the centroid direction
  const float wx = -H.d[1], wy = H.d[0];
  const float bm = 0.5f * ((lx + hx) * wx + (ly + hy) * wy);
  const float br = 0.5f * ((hx - lx) * fabsf(wx) + (hy - ly) * fabsf(wy));
  return hull_gap(H, wx, wy, 0.0f, bm - br, bm + br, m);
}

// True when the segment (s0, s1) is farther than R from the segment a -> a + d
// (L = |d|), by one of three axes.
__device__ __forceinline__ bool capsule2_misses(const double* a, const double* d, double L2, double RL, double R,
                                                const double* s0, const double* s1) {
  const double u0 = s0[0] - a[0], u1 = s0[1] - a[1], v0 = s1[0] - a[0], v1 = s1[1] - a[1];
  const double cu = d[0] * u1 - d[1] * u0, cv = d[0] * v1 - d[1] * v0;
  if (fmin(cu, cv) > RL || fmax(cu, cv) < -RL) return true;
  const double du = d[0] * u0 + d[1] * u1, dv = d[0] * v0 + d[1] * v1;
  if (fmax(du, dv) < -RL || fmin(du, dv) > L2 + RL) return true;
  const double e0 = v0 - u0, e1 = v1 - u1;
  const double ea = e1 * u0 - e0 * u1, eb = ea - (e1 * d[0] - e0 * d[1]);  // both ends of the centroid segment
  const double m2 = R * R * (e0 * e0 + e1 * e1);
  return ((ea > 0.0) == (eb > 0.0)) && fmin(ea * ea, eb * eb) > m2;
}

}  // namespace

__global__ void __launch_bounds__(256, 2) k_occ2d(const OccBatch* __restrict__ Lp) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ SegTile T;
  const OccBatch& B = *Lp;
  __shared__ int64_t s_tile;
  __shared__ int s_req, s_part, s_row, s_segs;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* S = reinterpret_cast<double*>(smem) + warp * 8 * B.pmax_max;
  uint32_t n_pp = 0, n_rays = 0, n_nodes = 0, n_prims = 0, n_traced = 0;
  for (;;) {
    if (threadIdx.x == 0) {
      const unsigned long long k = atomicAdd(B.q.ctr + kCtrTile, 1ull);
      const int64_t g = (int64_t)(k / (unsigned)B.groups);
      s_tile = -1;
      if (g < B.total_tiles) {
        s_req = find_req(B.tile_base, B.n_req, g);
        s_part = (int)(k - (unsigned long long)g * (unsigned)B.groups);
        s_tile = g - B.tile_base[s_req] + B.reqs[s_req].tile0;
        s_row = s_part * (kTile / B.groups);
      }
      s_segs = 0;
    }
    __syncthreads();
    if (s_tile < 0) break;
    const OccArgs& t = B.reqs[s_req];
    const PairArgs& a = B.preqs[s_req];
    const int row1 = (s_part + 1) * (kTile / B.groups);
    const int64_t N = t.N;
    const int pm = t.pmax;
    int64_t bi, bj;
    tile_coords(s_tile, t.nT, bi, bj);
    const int64_t ei = bi * kTile + lane, j = bj * kTile + lane;
    const bool oki = ei < N, okj = j < N;
    double cj[3] = {0.0, 0.0, 0.0}, rj = 0.0;
    int32_t gj = 0;
    if (okj) {
      cj[0] = t.cen[3 * j]; cj[1] = t.cen[3 * j + 1];
      rj = t.rad[j];
      gj = t.group[j];
    }
    double cc[3] = {0.0, 0.0, 0.0}, ri = 0.0;
    int32_t gi = 0;
    if (oki) {
      cc[0] = t.cen[3 * ei]; cc[1] = t.cen[3 * ei + 1];
      ri = t.rad[ei];
      gi = t.group[ei];
    }
    HullF H;
    double rmax, rj_max;
    tile_hull(oki, okj, cc, cj, ri, rj, H, rmax, rj_max);
    const int32_t gi0 = __shfl_sync(kFull, gi, 0), gj0 = __shfl_sync(kFull, gj, 0);
    const bool g_same = __all_sync(kFull, (!oki || gi == gi0) && (!okj || gj == gj0));
    // FP32 coordinates: 2^-20 of the scene's extent
    const float reach = __double2float_ru(rmax + t.cand_margin) + t.delta;
    if (warp == 0) {  // the leaves within reach, one tree level per round
      int* cur = T.walk.front;
      int* nxt = T.walk.front + kFront;
      if (lane < t.n_frontier) cur[lane] = t.frontier[lane];
      __syncwarp();
      int ncur = t.n_frontier, nleaf = 0;
      bool over = false;
      while (ncur > 0 && !over) {
        int nnext = 0;
        for (int b = 0; b < ncur; b += 32) {
          const int q = b + lane;
          bool pass = false, leaf = false;
          int k = 0, right = 0;
          if (q < ncur && cur[q] < t.n_nodes) {
            k = cur[q];
            const NodeF nd = t.nodesf[k];
            pass = !hull2_misses(H, nd.lo[0], nd.lo[1], nd.hi[0], nd.hi[1], reach);
            leaf = (nd.ab & 15) > 0;
            if (pass && !leaf) right = t.nodesf[k + 1].miss;
          }
          const uint32_t ml = __ballot_sync(kFull, pass && leaf), mi = __ballot_sync(kFull, pass && !leaf);
          const int pl = nleaf + __popc(ml & lanemask_lt());
          if (pass && leaf && pl < kTileLeaves) T.walk.leaves[pl] = k;
          nleaf += __popc(ml);
          const int pi = nnext + 2 * __popc(mi & lanemask_lt());
          if (pass && !leaf && pi + 1 < kFront) {
            nxt[pi] = k + 1;
            nxt[pi + 1] = right;
          }
          nnext += 2 * __popc(mi);
        }
        __syncwarp();
        if (nleaf > kTileLeaves || nnext > kFront) over = true;
        int* tmp = cur;
        cur = nxt;
        nxt = tmp;
        ncur = nnext;
      }
      // their segments, four leaves per round
      int ns = 0;
      for (int b = 0; b < nleaf && !over; b += 4) {
        const int li = b + (lane >> 3), u8 = lane & 7;
        bool keep = false;
        int leaf = 0, u = 0;
        if (li < nleaf) {
          leaf = T.walk.leaves[li];
          const int32_t ab = t.nodesf[leaf].ab;
          if (u8 < (ab & 15)) {
            u = (ab >> 4) + u8;
            const SegD sg = t.segs[u];
            const float x0 = (float)sg.x0, y0 = (float)sg.y0, x1 = (float)sg.x1, y1 = (float)sg.y1;
            keep = !(g_same && (sg.group == gi0 || sg.group == gj0)) &&
                   !hull2_misses(H, fminf(x0, x1), fminf(y0, y1), fmaxf(x0, x1), fmaxf(y0, y1), reach);
          }
        }
        const uint32_t m = __ballot_sync(kFull, keep);
        const int at = ns + __popc(m & lanemask_lt());
        if (keep && at < kSegs) {
          T.seg[at] = u;
          T.leaf[at] = leaf;
        }
        ns += __popc(m);
      }
      if (lane == 0) s_segs = over || ns > kSegs ? -1 : ns;
    }
    __syncthreads();
    const int nseg = s_segs;
    for (;;) {  // rows, as the warps get to them
      int li = 0;
      if (lane == 0) li = atomicAdd(&s_row, 1);
      li = __shfl_sync(kFull, li, 0);
      if (li >= row1) break;
      const int64_t i = bi * kTile + li;
      if (i >= N) break;
      const bool valid = okj && i < j;
      // the lane's pair: its segments, or n = -1 (its rays walk the tree)
      int n = nseg < 0 && valid ? -1 : 0;
      if (nseg > 0) {
        const double A[2] = {t.cen[3 * i], t.cen[3 * i + 1]};
        const double d[2] = {cj[0] - A[0], cj[1] - A[1]};
        const double L2 = d[0] * d[0] + d[1] * d[1], R = fmax(t.rad[i], rj) + t.cand_margin, RL = R * sqrt(L2);
        const int32_t g_i = t.group[i];
        // the row's own hull: its centroid and the column block's box
        HullF Hr;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const float l = __double2float_rd(A[k]), h = __double2float_ru(A[k]);
          Hr.c[0][k] = 0.5f * (l + h);
          Hr.h[0][k] = 0.5f * (h - l);
          Hr.c[1][k] = H.c[1][k];
          Hr.h[1][k] = H.h[1][k];
          Hr.d[k] = Hr.c[1][k] - Hr.c[0][k];
        }
        Hr.c[0][2] = Hr.h[0][2] = Hr.c[1][2] = Hr.h[1][2] = Hr.d[2] = 0.0f;
        const float row_reach = __double2float_ru(fmax(t.rad[i], rj_max) + t.cand_margin) + t.delta;
        for (int b = 0; b < nseg; b += 32) {
          bool keep = false;
          if (b + lane < nseg) {
            const SegD sg = t.segs[T.seg[b + lane]];
            const float x0 = (float)sg.x0, y0 = (float)sg.y0, x1 = (float)sg.x1, y1 = (float)sg.y1;
            keep = sg.group != g_i &&
                   !hull2_misses(Hr, fminf(x0, x1), fminf(y0, y1), fmaxf(x0, x1), fmaxf(y0, y1), row_reach);
          }
          for (uint32_t m = __ballot_sync(kFull, keep); m; m &= m - 1u) {  // lanes are pairs again
            const int at = b + __ffs(m) - 1;
            const SegD sg = t.segs[T.seg[at]];
            const double s0[2] = {sg.x0, sg.y0}, s1[2] = {sg.x1, sg.y1};
            if (valid && n >= 0 && sg.group != gj && !capsule2_misses(A, d, L2, RL, R, s0, s1)) {
              if (n < kPairSegs) T.list[warp][n][lane] = (uint16_t)at;
              n = n < kPairSegs ? n + 1 : -1;
            }
          }
        }
      }
      const bool some = n != 0;
      const uint32_t rest = __ballot_sync(kFull, some);
      fast_fp64<false, true>(a, a.tab + bi * kComp * pm * kTile, S, bi, bj, li + 8, lane, n_pp, n_rays, rest);
      if (rest == 0) continue;  // warp-uniform
      // the pairs with segments in reach (S holds the row's points)
      const int64_t oi = t.orig ? (int64_t)t.orig[i] : i, oj = okj ? (t.orig ? (int64_t)t.orig[j] : j) : 0;
      const bool sw = oi > oj;  // the reference casts from the lower caller index
      const int npi = t.np[i];
      int npj = some ? t.np[j] : 0;
      if (some && t.flat[i] && t.flat[j] && t.nrm[3 * i] == t.nrm[3 * j] && t.nrm[3 * i + 1] == t.nrm[3 * j + 1] &&
          t.nrm[3 * i + 2] == t.nrm[3 * j + 2])
        npj = 0;
      n_pp += (uint32_t)(npi * npj);
      const double* jb = t.tab + bj * kComp * pm * kTile + lane;
      double acc = 0.0;  // twice the pair's sum
      for (int q = 0; q < npj; ++q) {
        double xj[3], nj[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          xj[c] = jb[(c * pm + q) * kTile];
          nj[c] = jb[((3 + c) * pm + q) * kTile];
        }
        double inner = 0.0;
        for (int p = 0; p < npi; ++p) {
          const double xi[3] = {S[8 * p], S[8 * p + 1], S[8 * p + 2]}, ni[3] = {S[8 * p + 4], S[8 * p + 5], S[8 * p + 6]};
          const double rx = xj[0] - xi[0], ry = xj[1] - xi[1], rz = xj[2] - xi[2];
          const double r2 = (rx * rx + ry * ry) + rz * rz;
          const double k = kernel_scaled<false>(rx, ry, rz, r2, ni, nj);
          if (!(k > 0.0)) continue;
          ++n_rays;
          // the segment as the reference passes it, and its bounding box
          const double ax = sw ? xj[0] : xi[0], ay = sw ? xj[1] : xi[1], bx = sw ? xi[0] : xj[0],
                       by = sw ? xi[1] : xj[1];
          const double lx = fmin(ax, bx), hx = fmax(ax, bx), ly = fmin(ay, by), hy = fmax(ay, by);
          const double from[2] = {ax, ay}, to[2] = {bx, by};
          bool blocked = false;
          ++n_traced;
          if (n >= 0) {
            for (int k = 0; k < n && !blocked; ++k) {
              const int at = T.list[warp][k][lane];
              const NodeD& nd = t.nodes[T.leaf[at]];
              ++n_nodes;
              if (nd.lo[0] > hx || nd.hi[0] < lx || nd.lo[1] > hy || nd.hi[1] < ly) continue;
              ++n_prims;
              blocked = seg_blocks(t.segs[T.seg[at]], from, to);
            }
          } else {
            const int32_t g_i = t.group[i];
            for (int k = 0; k < t.n_nodes && !blocked;) {  // miss links point forward
              const NodeD nd = t.nodes[k];
              ++n_nodes;
              if (nd.lo[0] > hx || nd.hi[0] < lx || nd.lo[1] > hy || nd.hi[1] < ly) {
                k = nd.miss;
                continue;
              }
              for (int u = nd.a; u < nd.a + nd.b && !blocked; ++u) {
                const SegD sg = t.segs[u];
                if (sg.group == g_i || sg.group == gj) continue;
                ++n_prims;
                blocked = seg_blocks(sg, from, to);
              }
              k = nd.b > 0 ? nd.miss : k + 1;
            }
          }
          if (!blocked) inner = fma(S[8 * p + 3], k, inner);
        }
        acc = fma(jb[(6 * pm + q) * kTile], inner, acc);
      }
      if (some) {
        const double raw = 0.5 * acc;
        t.F[oi + oj * N] = raw / t.area[i];
        t.F[oj + oi * N] = raw / t.area[j];
      }
      __syncwarp();
    }
    __syncthreads();
  }
  if (B.counters) {
    const uint32_t v[4] = {n_pp, n_rays, n_nodes, n_prims};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint64_t s = warp_sum_u64(v[k]);
      if (lane == 0 && s) atomicAdd(B.counters + k, (unsigned long long)s);
    }
    const uint64_t s = warp_sum_u64(n_traced);
    if (lane == 0 && s) atomicAdd(B.q.ctr + kCtrRec64, (unsigned long long)s);
  }
}

cudaError_t launch_occ2d(int pmax, const OccBatch* b, int sm_count, cudaStream_t st) {
  const size_t smem = stage_bytes(pmax);
  const cudaError_t e = cudaFuncSetAttribute(k_occ2d, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k_occ2d<<<(unsigned)(2 * sm_count), 256, smem, st>>>(b);
  return cudaGetLastError();
}

}  // namespace rvf
