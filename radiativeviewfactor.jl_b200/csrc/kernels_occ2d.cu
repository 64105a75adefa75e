// kernels_occ2d.cu -- curve meshes with obstructions: quadrature, shadow
// segments and F of a tile in one kernel.
//
// Replaces _vf_pair_kernel! (src/GPUKernels.jl:226-323) for curves, whose rays
// the reference walks through the whole segment tree (src/BVH.jl:265-322).  A
// block claims a tile and collects the segments within reach of the tile's
// hull; row by row, a lane per pair lists those within reach of its own capsule
// (the segment between the elements' centroids grown by their
// point radius and by cand_margin, which bounds how far from a ray a computed
// hit of the segment test can lie).  Pairs without one have visible rays only and
// run the quadrature-only loop; the tests of the others' rays are dealt out to the
// lanes, with the reference's segment test; a hit counts when the ray's box
// overlaps the segment's leaf (the leaf box lies in every ancestor's, so the
// reference's walk reaches it exactly when it does): the decisions are the walk's.
// A tile with more than kSegs segments within reach, or a row with more than
// kRowItems tests (half of them in launches of few tiles, whose rows run one
// after another), is deferred: the queue pipeline (kernels_wave.cu), whose rays
// walk the tree, takes its pairs after this kernel.
//
// Measured on a B200, 2-D cavity of 4,000 Line3 with four circles of 200 as
// obstruction, nquad 4: 4.2 ms a solve; walking the tree for every ray took
// 47 ms (39 segment and 16 box tests a ray, from shared memory at 79% of its
// bandwidth), a lane testing its own pair's list 4.8 ms (lists differ in length
// between the lanes).  Bound by issue: a row's set-up weighs against 16 point pairs.
// Fine obstructions, where rows of coarse walls reach thousands of segments (ms,
// rows beyond the lists walking in this kernel / deferred / all in the queue
// pipeline): 3,120 Line3 with 3,000 segments, nquad 8, 129 / 14.2 / 29.0; 832 Line3 with
// 800 segments, nquad 8, 9.8 / 1.9 / 1.5; 2,800 Line3 with 2,000 segments, nquad 3,
// 3.2 / 3.5 / 12.2.  Limits of 256, 512 and 1,024 tests a row were 14%, 5% and 1% slower
// over 121 solves.
#include <cuda_runtime.h>

#include <cstdint>

#include "device_pairs.cuh"
#include "device_segs.cuh"

namespace rvf {

__global__ void __launch_bounds__(256, 2) k_occ2d(const OccBatch* __restrict__ Lp) {
  extern __shared__ __align__(128) unsigned char smem[];
  SegTile& T = *reinterpret_cast<SegTile*>(smem);
  const OccBatch& B = *Lp;
  __shared__ int64_t s_tile;
  __shared__ int s_req, s_part, s_row, s_segs;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* S = reinterpret_cast<double*>(smem + sizeof(SegTile)) + warp * 8 * B.pmax_max;
  uint32_t n_pp = 0, n_rays = 0, n_traced = 0, n_defer = 0;
  TravCount tc;
  const int limit = B.total_tiles <= 64 ? kRowItems / 2 : kRowItems;
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
    const SegScene sc{t.nodes, t.nodesf, t.n_nodes, t.segs, t.frontier, t.n_frontier, t.cand_margin, t.delta};
    if (warp == 0) {
      const int n = tile_segments(sc, H, rmax, g_same, gi0, gj0, T);
      if (lane == 0) s_segs = n;
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
      // the row's (pair, segment) items, or n = -1 (its rays walk the tree)
      const double A[3] = {t.cen[3 * i], t.cen[3 * i + 1], 0.0};
      uint32_t rest;
      const int n = row_segments(sc, H, T, nseg, warp, A, cj, t.rad[i], rj, rj_max, valid, true, t.group[i], gj, rest,
                                 limit);
      const bool defer = n < 0 && rest != 0;  // warp-uniform
      if (defer) {
        if (lane == 0) {  // (zeroed before the launch: a store in every row cost 14% of the kernel)
          t.deferred[s_tile] = kClsSlow;
          t.tmask[s_tile * kTile + li] = rest;
        }
        ++n_defer;
        continue;
      }
      const bool some = (rest >> lane) & 1u;
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
      const int qmax = __reduce_max_sync(kFull, npj);
      double acc = 0.0;  // twice the pair's sum
      for (int q = 0; q < qmax; ++q) {
        const bool lq = q < npj;
        double xj[3] = {0.0, 0.0, 0.0}, nj[3] = {0.0, 0.0, 0.0};
        if (lq) {
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            xj[c] = jb[(c * pm + q) * kTile];
            nj[c] = jb[((3 + c) * pm + q) * kTile];
          }
        }
        double inner = 0.0;
        for (int p = 0; p < npi; ++p) {
          const double xi[3] = {S[8 * p], S[8 * p + 1], S[8 * p + 2]}, ni[3] = {S[8 * p + 4], S[8 * p + 5], S[8 * p + 6]};
          const double rx = xj[0] - xi[0], ry = xj[1] - xi[1], rz = xj[2] - xi[2];
          const double r2 = (rx * rx + ry * ry) + rz * rz;
          const double k = lq ? kernel_scaled<false>(rx, ry, rz, r2, ni, nj) : 0.0;
          const bool cast = k > 0.0;
          const uint32_t casts = __ballot_sync(kFull, cast);
          if (casts == 0) continue;  // warp-uniform
          n_rays += cast ? 1 : 0;
          n_traced += cast ? 1 : 0;
          // the segment as the reference passes it
          const double from[2] = {sw ? xj[0] : xi[0], sw ? xj[1] : xi[1]};
          const double to[2] = {sw ? xi[0] : xj[0], sw ? xi[1] : xj[1]};
          const bool blocked = (items_block(sc, T, warp, n, casts, from, to, tc.nodes, tc.prims) >> lane) & 1u;
          if (cast && !blocked) inner = fma(S[8 * p + 3], k, inner);
        }
        if (lq) acc = fma(jb[(6 * pm + q) * kTile], inner, acc);
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
  if (lane == 0 && n_defer) atomicAdd(B.q.ctr + kCtrWalk, (unsigned long long)n_defer);
  if (B.counters) {
    const uint32_t v[4] = {n_pp, n_rays, tc.nodes, tc.prims};
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
  const size_t smem = sizeof(SegTile) + stage_bytes(pmax);
  const cudaError_t e = cudaFuncSetAttribute(k_occ2d, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k_occ2d<<<(unsigned)(2 * sm_count), 256, smem, st>>>(b);
  return cudaGetLastError();
}

}  // namespace rvf
