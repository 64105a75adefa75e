// kernels_cull.cu -- tile classification before the pair pipeline.
//
// The reference casts a shadow ray for every point pair with K > 0
// (src/GPUKernels.jl:289-304) and walks the whole flat BVH for it
// (src/GPUBVH.jl:202-285).  Most of those rays cannot be blocked: with the
// reference's transposed triangle read (src/GPUBVH.jl:243-245) the triangles
// a ray actually tests are thin slivers, and a ray only reaches a triangle
// after passing the slab test of its (true-geometry) leaf box.  One warp per
// 32 x 32 tile of the upper triangle decides, with certified bounds, which
// pairs of the tile have a ray that can be blocked at all:
//
//  1. The tile's hull.  Every shadow ray of pair (i, j) lies within
//     R_ij = max(rad_i, rad_j) of the centroid segment [c_i, c_j] (convexity;
//     rad = largest distance of a quadrature point from the centroid), and
//     that segment lies in H = conv(B_I u B_J), B_I the box of the centroids
//     of the tile's row block.  So every ray of the tile lies within
//     R_t = max rad (+ the cull margin) of H.
//  2. The tile's list.  A breadth-first walk of the tree from the start
//     frontier drops every node whose box is farther than R_t from H (a
//     separating axis: the coordinate axes and the centroid direction crossed
//     with them) -- no ray of the tile can pass its slab test, so the
//     reference never tests its triangles -- and then every triangle farther
//     than R_t + M_T from H (16 axes: coordinate axes, the normal, and the
//     edges crossed with the centroid direction and the coordinate axes),
//     M_T being the bound on how far rounding moves a hit of the reference's
//     Moller-Trumbore test (the pair-list argument of kernels_wave.cu).
//     Triangles of the groups of both blocks (when each block has a single
//     group) are skipped, as the reference skips a ray's own groups
//     (src/GPUBVH.jl:239-240).  Both tests run in FP32 with the allowance
//     em = S 2^-16 of the pair lists.
//  3. The pair mask.  When the list is not empty, each pair keeps a bit iff
//     one listed triangle survives the pair-list kernel's own tests (its leaf
//     box against the pair's capsule, the group skip, the separating-axis
//     test against the capsule): the pair's rays may then be blocked and go
//     through the ray pipeline; every other pair's rays are certainly visible.
//
// Output per tile: a class byte (kClsSlow: some pair may be blocked, with
// its mask of 32 words, row li -> bit lj; kClsNear: some pair is near field
// for mixed precision; kClsTiny: some pair's points may nearly coincide).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "device_hull.cuh"
#include "device_lists.cuh"
#include "kernels.h"

namespace rvf {

namespace {

constexpr int kCullWarps = 4;
constexpr int kLongLeaves = 200;  // (about 1,024 triangles)

}  // namespace

// One warp per tile, grid-stride over the tiles of one request.
// resident blocks per SM the classification is compiled for
#ifndef RVF_CULL_MIN_BLOCKS
#define RVF_CULL_MIN_BLOCKS 1
#endif
// MASK: with step 3.  Without it (quadrature solves, whose occlusion kernel
// builds every pair's list itself, kernels_occ.cu) a tile is decided by its
// first surviving triangle.
template <bool MASK>
__global__ void __launch_bounds__(kCullWarps * 32, RVF_CULL_MIN_BLOCKS) k_tile_class(const TileClassArgs a) {
  __shared__ int s_front[kCullWarps][2 * kTileFront];
  __shared__ int s_leaf[kCullWarps][kTileLeaves];
  __shared__ int s_list[kCullWarps][MASK ? kTileTris : 1];
  __shared__ int s_rleaf[kCullWarps][MASK ? kTileLeaves : 1];  // runs of the list: leaf node
  __shared__ int s_rspan[kCullWarps][MASK ? kTileLeaves : 1];  //   first list entry * 16 + count
  __shared__ int s_row[kCullWarps][MASK ? kTileLeaves : 1];    // a row's runs
  __shared__ float s_cap[kCullWarps][32][12];  // a row's pairs: capsule start, end, direction, R, group
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int* front = s_front[warp];
  int* leaves = s_leaf[warp];
  int* list = s_list[warp];
  int* rleaf = s_rleaf[warp];
  int* rspan = s_rspan[warp];
  int* rowl = s_row[warp];
  const int64_t N = a.N;
  uint32_t n_culled = 0, n_masked = 0, n_over = 0;
  for (;;) {
    // tiles claimed one at a time: their costs differ by orders of magnitude
    unsigned long long tc = 0;
    if (lane == 0) tc = atomicAdd(a.claim, 1ull);
    tc = __shfl_sync(kFull, tc, 0);
    const int64_t t = MASK ? (int64_t)(tc / (unsigned)a.parts) : (int64_t)tc;
    if (t >= a.n_tiles) break;
    // with few tiles a claim is a part of a tile's mask rows (the first part also writes what is the tile's)
    const int part = MASK ? (int)(tc - (unsigned long long)t * (unsigned)a.parts) : 0;
    int64_t bi, bj;
    tile_coords(t, a.nT, bi, bj);
    const int64_t ei = bi * kTile + lane, ej = bj * kTile + lane;
    const bool oki = ei < N, okj = ej < N;
    double ci[3] = {0.0, 0.0, 0.0}, cj[3] = {0.0, 0.0, 0.0};
    double ri = 0.0, rj = 0.0, di = 0.0, dj = 0.0;
    int32_t gi = 0, gj = 0;
    if (oki) {
      ci[0] = a.cen[3 * ei]; ci[1] = a.cen[3 * ei + 1]; ci[2] = a.cen[3 * ei + 2];
      ri = a.rad ? a.rad[ei] : 0.0;
      di = a.diam[ei];
      gi = a.group[ei];
    }
    if (okj) {
      cj[0] = a.cen[3 * ej]; cj[1] = a.cen[3 * ej + 1]; cj[2] = a.cen[3 * ej + 2];
      rj = a.rad ? a.rad[ej] : 0.0;
      dj = a.diam[ej];
      gj = a.group[ej];
    }
    // near-field and nearly coincident pairs (lane = j, loop over the row block)
    bool near = false, tiny = false;
    bool classify_near = a.near_factor >= 0.0 || a.tiny_gap >= 0.0;  // mixed precision only
    HullF H;              // the tile's hull
    double rmax = 0.0, rj_max = 0.0;
    if (classify_near || (a.occ && a.dim3)) tile_hull(oki, okj, ci, cj, ri, rj, H, rmax, rj_max);
    if (classify_near) {
      // no pair of blocks whose centroid boxes lie farther apart than both
      // thresholds (2^-20 of the coordinates allows for the boxes' FP32 rounding)
      float dm = (float)fmax(di, dj), g2 = 0.0f;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) dm = fmaxf(dm, __shfl_xor_sync(kFull, dm, o));
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float s = H.h[0][c] + H.h[1][c];
        const float g = fabsf(H.d[c]) - s - 9.5367431640625e-07f * (fabsf(H.c[0][c]) + fabsf(H.c[1][c]) + s);
        if (g > 0.0f) g2 = fmaf(g, g, g2);
      }
      const float lim = 1.00001f * fmaxf(dm * (float)fmax(a.near_factor, 0.0), (float)(2.0 * rmax + fmax(a.tiny_gap, 0.0)));
      classify_near = !(g2 > lim * lim);
    }
    for (int li = 0; li < (classify_near ? kTile : 0); ++li) {
      const double x0 = __shfl_sync(kFull, ci[0], li), x1 = __shfl_sync(kFull, ci[1], li),
                   x2 = __shfl_sync(kFull, ci[2], li);
      const double rr = __shfl_sync(kFull, ri, li), dd = __shfl_sync(kFull, di, li);
      const int64_t i = bi * kTile + li;
      if (!(okj && i < N && i < ej)) continue;
      const double d0 = cj[0] - x0, d1 = cj[1] - x1, d2 = cj[2] - x2;
      const double q = d0 * d0 + d1 * d1 + d2 * d2;
      if (a.near_factor >= 0.0) {
        const double dm = fmax(dd, dj) * a.near_factor;
        near = near || q < dm * dm;
      }
      if (a.tiny_gap >= 0.0) {
        const double s = rr + rj + a.tiny_gap;
        tiny = tiny || q <= s * s;
      }
    }
    uint8_t cls = (__any_sync(kFull, near) ? kClsNear : 0) | (__any_sync(kFull, tiny) ? kClsTiny : 0);
    bool all_ones = false;  // occlusion the tile cannot classify: every pair keeps its rays
    int nl = 0;             // listed triangles
    int n_leaves = 0;       // leaves the hull reaches
    int nrun = 0;           // leaves with listed triangles (runs of the list)
    float rmaxJ = 0.0f;     // largest point radius of the column block
    if (a.occ && !a.dim3) {
      all_ones = true;
    } else if (a.occ) {
      rmaxJ = __double2float_ru(rj_max);
      // one group per block: its triangles are skipped by every ray of the tile
      const int32_t gi0 = __shfl_sync(kFull, gi, 0), gj0 = __shfl_sync(kFull, gj, 0);
      const bool g_same = a.skip_groups && __all_sync(kFull, (!oki || gi == gi0) && (!okj || gj == gj0));
      const float Rt = __double2float_ru(rmax + a.cull_margin);
      const float mbox = Rt + a.sat_em;
      // breadth-first walk from the start frontier
      int* cur = front;
      int* nxt = front + kTileFront;
      if (lane < a.n_frontier) cur[lane] = a.frontier[lane];
      __syncwarp();
      int ncur = a.n_frontier, nleaf = 0;
      bool over = false;
      while (ncur > 0 && !over) {  // one tree level per round
        int nnext = 0;
        for (int b = 0; b < ncur; b += 32) {
          const int q = b + lane;
          bool pass = false, leaf = false;
          int k = 0, right = 0;
          if (q < ncur && cur[q] < a.n_nodes) {
            k = cur[q];
            const NodeF nd = a.nodesf[k];
            pass = !hull_misses_box(H, nd, mbox);
            leaf = (nd.ab & 15) > 0;
            if (pass && !leaf) right = a.nodesf[k + 1].miss;
          }
          const uint32_t ml = __ballot_sync(kFull, pass && leaf), mi = __ballot_sync(kFull, pass && !leaf);
          const int pl = nleaf + __popc(ml & lanemask_lt());
          if (pass && leaf && pl < kTileLeaves) leaves[pl] = k;
          nleaf += __popc(ml);
          const int pi = nnext + 2 * __popc(mi & lanemask_lt());
          if (pass && !leaf && pi + 1 < kTileFront) {
            nxt[pi] = k + 1;
            nxt[pi + 1] = right;
          }
          nnext += 2 * __popc(mi);
        }
        __syncwarp();
        if (nleaf > kTileLeaves || nnext > kTileFront) over = true;
        int* tmp = cur;
        cur = nxt;
        nxt = tmp;
        ncur = nnext;
      }
      n_leaves = nleaf;
      // triangles of the candidate leaves, four leaves of up to 8 per round
      for (int b = 0; b < nleaf && !over; b += 4) {
        const int li = b + (lane >> 3), u8 = lane & 7;
        bool keep = false;
        int u = 0;
        if (li < nleaf) {
          const int32_t ab = a.nodesf[leaves[li]].ab;
          if (u8 < (ab & 15)) {
            u = (ab >> 4) + u8;
            const float4 p0 = a.sat[3 * u], p1 = a.sat[3 * u + 1], p2 = a.sat[3 * u + 2];
            const int32_t g = __float_as_int(p1.w);
            keep = !(g_same && (g == gi0 || g == gj0)) && !hull_misses_tri(H, p0, p1, p2, Rt + p0.w + a.sat_em);
          }
        }
        const uint32_t m = __ballot_sync(kFull, keep);
        if constexpr (!MASK) {
          nl = __popc(m);
          if (nl > 0) break;
          continue;
        }
        const int pos = nl + __popc(m & lanemask_lt());
        if (keep && pos < kTileTris) list[pos] = u;
        // one run per leaf of this round that kept triangles
        if (lane < 4 && b + lane < nleaf) {
          const uint32_t lm = (m >> (8 * lane)) & 0xffu;
          if (lm) {
            int before = 0;
            for (int k = 0; k < lane; ++k) before += ((m >> (8 * k)) & 0xffu) ? 1 : 0;
            const int r = nrun + before;
            rleaf[r] = leaves[b + lane];
            rspan[r] = (nl + __popc(m & ((1u << (8 * lane)) - 1u))) * 16 + __popc(lm);
          }
        }
        int nnew = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) nnew += ((m >> (8 * k)) & 0xffu) ? 1 : 0;
        nrun += nnew;
        nl += __popc(m);
        if (nl > kTileTris) over = true;
        __syncwarp();
      }
      __syncwarp();
      all_ones = over;
    }
    if constexpr (!MASK) {
      if (all_ones || nl > 0) cls |= kClsSlow | (all_ones ? kClsWide : 0) | (all_ones || n_leaves >= kLongLeaves ? kClsLong : 0);
      else if (a.occ) ++n_culled;
      n_over += all_ones && lane == 0 ? 1 : 0;
    } else if (all_ones) {
      cls |= kClsSlow;
      if (part == 0) {
        a.mask[t * kTile + lane] = 0xffffffffu;
        n_masked += 32;
        n_over += lane == 0 ? 1 : 0;
      }
    } else if (nl > 0) {
      // per pair: some listed triangle survives the pair-list tests.  Row by
      // row, the warp first keeps the runs (leaves with listed triangles)
      // whose box the row's own hull (its centroid and the column block's box,
      // radius max(rad_i, rad_J)) can reach, 32 at a time; each lane then
      // tests its pair against those leaves and their triangles.
      cls |= kClsSlow;
      const int rows = kTile / a.parts;
      for (int li = part * rows; li < (part + 1) * rows; ++li) {
        const int64_t i = bi * kTile + li;
        const double x0 = __shfl_sync(kFull, ci[0], li), x1 = __shfl_sync(kFull, ci[1], li),
                     x2 = __shfl_sync(kFull, ci[2], li);
        const double rr = __shfl_sync(kFull, ri, li);
        const int32_t g_i = __shfl_sync(kFull, gi, li);
        if (i >= N) {
          if (lane == 0) a.mask[t * kTile + li] = 0u;
          continue;
        }
        HullF Hr;
        const double xr[3] = {x0, x1, x2};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const float l = __double2float_rd(xr[c]), h = __double2float_ru(xr[c]);
          Hr.c[0][c] = 0.5f * (l + h);
          Hr.h[0][c] = 0.5f * (h - l);
          Hr.c[1][c] = H.c[1][c];
          Hr.h[1][c] = H.h[1][c];
          Hr.d[c] = Hr.c[1][c] - Hr.c[0][c];
        }
        const float Rr = fmaxf(__double2float_ru(rr), rmaxJ) + __double2float_ru(a.cull_margin) + a.sat_em;
        int nr = 0;
        for (int b = 0; b < nrun; b += 32) {
          const int r = b + lane;
          const bool keep = r < nrun && !hull_misses_box(Hr, a.nodesf[rleaf[r]], Rr);
          const uint32_t m = __ballot_sync(kFull, keep);
          if (keep) rowl[nr + __popc(m & lanemask_lt())] = r;
          nr += __popc(m);
        }
        __syncwarp();
        const bool valid = okj && i < ej;
        CapsuleF cap{};
        float bf[3] = {0.f, 0.f, 0.f}, df[3] = {0.f, 0.f, 0.f};
        float Rf = 0.0f;
        if (valid && nr > 0) {
          const double R = fmax(rr, rj) + a.cull_margin;
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const double dd = cj[c] - xr[c];
            cap.A[c] = (float)xr[c];
            bf[c] = (float)cj[c];
            cap.zero[c] = dd == 0.0;
            cap.inv[c] = cap.zero[c] ? 0.0f : (float)(1.0 / dd);
          }
          cap.R = (float)R + a.sat_em;
#pragma unroll
          for (int c = 0; c < 3; ++c) df[c] = bf[c] - cap.A[c];
          Rf = (float)R;
        }
        // Each pair's capsule against each run's leaf (lanes are pairs), then
        // the (pair, triangle) tests of each run dealt out to the lanes --
        // lane w of a round takes test w: pair w / count, triangle w % count
        // -- so the lanes stay busy however few pairs reach a leaf.  A pair
        // leaves once one of its triangles survives.
        float* cd = s_cap[warp][lane];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          cd[c] = cap.A[c];
          cd[3 + c] = bf[c];
          cd[6 + c] = df[c];
        }
        cd[9] = Rf;
        cd[10] = __int_as_float(gj);
        const uint32_t none = __ballot_sync(kFull, !valid);
        // the pairs reaching each run's leaf, in the walk's leaf array (not
        // needed once the runs are recorded)
        uint32_t* pms = reinterpret_cast<uint32_t*>(leaves);
        for (int e = 0; e < nr; ++e) {
          const bool pass = valid && !capsule_misses_box(cap, a.nodesf[rleaf[rowl[e]]]);
          const uint32_t pm = __ballot_sync(kFull, pass);
          if (lane == 0) pms[e] = pm;
        }
        __syncwarp();
        uint32_t hit = 0;
        for (int e = 0; e < nr; ++e) {
          const uint32_t pm = pms[e] & ~hit & ~none;
          if (pm == 0) continue;  // warp-uniform
          const int span = rspan[rowl[e]], k0 = span >> 4, cnt = span & 15;
          const int total = __popc(pm) * cnt;
          uint32_t h = 0;
          for (int w = lane; w < total; w += 32) {
            const int pi = w / cnt, ti = w - pi * cnt;
            const int p = nth_set_bit(pm, pi);
            const float* q = s_cap[warp][p];
            const int u = list[k0 + ti];
            const float4 p0 = a.sat[3 * u], p1 = a.sat[3 * u + 1], p2 = a.sat[3 * u + 2];
            const int32_t g = __float_as_int(p1.w);
            if (a.skip_groups && (g == g_i || g == __float_as_int(q[10]))) continue;
            const float qa[3] = {q[0], q[1], q[2]}, qd[3] = {q[6], q[7], q[8]};
            if (!pair_misses_tri(qa, qd, q[9], a.sat_em, p0, p1, p2)) h |= 1u << p;
          }
          hit |= __reduce_or_sync(kFull, h);
        }
        const bool bit = (hit >> lane) & 1u;
        __syncwarp();
        const uint32_t m = __ballot_sync(kFull, bit);
        if (lane == 0) {
          a.mask[t * kTile + li] = m;
          n_masked += __popc(m);
        }
      }
    } else if (a.occ) {
      n_culled += part == 0 ? 1 : 0;
    }
    if (lane == 0 && part == 0) a.cls[t] = cls;
  }
  if (a.counters) {
    const uint64_t s_c = warp_sum_u64(lane == 0 ? n_culled : 0), s_m = warp_sum_u64(n_masked),
                   s_o = warp_sum_u64(n_over);
    if (lane == 0) {
      atomicAdd(a.counters + 0, s_c);
      atomicAdd(a.counters + 1, s_m);
      atomicAdd(a.counters + 2, s_o);
    }
  }
}

cudaError_t launch_tile_class(const TileClassArgs& args, int sm_count, cudaStream_t st) {
  if (args.n_tiles <= 0) return cudaSuccess;
  TileClassArgs a = args;
  a.parts = 1;
  auto launch = [&](auto fn) -> cudaError_t {
    int per_sm = 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kCullWarps * 32, 0) != cudaSuccess || per_sm < 1)
      per_sm = 1;
    const int64_t resident = (int64_t)sm_count * per_sm;
    // masks: four claims a warp, so that the heaviest tiles do not end alone (2,346 tiles of
    // Monte Carlo masks around a box: 2.9 ms with whole tiles, 1.6 ms with parts of them)
    while (a.mask && a.parts < 8 && a.n_tiles * a.parts < 4 * kCullWarps * resident) a.parts *= 2;
    const int64_t want = (a.n_tiles * a.parts + kCullWarps - 1) / kCullWarps;
    const int grid = (int)std::min<int64_t>(want, resident);
    const cudaError_t e = cudaMemsetAsync(a.claim, 0, sizeof(unsigned long long), st);
    if (e != cudaSuccess) return e;
    fn<<<(unsigned)grid, kCullWarps * 32, 0, st>>>(a);
    return cudaGetLastError();
  };
  return a.mask ? launch(k_tile_class<true>) : launch(k_tile_class<false>);
}

}  // namespace rvf
