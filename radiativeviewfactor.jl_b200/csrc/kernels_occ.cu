// kernels_occ.cu -- the tiles of a surface mesh whose shadow rays may be
// blocked: pair lists, quadrature, shadow rays and F without ray queues.
//
// Replaces _vf_pair_kernel! (src/GPUKernels.jl:226-323) with its shadow rays
// (gpu_intersect_bvh, src/GPUBVH.jl:202-285) for the tiles that the tile
// classification (kernels_cull.cu) could not clear.  Three kernels per chunk:
//  1. k_occ_list, a block per tile: walks the tree with the tile's hull, keeps
//     the triangles any ray of the tile can hit as runs of one leaf each
//     (shared memory), and builds every pair's list row by row, a warp per
//     row: the leaves the pair's capsule reaches and, of each, the triangles
//     the capsule test keeps, as (leaf, mask of its 8 triangles) entries.
//     Pairs with a list are queued, the tile's mask rows name them.
//  2. k_occ_rest: the tiles' other pairs, whose rays are all visible, with the
//     quadrature-only loop.
//  3. k_occ_pairs, a warp per queued pair: a lane holds two of its rays and
//     the warp walks the pair's list, so every lane tests the same box or
//     triangle (one broadcast load, no divergence in list lengths); the
//     visible terms are summed in a fixed order and F is written.
// The lists hold every triangle a ray of the pair can hit (device_lists.cuh),
// and a ray that passes a listed leaf's box passes every ancestor's, so the
// decisions are the reference's.  Rays are tested in FP32 with certified
// decisions (device_mixed.cuh) in both precisions; a ray with an uncertain one
// is tested again in FP64 with the reference's arithmetic, and a ray without a
// usable list, or with an infinite 1/d, walks the tree.
//
// Measured on a B200, closed cube of 43,200 Tri3 with a box of 1,728 triangles,
// 7 points (FP64 / mixed precision, one solve): lists 43 / 43 ms, rest 13 / 16
// ms, pairs 89 / 105 ms, 144 / 164 ms together, bound by instruction issue
// (65-75% of the slots).  Of the pairs' time about 24 / 30 ms set the rays up,
// 58 ms test lists, the rest tests uncertain rays again.  The queue pipeline
// (kernels_wave.cu), which also needs the classification's pair masks (36 ms), took
// 310 / 224 ms for the same tiles: a record per ray and a slot and list per pair
// through global memory, read back with dependent loads at 12 to 15 of 32 active
// lanes.  Where lists do not hold a tile (fine obstructions) or FP32 is too coarse that
// pipeline is the faster one and takes the solve (wave_host.cpp: occ_by_queue,
// fp32_too_coarse).
// Measured and not kept: the uncertain rays of a pass tested in FP64 a lane each
// instead of one after another (axis-aligned meshes, 9 points, mixed: 16.5 -> 14.3 ms;
// the closed cube 216.3 -> 223.2 ms: registers of the kernel around it); all three steps in one kernel, lane = (pair, q) (284 /
// 311 ms: 16 warps per SM cannot hide the list building's latency, four pairs'
// lists differ in length); the (ray, triangle) tests packed into full warps
// through shared memory (144 / 190 ms of pair kernel); the passing rays of a
// leaf packed into the first lanes (111 / 158 ms); a leaf's triangles before its box
// (131 / 150 ms against 95 / 112 then: the box stops most warps); the next entry's
// box or triangle loaded ahead (within 1%, up to 3% slower); a second culling of
// the lists by the points' extent across the pair's direction (18% fewer list pairs,
// lists +8 / +15 ms, pairs -14 / -8 ms; mixed precision must keep the sums of the
// capsule's lists); a lane per pair in the list tests where many pairs reach a leaf
// (within 1%).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "device_hull.cuh"
#include "device_pairs.cuh"

namespace rvf {

namespace {

constexpr int kOccTris = 2048;   // triangles of a tile's list (more: the pairs' own walks)
constexpr int kOccRuns = 256;    // its leaves
constexpr int kOccList = 32;     // leaves of a pair's list (more: the pair's own walk)
constexpr int kOccOwn = 64;      // leaves of a list from the pair's own walk (more: its rays walk the tree)
constexpr int kOccFront = 64;    // breadth-first frontier of a pair's own walk
static_assert(kOccRuns <= kTileLeaves && kOccRuns <= 256, "a list entry keeps the run in 8 bits");
static_assert(kOccOwn <= 64, "k_occ_pairs holds a list in two registers a lane");

struct OccWarp {
  uint16_t list[kOccList][32];             // [entry][pair of the row]: run << 8 | mask of its listed triangles
  float cap[32][9];                        // the row's pairs: capsule start, direction, R, group (odd stride)
  uint8_t order[32];                       // the pairs reaching the current run
  union {
    uint32_t reach[kOccRuns];              // the pairs whose capsule reaches each of the row's runs
    struct {
      int front[2 * kOccFront];
      int leaves[kOccOwn];
      uint32_t own[kOccOwn];
    } walk;                                // a pair's own walk
  };
  uint8_t runs[kOccRuns];                  // the row's runs
};

struct OccTile {
  NodeF box[kOccRuns];       // the runs' leaves
  int span[kOccRuns];        // first list entry << 4 | count
  int leaf[kOccRuns];        // leaf node
  uint8_t bits[kOccRuns];    // the leaf's listed triangles
  int list[kOccTris];        // triangles in leaf order
  int leaves[kTileLeaves];   // the walk's leaves
  uint32_t kept[kTileLeaves / 4];            // four leaves' kept triangles, 8 bits each
  int tri_at[kTileLeaves / 4], run_at[kTileLeaves / 4];
  OccWarp warp[8];
};

// The list of one pair by its own walk of the tree (as build_pair_list in
// kernels_wave.cu): leaves and triangle masks into `own`; the number of
// entries, or -1 when a capacity is exceeded.  Warp-uniform.
__device__ __noinline__ int occ_own_list(const OccArgs& t, int64_t i, int64_t j, int* front, int* leaves,
                                         uint32_t* own) {
  const int lane = threadIdx.x & 31;
  CapsuleF cap;
  float bf[3], df[3];
  const double R = fmax(t.rad[i], t.rad[j]) + t.cull_margin;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double A = t.cen[3 * i + c], B = t.cen[3 * j + c];
    const double dd = B - A;
    cap.A[c] = (float)A;
    bf[c] = (float)B;
    cap.zero[c] = dd == 0.0;
    cap.inv[c] = cap.zero[c] ? 0.0f : (float)(1.0 / dd);
    df[c] = bf[c] - cap.A[c];
  }
  cap.R = (float)R + t.sat_em;
  const float Rf = (float)R;
  int* cur = front;
  int* nxt = front + kOccFront;
  if (lane < t.n_frontier) cur[lane] = t.frontier[lane];
  __syncwarp();
  int ncur = t.n_frontier, nleaf = 0;
  while (ncur > 0) {  // one tree level per round
    int nnext = 0;
    for (int b = 0; b < ncur; b += 32) {
      const int q = b + lane;
      bool pass = false, leaf = false;
      int k = 0, right = 0;
      if (q < ncur && cur[q] < t.n_nodes) {
        k = cur[q];
        const NodeF nd = t.nodesf[k];
        pass = !capsule_misses_box(cap, nd);
        leaf = (nd.ab & 15) > 0;
        if (pass && !leaf) right = t.nodesf[k + 1].miss;
      }
      const uint32_t ml = __ballot_sync(kFull, pass && leaf), mi = __ballot_sync(kFull, pass && !leaf);
      const int pl = nleaf + __popc(ml & lanemask_lt());
      if (pass && leaf && pl < kOccOwn) leaves[pl] = k;
      nleaf += __popc(ml);
      const int pi = nnext + 2 * __popc(mi & lanemask_lt());
      if (pass && !leaf && pi + 1 < kOccFront) {
        nxt[pi] = k + 1;
        nxt[pi + 1] = right;
      }
      nnext += 2 * __popc(mi);
    }
    __syncwarp();
    if (nleaf > kOccOwn || nnext > kOccFront) return -1;
    int* tmp = cur;
    cur = nxt;
    nxt = tmp;
    ncur = nnext;
  }
  const int32_t gi = t.group[i], gj = t.group[j];
  int n = 0;
  for (int b = 0; b < nleaf; b += 4) {
    const int li = b + (lane >> 3), u8 = lane & 7;
    bool keep = false;
    if (li < nleaf) {
      const int32_t ab = t.nodesf[leaves[li]].ab;
      if (u8 < (ab & 15)) {
        const int u = (ab >> 4) + u8;
        const float4 p0 = t.sat[3 * u], p1 = t.sat[3 * u + 1], p2 = t.sat[3 * u + 2];
        const int32_t g = __float_as_int(p1.w);
        keep = g != gi && g != gj && !pair_misses_tri(cap.A, df, Rf, t.sat_em, p0, p1, p2);
      }
    }
    const uint32_t m = __ballot_sync(kFull, keep);
    const uint32_t mine = lane < 4 && b + lane < nleaf ? (m >> (8 * lane)) & 255u : 0u;
    const uint32_t some = __ballot_sync(kFull, mine != 0);
    if (mine) own[n + __popc(some & lanemask_lt())] = ((uint32_t)leaves[b + lane] << 8) | mine;
    n += __popc(some);
  }
  __syncwarp();
  return n;
}

// Step 3 of a mixed-precision row with near-field, nearly coincident or
// blockable pairs: the visible pairs (lanes outside `skip`) with the mixed
// generation's arithmetic -- FP64 for near-field pairs and grazing point
// pairs, FP32 otherwise.
__device__ __noinline__ void row_visible_mixed(const MixedArgs& a, int64_t bi, int64_t bj, int li, uint32_t skip,
                                               bool near, uint32_t* cnt) {
  const int lane = threadIdx.x & 31;
  const int64_t N = a.N, i = bi * kTile + li, j = bj * kTile + lane;
  const int pm = a.pmax;
  const bool valid = j < N && i < j && !((skip >> lane) & 1u);
  const int64_t oi = a.orig ? (int64_t)a.orig[i] : i, oj = j < N ? (a.orig ? (int64_t)a.orig[j] : j) : 0;
  const int npi = a.np[i];
  int npj = valid ? a.np[j] : 0;
  if (valid && a.flat[i] && a.flat[j] && a.nrm[3 * i] == a.nrm[3 * j] && a.nrm[3 * i + 1] == a.nrm[3 * j + 1] &&
      a.nrm[3 * i + 2] == a.nrm[3 * j + 2])
    npj = 0;
  const int qmax = __reduce_max_sync(kFull, npj);
  near = near && valid;
  cnt[3] += near && npj > 0 ? 1 : 0;
  const double ci0 = a.cen[3 * i], ci1 = a.cen[3 * i + 1], ci2 = a.cen[3 * i + 2];
  const float d0 = valid ? (float)(a.cen[3 * j] - ci0) : 0.f, d1 = valid ? (float)(a.cen[3 * j + 1] - ci1) : 0.f,
              d2 = valid ? (float)(a.cen[3 * j + 2] - ci2) : 0.f;
  const float* itf = a.tabf + bi * kComp * pm * kTile + li;
  const float* jtf = a.tabf + bj * kComp * pm * kTile + lane;
  const double* it = a.tab + bi * kComp * pm * kTile + li;
  const double* jt = a.tab + bj * kComp * pm * kTile + lane;
  double accd = 0.0;
  float acc32 = 0.0f;
  for (int q = 0; q < qmax; ++q) {
    const bool lq = q < npj, far = lq && !near;
    float oq0 = 0.f, oq1 = 0.f, oq2 = 0.f, nq0 = 0.f, nq1 = 0.f, nq2 = 0.f, wq = 0.f;
    if (far) {
      oq0 = jtf[(0 * pm + q) * kTile]; oq1 = jtf[(1 * pm + q) * kTile]; oq2 = jtf[(2 * pm + q) * kTile];
      nq0 = jtf[(3 * pm + q) * kTile]; nq1 = jtf[(4 * pm + q) * kTile]; nq2 = jtf[(5 * pm + q) * kTile];
      wq = jtf[(6 * pm + q) * kTile];
    }
    float inner = 0.0f;
    for (int p = 0; p < npi; ++p) {
      const float op0 = itf[(0 * pm + p) * kTile], op1 = itf[(1 * pm + p) * kTile], op2 = itf[(2 * pm + p) * kTile];
      const float np0 = itf[(3 * pm + p) * kTile], np1 = itf[(4 * pm + p) * kTile], np2 = itf[(5 * pm + p) * kTile];
      const float wp = itf[(6 * pm + p) * kTile];
      const float rx = d0 + (oq0 - op0), ry = d1 + (oq1 - op1), rz = d2 + (oq2 - op2);
      const float r2 = fmaf(rx, rx, fmaf(ry, ry, rz * rz));
      const float di = fmaf(np0, rx, fmaf(np1, ry, np2 * rz));
      const float dj = -fmaf(nq0, rx, fmaf(nq1, ry, nq2 * rz));
      const bool graze = far && (r2 < 1e-18f || di * di <= 1e-10f * r2 || dj * dj <= 1e-10f * r2);
      float K32 = 0.0f;
      if (far && !graze && di > 0.0f && dj > 0.0f) K32 = (di * dj) * rcp_approx(3.14159265f * (r2 * r2));
      cnt[1] += K32 > 0.0f ? 1 : 0;
      if (far && !graze) inner = fmaf(wp, K32, inner);
      if (lq && (near || graze)) {
        double xi[3], ni[3], xj[3], nj[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          xi[k] = it[(k * pm + p) * kTile];
          ni[k] = it[((3 + k) * pm + p) * kTile];
          xj[k] = jt[(k * pm + q) * kTile];
          nj[k] = jt[((3 + k) * pm + q) * kTile];
        }
        const double rx64 = xj[0] - xi[0], ry64 = xj[1] - xi[1], rz64 = xj[2] - xi[2];
        const double r264 = (rx64 * rx64 + ry64 * ry64) + rz64 * rz64;
        const double K64 = k_fast<true>(rx64, ry64, rz64, r264, ni, nj);
        accd += jt[(6 * pm + q) * kTile] * (it[(6 * pm + p) * kTile] * K64);
        const bool cast = K64 > 0.0 && sqrt(r264) > 1e-15;
        cnt[1] += cast ? 1 : 0;
        cnt[2] += cast ? 1 : 0;
        cnt[4] += graze ? 1 : 0;
      }
    }
    acc32 = fmaf(wq, inner, acc32);
  }
  cnt[0] += npi * npj;
  const double raw = accd + (double)acc32;
  if (valid) {
    a.F[oi + oj * N] = raw / a.area[i];
    a.F[oj + oi * N] = raw / a.area[j];
  } else if (j == i) {
    a.F[oi + oi * N] = 0.0 / a.area[i];
  }
}

// A tile's triangle list by the block, in the walk order of the tile
// classification.  `capped`: the classification's capacities are
// exceeded (every pair counts as blockable); returns false when the list does
// not fit here either.
__device__ bool occ_tile_list(const OccArgs& t, const HullF& H, float Rt, bool g_same, int32_t gi0, int32_t gj0,
                              OccTile& T, int* s_n, bool& capped) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // the walk's frontiers, in the warps' list space (not in use yet)
  int* front = reinterpret_cast<int*>(&T.warp[0]);
  static_assert(sizeof(OccWarp) >= 2 * kTileFront * sizeof(int), "frontiers fit a warp's space");
  if (warp == 0) {
    int* cur = front;
    int* nxt = front + kTileFront;
    if (lane < t.n_frontier) cur[lane] = t.frontier[lane];
    __syncwarp();
    int ncur = t.n_frontier, nleaf = 0;
    bool over = false;
    while (ncur > 0 && !over) {  // one tree level per round
      int nnext = 0;
      for (int b = 0; b < ncur; b += 32) {
        const int q = b + lane;
        bool pass = false, leaf = false;
        int k = 0, right = 0;
        if (q < ncur && cur[q] < t.n_nodes) {
          k = cur[q];
          const NodeF nd = t.nodesf[k];
          pass = !hull_misses_box(H, nd, Rt + t.sat_em);
          leaf = (nd.ab & 15) > 0;
          if (pass && !leaf) right = t.nodesf[k + 1].miss;
        }
        const uint32_t ml = __ballot_sync(kFull, pass && leaf), mi = __ballot_sync(kFull, pass && !leaf);
        const int pl = nleaf + __popc(ml & lanemask_lt());
        if (pass && leaf && pl < kTileLeaves) T.leaves[pl] = k;
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
    if (lane == 0) s_n[0] = over ? -1 : nleaf;
  }
  __syncthreads();
  const int nleaf = s_n[0];
  capped = nleaf < 0;
  if (capped) return false;
  const int quads = (nleaf + 3) / 4;
  for (int qd = warp; qd < quads; qd += 8) {
    const int li = 4 * qd + (lane >> 3), u8 = lane & 7;
    bool keep = false;
    if (li < nleaf) {
      const int32_t ab = t.nodesf[T.leaves[li]].ab;
      if (u8 < (ab & 15)) {
        const int u = (ab >> 4) + u8;
        const float4 p0 = t.sat[3 * u], p1 = t.sat[3 * u + 1], p2 = t.sat[3 * u + 2];
        const int32_t g = __float_as_int(p1.w);
        keep = !(g_same && (g == gi0 || g == gj0)) && !hull_misses_tri(H, p0, p1, p2, Rt + p0.w + t.sat_em);
      }
    }
    const uint32_t m = __ballot_sync(kFull, keep);
    if (lane == 0) T.kept[qd] = m;
  }
  __syncthreads();
  if (warp == 0) {  // where each four leaves' triangles and runs go
    int nt = 0, nr = 0;
    for (int b = 0; b < quads; b += 32) {
      const uint32_t m = b + lane < quads ? T.kept[b + lane] : 0u;
      const int mt = __popc(m);
      const int mr = ((m & 0xffu) ? 1 : 0) + ((m & 0xff00u) ? 1 : 0) + ((m & 0xff0000u) ? 1 : 0) + ((m >> 24) ? 1 : 0);
      int it = mt, ir = mr;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int vt = __shfl_up_sync(kFull, it, o), vr = __shfl_up_sync(kFull, ir, o);
        if (lane >= o) {
          it += vt;
          ir += vr;
        }
      }
      if (b + lane < quads) {
        T.tri_at[b + lane] = nt + it - mt;
        T.run_at[b + lane] = nr + ir - mr;
      }
      nt += __shfl_sync(kFull, it, 31);
      nr += __shfl_sync(kFull, ir, 31);
    }
    if (lane == 0) {
      s_n[1] = nt;
      s_n[2] = nr;
    }
  }
  __syncthreads();
  capped = s_n[1] > kTileTris;
  if (s_n[1] > kOccTris) return false;
  for (int qd = warp; qd < quads; qd += 8) {
    const uint32_t m = T.kept[qd];
    const int li = 4 * qd + (lane >> 3), u8 = lane & 7;
    if ((m >> lane) & 1u) {
      const int32_t ab = t.nodesf[T.leaves[li]].ab;
      T.list[T.tri_at[qd] + __popc(m & lanemask_lt())] = (ab >> 4) + u8;
    }
    if (lane < 4) {
      const uint32_t lm = (m >> (8 * lane)) & 0xffu;
      if (lm) {
        int before = 0;
        for (int k = 0; k < lane; ++k) before += ((m >> (8 * k)) & 0xffu) ? 1 : 0;
        const int r = T.run_at[qd] + before;
        const int leaf = T.leaves[4 * qd + lane];
        T.leaf[r] = leaf;
        T.box[r] = t.nodesf[leaf];
        T.span[r] = ((T.tri_at[qd] + __popc(m & ((1u << (8 * lane)) - 1u))) << 4) | __popc(lm);
        T.bits[r] = (uint8_t)lm;
      }
    }
  }
  return true;
}

}  // namespace

// 1. Pair lists of the launch's tiles.  Bound by the capsule tests' FP32 issue
// and the latency of their gathers.
__global__ void __launch_bounds__(256, 3) k_occ_list(const OccBatch* __restrict__ Lp) {
  extern __shared__ __align__(128) unsigned char smem[];
  OccTile& T = *reinterpret_cast<OccTile*>(smem);
  const OccBatch& B = *Lp;
  const OccQ& Q = B.q;
  __shared__ int64_t s_tile;
  __shared__ int s_req, s_part, s_row;
  __shared__ int s_n[3];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  OccWarp& W = T.warp[warp];
  uint32_t n_masked = 0, n_list = 0, n_walk = 0;
  for (;;) {
    if (threadIdx.x == 0) {
      s_tile = -1;
      // a tile needs at most 1,024 queue slots; the launch's blocks may each hold one more tile
      const unsigned long long used = *(volatile unsigned long long*)(Q.ctr + kCtrSlots) +
                                      *(volatile unsigned long long*)(Q.ctr + kCtrWalk),
                               pool = *(volatile unsigned long long*)(Q.ctr + kCtrPool),
                               next = *(volatile unsigned long long*)(Q.ctr + kCtrTile);
      // a full pool ends the chunk between tiles, not between a tile's parts (the next chunk would do the first
      // ones again): a block that claimed a part comes back for the rest; pairs that find the pool full walk
      if (used + (unsigned long long)gridDim.x * kTile * kTile <= (unsigned long long)Q.scap &&
          (pool <= (unsigned long long)Q.pool_cap || next % (unsigned)B.groups != 0)) {
        const unsigned long long k = atomicAdd(Q.ctr + kCtrTile, 1ull);
        const int64_t g = (int64_t)(k / (unsigned)B.groups);
        if (g < B.total_tiles) {
          s_req = find_req(B.tile_base, B.n_req, g);
          s_part = (int)(k - (unsigned long long)g * (unsigned)B.groups);
          s_tile = g - B.tile_base[s_req];
          s_row = s_part * (kTile / B.groups);
        }
      }
    }
    __syncthreads();
    if (s_tile < 0) break;
    const OccArgs& t = B.reqs[s_req];
    const int64_t tile = t.work[s_tile + t.tile0];
    const int row1 = (s_part + 1) * (kTile / B.groups);
    const int64_t N = t.N;
    int64_t bi, bj;
    tile_coords(tile, t.nT, bi, bj);
    const uint8_t cls = t.tcls[tile];
    const int64_t ei = bi * kTile + lane, j = bj * kTile + lane;
    const bool oki = ei < N, okj = j < N;
    double cj[3] = {0.0, 0.0, 0.0};
    double rj = 0.0;
    int32_t gj = 0;
    if (okj) {
      cj[0] = t.cen[3 * j]; cj[1] = t.cen[3 * j + 1]; cj[2] = t.cen[3 * j + 2];
      rj = t.rad[j];
      gj = t.group[j];
    }
    int nrun = 0;
    bool capped = false, listed = true;
    HullF H;
    float rmaxJ = 0.0f;
    if (cls & kClsSlow) {
      double cc[3] = {0.0, 0.0, 0.0};
      double ri = 0.0;
      int32_t gi = 0;
      if (oki) {
        cc[0] = t.cen[3 * ei]; cc[1] = t.cen[3 * ei + 1]; cc[2] = t.cen[3 * ei + 2];
        ri = t.rad[ei];
        gi = t.group[ei];
      }
      double rmax, rj_max;
      tile_hull(oki, okj, cc, cj, ri, rj, H, rmax, rj_max);
      rmaxJ = __double2float_ru(rj_max);
      const int32_t gi0 = __shfl_sync(kFull, gi, 0), gj0 = __shfl_sync(kFull, gj, 0);
      const bool g_same = __all_sync(kFull, (!oki || gi == gi0) && (!okj || gj == gj0));
      const float Rt = __double2float_ru(rmax + t.cull_margin);
      listed = occ_tile_list(t, H, Rt, g_same, gi0, gj0, T, s_n, capped);
      if (!listed) capped = true;
      else nrun = s_n[2];
    }
    __syncthreads();
    for (;;) {  // rows, as the warps get to them
      int li = 0;
      if (lane == 0) li = atomicAdd(&s_row, 1);
      li = __shfl_sync(kFull, li, 0);
      if (li >= row1) break;
      const int64_t i = bi * kTile + li;
      if (i >= N) break;
      const bool valid = okj && i < j;
      int n = 0;  // the lane's pair: list entries, -1: to be built by its own walk, -2: none
      if (nrun > 0) {
        const double xr[3] = {t.cen[3 * i], t.cen[3 * i + 1], t.cen[3 * i + 2]};
        const double rr = t.rad[i];
        const int32_t g_i = t.group[i];
        // the row's runs: leaves its own hull reaches (its centroid and the column block's box)
        HullF Hr;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const float l = __double2float_rd(xr[k]), h = __double2float_ru(xr[k]);
          Hr.c[0][k] = 0.5f * (l + h);
          Hr.h[0][k] = 0.5f * (h - l);
          Hr.c[1][k] = H.c[1][k];
          Hr.h[1][k] = H.h[1][k];
          Hr.d[k] = Hr.c[1][k] - Hr.c[0][k];
        }
        const float Rr = fmaxf(__double2float_ru(rr), rmaxJ) + __double2float_ru(t.cull_margin) + t.sat_em;
        int nr = 0;
        for (int b = 0; b < nrun; b += 32) {
          const int r = b + lane;
          const bool keep = r < nrun && !hull_misses_box(Hr, T.box[r], Rr);
          const uint32_t m = __ballot_sync(kFull, keep);
          if (keep) W.runs[nr + __popc(m & lanemask_lt())] = (uint8_t)r;
          nr += __popc(m);
        }
        __syncwarp();
        if (nr > 0) {
          CapsuleF cap{};
          float* cd = W.cap[lane];
          const double R = fmax(rr, rj) + t.cull_margin;
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            const double dd = cj[k] - xr[k];
            const float A = (float)xr[k], bf = (float)cj[k];
            cap.A[k] = A;
            cap.zero[k] = dd == 0.0;
            cap.inv[k] = cap.zero[k] ? 0.0f : (float)(1.0 / dd);
            cd[k] = A;
            cd[3 + k] = bf - A;
          }
          cap.R = (float)R + t.sat_em;
          cd[6] = (float)R;
          cd[7] = __int_as_float(gj);
          for (int e = 0; e < nr; ++e) {
            const bool pass = valid && !capsule_misses_box(cap, T.box[W.runs[e]]);
            const uint32_t pm = __ballot_sync(kFull, pass);
            if (lane == 0) W.reach[e] = pm;
          }
          __syncwarp();
          for (int e = 0; e < nr; ++e) {
            const uint32_t pm = W.reach[e];
            if (pm == 0) continue;  // warp-uniform
            const int r = W.runs[e];
            const int span = T.span[r], k0 = span >> 4, ct = span & 15;
            const int total = __popc(pm) * ct;
            // test w: pair w / ct of those reaching the leaf, triangle w % ct;
            // the bits of one pair are consecutive over the rounds' ballots
            const bool in = (pm >> lane) & 1u;
            const int rank = __popc(pm & lanemask_lt()), first = rank * ct;
            if (in) W.order[rank] = (uint8_t)lane;
            __syncwarp();
            const float per = 1.0f / (float)ct;  // w + 1/2 is at least 1/16 from a multiple of ct: exact below 256
            uint32_t mine = 0;
            for (int b = 0; b < total; b += 32) {
              const int w = b + lane;
              bool keep = false;
              if (w < total) {
                const int pi = (int)(((float)w + 0.5f) * per), ti = w - pi * ct;
                const float* q = W.cap[W.order[pi]];
                const int u = T.list[k0 + ti];
                const float4 p0 = t.sat[3 * u], p1 = t.sat[3 * u + 1], p2 = t.sat[3 * u + 2];
                const int32_t g = __float_as_int(p1.w);
                if (g != g_i && g != __float_as_int(q[7])) {
                  const float qa[3] = {q[0], q[1], q[2]}, qd[3] = {q[3], q[4], q[5]};
                  keep = !pair_misses_tri(qa, qd, q[6], t.sat_em, p0, p1, p2);
                }
              }
              const uint32_t m = __ballot_sync(kFull, keep);
              const int s = first - b;  // where the lane's bits begin in this round
              if (in && s > -8 && s < 32) mine |= s >= 0 ? m >> s : m << -s;
            }
            __syncwarp();  // before the next run's order
            mine &= (1u << ct) - 1u;
            if (in && mine && n >= 0) {
              if (n < kOccList) W.list[n][lane] = (uint16_t)((r << 8) | mine);
              n = n < kOccList ? n + 1 : -1;
            }
          }
          __syncwarp();
        }
      }
      if (!listed) n = valid ? -1 : 0;
      const uint32_t masked = __ballot_sync(kFull, valid && (capped || n != 0));
      n_masked += lane == 0 ? __popc(masked) : 0;
      // queued: the pairs with a list; in mixed precision every pair of a
      // tile beyond the classification's capacities (the terms of its rays
      // through the root box are added in FP64)
      const uint32_t queued = t.mixed ? masked : __ballot_sync(kFull, n != 0);
      if (lane == 0) t.tmask[tile * kTile + li] = queued;
      if (queued == 0) continue;
      const bool mine = (queued >> lane) & 1u;
      unsigned long long off = 0;
      if (!t.lists && mine) n = -2;  // pair lists switched off: the rays walk the tree
      const int want = mine && n > 0 ? n : 0;
      int incl = want;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += v;
      }
      const int total = __shfl_sync(kFull, incl, 31);
      if (total > 0) {
        if (lane == 0) off = atomicAdd(Q.ctr + kCtrPool, (unsigned long long)total);
        off = __shfl_sync(kFull, off, 0) + (incl - want);
        if (want && (int64_t)off + want > Q.pool_cap) n = -2;  // pool full: this pair walks
        else
          for (int k = 0; k < want; ++k) {
            const uint32_t v = W.list[k][lane];
            const int r = (int)(v >> 8);
            // the run's listed triangles back to the leaf's eight
            uint32_t kept = T.bits[r], m = 0;
            for (uint32_t b = v & 255u; kept; b >>= 1) {
              const uint32_t low = kept & (0u - kept);
              if (b & 1u) m |= low;
              kept ^= low;
            }
            Q.pool[off + k] = ((uint32_t)T.leaf[r] << 8) | m;
          }
      }
      // lists that did not fit, by the pairs' own walks
      for (uint32_t own = __ballot_sync(kFull, mine && n == -1); own; own &= own - 1u) {
        const int pl = __ffs(own) - 1;
        int no = occ_own_list(t, i, bj * kTile + pl, W.walk.front, W.walk.leaves, W.walk.own);
        unsigned long long oo = 0;
        if (no > 0) {
          if (lane == 0) oo = atomicAdd(Q.ctr + kCtrPool, (unsigned long long)no);
          oo = __shfl_sync(kFull, oo, 0);
          if ((int64_t)oo + no > Q.pool_cap) no = -1;
          else
            for (int k = lane; k < no; k += 32) Q.pool[oo + k] = W.walk.own[k];
        }
        __syncwarp();
        if (lane == pl) {
          n = no < 0 ? -2 : no;
          off = oo;
        }
      }
      // list pairs from the front of the slots, the others from the back
      const uint32_t walks = __ballot_sync(kFull, mine && n < 0), lists = queued & ~walks;
      unsigned long long slot = 0, wslot = 0;
      if (lane == 0 && lists) slot = atomicAdd(Q.ctr + kCtrSlots, (unsigned long long)__popc(lists));
      if (lane == 0 && walks) wslot = atomicAdd(Q.ctr + kCtrWalk, (unsigned long long)__popc(walks));
      slot = __shfl_sync(kFull, slot, 0) + __popc(lists & lanemask_lt());
      wslot = __shfl_sync(kFull, wslot, 0) + __popc(walks & lanemask_lt());
      if (mine) {
        // what the pair kernel would find out once per pair, here by a lane per pair
        uint32_t flags = 0;
        if (t.flat[i] && t.flat[j] && t.nrm[3 * i] == t.nrm[3 * j] && t.nrm[3 * i + 1] == t.nrm[3 * j + 1] &&
            t.nrm[3 * i + 2] == t.nrm[3 * j + 2])
          flags |= kOccSame;
        if (t.mixed) {
          const double d0 = cj[0] - t.cen[3 * i], d1 = cj[1] - t.cen[3 * i + 1], d2 = cj[2] - t.cen[3 * i + 2];
          const double dm = fmax(t.diam[i], t.diam[j]) * t.near_factor, dd = d0 * d0 + d1 * d1 + d2 * d2;
          const double sr = t.rad[i] + rj;
          if (dd < dm * dm) flags |= kOccNear | kOccTight;  // (near: rays formed in FP64)
          else if (sr * sr <= 0.36 * dd) flags |= kOccTight;
          if (pair_misses_box<true>(t.cen + 3 * i, cj, fmax(t.rad[i], rj) + t.cull_margin, t.nodes[0]))
            flags |= kOccOut;
        }
        OccSlot s;
        s.i = (int32_t)i;
        s.j = (int32_t)j;
        s.req = (int32_t)((uint32_t)s_req | flags);
        s.n = n < 0 ? -1 : n;
        s.off = (int64_t)off;
        Q.slots[n < 0 ? Q.scap - 1 - (int64_t)wslot : (int64_t)slot] = s;
        n_list += n >= 0 ? 1 : 0;
        n_walk += n < 0 ? 1 : 0;
      }
      __syncwarp();
    }
    __syncthreads();
  }
  if (B.counters) {
    const uint64_t s_l = warp_sum_u64(n_list), s_w = warp_sum_u64(n_walk), s_m = warp_sum_u64(n_masked);
    if (lane == 0 && (s_l | s_w | s_m)) {
      atomicAdd(B.counters + 11, (unsigned long long)s_l);
      atomicAdd(B.counters + 12, (unsigned long long)s_w);
      atomicAdd(B.counters + 14, (unsigned long long)s_m);
    }
  }
}

// 2. The tiles' pairs outside their mask rows: a warp per row (or per four
// rows of a tile when there are many).
template <bool MIXED>
__global__ void __launch_bounds__(256, 2) k_occ_rest(const OccBatch* __restrict__ Lp) {
  extern __shared__ __align__(128) unsigned char smem[];
  const OccBatch& B = *Lp;
  double* S = reinterpret_cast<double*>(smem) + (threadIdx.x >> 5) * 8 * B.pmax_max;
  const int lane = threadIdx.x & 31;
  const unsigned long long claimed = *(volatile unsigned long long*)(B.q.ctr + kCtrTile) / (unsigned)B.groups;
  const int64_t n_tiles = claimed < (unsigned long long)B.total_tiles ? (int64_t)claimed : B.total_tiles;
  uint32_t cnt[6] = {0, 0, 0, 0, 0, 0};
  for (;;) {
    unsigned long long k = 0;
    if (lane == 0) k = atomicAdd(B.q.ctr + kCtrHead32, 1ull);
    k = __shfl_sync(kFull, k, 0);
    const int64_t g = (int64_t)(k / (unsigned)B.rest_parts);
    if (g >= n_tiles) break;
    const int part = (int)(k - (unsigned long long)g * (unsigned)B.rest_parts);
    const int r = find_req(B.tile_base, B.n_req, g);
    const OccArgs& t = B.reqs[r];
    const int64_t tile = t.work[g - B.tile_base[r] + t.tile0];
    int64_t bi, bj;
    tile_coords(tile, t.nT, bi, bj);
    for (int li = part; li < kTile; li += B.rest_parts) {
      const int64_t i = bi * kTile + li;
      if (i >= t.N) break;
      const uint32_t skip = t.tmask[tile * kTile + li];
      if constexpr (MIXED) {
        const MixedArgs& a = B.mreqs[r];
        const int64_t j = bj * kTile + lane;
        bool near = false, close = false;
        if (j < a.N && i < j) {
          const double d0 = a.cen[3 * j] - a.cen[3 * i], d1 = a.cen[3 * j + 1] - a.cen[3 * i + 1],
                       d2 = a.cen[3 * j + 2] - a.cen[3 * i + 2];
          const double q = d0 * d0 + d1 * d1 + d2 * d2;
          const double dm = fmax(a.diam[i], a.diam[j]) * a.near_factor;
          near = q < dm * dm;
          const double sr = a.rad[i] + a.rad[j] + a.tiny_gap;
          close = near || q <= sr * sr;
        }
        if (skip == 0 && !__any_sync(kFull, close))
          fast_mixed<true>(a, a.tabf + bi * kComp * a.pmax * kTile, bi, bj, li + 8, lane, cnt[0], cnt[1]);
        else row_visible_mixed(a, bi, bj, li, skip, near, cnt);
      } else {
        const PairArgs& a = B.preqs[r];
        fast_fp64<true, true>(a, a.tab + bi * kComp * a.pmax * kTile, S, bi, bj, li + 8, lane, cnt[0], cnt[1], skip);
      }
    }
  }
  if (B.counters) {
    const int at[5] = {0, 1, 4, 5, 6};
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const uint64_t s = warp_sum_u64(cnt[k]);
      if (lane == 0 && s) atomicAdd(B.counters + at[k], (unsigned long long)s);
    }
  }
}

// The reference's ray (i, p) -> (j, q), or false when none is cast.
__device__ __forceinline__ bool occ_ray64(const OccArgs& t, int64_t i, int64_t j, int p, int q, bool sw, RayD& R) {
  const int pm = t.pmax;
  double xi[3], xj[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    xi[k] = t.tab[tab_at(i, k, p, pm)];
    xj[k] = t.tab[tab_at(j, k, q, pm)];
  }
  const double rx = xj[0] - xi[0], ry = xj[1] - xi[1], rz = xj[2] - xi[2];
  const double r2 = (rx * rx + ry * ry) + rz * rz;
  return sw ? make_ray(xj, -rx, -ry, -rz, r2, R) : make_ray(xi, rx, ry, rz, r2, R);
}
// Whether it passes the root box.
__device__ __noinline__ bool occ_reaches64(const OccArgs& t, int64_t i, int64_t j, int p, int q, bool sw) {
  RayD R;
  return occ_ray64(t, i, j, p, q, sw, R) && slab_d(t.nodes[0], R);
}

// Whether the FP64 ray (i, p) -> (j, q) is blocked, with the reference's
// arithmetic, the warp's lanes taking its list's leaves.  A ray without a list,
// or with 1/d not finite, walks the tree (every lane the same walk).
// Warp-uniform call and result.
struct Blocked64 {
  bool blocked;
  uint32_t nodes, prims;  // the lane's tests
};
__device__ __noinline__ Blocked64 occ_blocked64(const OccArgs& t, int64_t i, int64_t j, int p, int q, bool sw,
                                                const uint32_t* list, int n) {
  const int lane = threadIdx.x & 31;
  Blocked64 c{false, 0, 0};
  RayD R;
  if (!occ_ray64(t, i, j, p, q, sw, R) || !slab_d(t.nodes[0], R)) return c;
  const bool finite = !R.zdir && isfinite(R.inv[0]) && isfinite(R.inv[1]) && isfinite(R.inv[2]);
  if (n >= 0 && finite) {
    for (int b = 0; b < n && !c.blocked; b += 32) {
      bool hit = false;
      if (b + lane < n) {
        const uint32_t e = list[b + lane];
        const NodeD& leaf = t.nodes[e >> 8];
        ++c.nodes;
        if (slab_d(leaf, R))
          for (uint32_t m = e & 255u; m && !hit; m &= m - 1u) {
            ++c.prims;
            hit = mt_d(t.tris[leaf.a + __ffs(m) - 1], R);
          }
      }
      c.blocked = __any_sync(kFull, hit);
    }
    return c;
  }
  const int32_t gi = t.group[i], gj = t.group[j];
  for (int k = 0; k < t.n_nodes;) {  // miss links point forward (checked when the tree is uploaded)
    const NodeD& nd = t.nodes[k];
    c.nodes += lane == 0 ? 1 : 0;
    if (!slab_d(nd, R)) {
      k = nd.miss;
      continue;
    }
    // a leaf's triangles (at most eight), one a lane
    bool hit = false;
    if (lane < nd.b) {
      const TriD& tr = t.tris[nd.a + lane];
      if (tr.group != gi && tr.group != gj) {
        ++c.prims;
        hit = mt_d(tr, R);
      }
    }
    if (__any_sync(kFull, hit)) {
      c.blocked = true;
      return c;
    }
    k = nd.b > 0 ? nd.miss : k + 1;
  }
  return c;
}

// The warp's FP32 rays by walks of the tree, one ray a lane, the leaf tests
// dealt out to the lanes (device_trace.cuh): kHit, kMiss or kUnsure.
__device__ __noinline__ int occ_walk32(const OccArgs& t, bool live, const RayF R, int32_t gi, int32_t gj, RayBankF& ws,
                                       uint32_t* tests) {
  PolF3 pol;
  pol.R = R;
  pol.tris = t.trisf;
  TravCount tc;
  if (live) pol.store(ws, threadIdx.x & 31, gi, gj);
  const int s = trace_batch<true>(live, GlobalNodes<NodeF>{t.nodesf}, t.n_nodes, ws, pol, tc);
  tests[0] += tc.nodes;
  tests[1] += tc.prims;
  tests[2] += tc.unsure_slab;
  tests[3] += tc.unsure_prim;
  return s;
}

// 3. The queued pairs.  The pair's quadrature points are staged in shared
// memory, eight values a point.  WALK: the pairs without a list (elements coarse
// against the obstruction), queued from the other end of the slots; their rays
// walk the tree.  In a kernel of its own: the walk's code and shared memory cost
// the list pairs 8 to 16% (closed cube of 43,200 elements).
template <bool MIXED, bool WALK>
__global__ void __launch_bounds__(256, WALK ? 3 : 2) k_occ_pairs(const OccBatch* __restrict__ Lp) {
  extern __shared__ __align__(128) unsigned char smem[];
  const OccBatch& B = *Lp;
  const OccQ& Q = B.q;
  const int lane = threadIdx.x & 31;
  using Real = typename std::conditional<MIXED, float, double>::type;
  Real* Pi = reinterpret_cast<Real*>(smem + (WALK ? 8 * sizeof(RayBankF) : 0)) + (size_t)(threadIdx.x >> 5) * 16 * B.pmax_max;
  uint32_t walk_tests[4] = {0, 0, 0, 0};
  Real* Pj = Pi + 8 * B.pmax_max;
  const int64_t ns = (int64_t) * (volatile unsigned long long*)(Q.ctr + (WALK ? kCtrWalk : kCtrSlots));
  // point pairs, rays, FP64 rays, near pairs, grazing point pairs, unusable directions
  uint32_t n_pp = 0, n_rays = 0, n_rays64 = 0, n_near = 0, n_graze = 0, n_bad = 0;
  uint32_t n_nodes = 0, n_prims = 0, n_traced = 0, n_unsure = 0, n_us = 0, n_up = 0;
  for (;;) {
    // up to eight pairs per claim (neighbours share points in L1), fewer
    // towards the end: lists differ in length by two orders of magnitude
    unsigned long long s0 = 0, len = 1;
    if (lane == 0) {
      const unsigned long long at = *(volatile unsigned long long*)(Q.ctr + (WALK ? kCtrWalkHead : kCtrHead64));
      const unsigned long long left = at < (unsigned long long)ns ? ((unsigned long long)ns - at) / (8ull * gridDim.x * 8) : 0;
      len = left < 1 ? 1 : left > 8 ? 8 : left;
      s0 = atomicAdd(Q.ctr + (WALK ? kCtrWalkHead : kCtrHead64), len);
    }
    s0 = __shfl_sync(kFull, s0, 0);
    len = __shfl_sync(kFull, len, 0);
    if ((int64_t)s0 >= ns) break;
    const int64_t s1 = min(ns, (int64_t)(s0 + len));
    for (int64_t s = (int64_t)s0; s < s1; ++s) {
      const OccSlot ps = Q.slots[WALK ? Q.scap - 1 - s : s];
      const OccArgs& t = B.reqs[ps.req & 255];
      const int64_t i = ps.i, j = ps.j, N = t.N;
      const int pm = t.pmax;
      const int64_t oi = t.orig ? (int64_t)t.orig[i] : i, oj = t.orig ? (int64_t)t.orig[j] : j;
      const bool sw = oi > oj;  // the reference casts from the lower caller index
      const int npi = t.np[i];
      const int npj = ps.req & kOccSame ? 0 : t.np[j];  // one normal, bit for bit: K = 0
      const uint32_t* list = Q.pool + ps.off;
      const uint32_t e0 = lane < ps.n ? list[lane] : 0u, e1 = 32 + lane < ps.n ? list[32 + lane] : 0u;
      const NodeF* nodesf = t.nodesf;
      const TriF* trisf = t.trisf;
      const float delta = t.delta;
      const MtTol tol = !MIXED || (ps.req & kOccTight) ? kMtTight : kMtLoose;
      const double* it = t.tab + tab_at(i, 0, 0, pm);
      const double* jt = t.tab + tab_at(j, 0, 0, pm);
      const float per = 1.0f / (float)pm;  // v + 1/2 is at least 1/128 from a multiple of pm, v < 448
      {
        const Real* ti;
        const Real* tj;
        if constexpr (MIXED) {
          ti = t.tabf + tab_at(i, 0, 0, pm);
          tj = t.tabf + tab_at(j, 0, 0, pm);
        } else {
          ti = it;
          tj = jt;
        }
        for (int v = lane; v < kComp * pm; v += 32) {
          const int c = (int)(((float)v + 0.5f) * per), p = v - c * pm;
          Pi[8 * p + c] = ti[v * kTile];
          Pj[8 * p + c] = tj[v * kTile];
        }
        __syncwarp();
      }
      double ci[3], dc[3];
      bool near = false, cullp = false;
      float r2_min = 1e-18f;  // shorter far rays go to FP64 (kMtLoose)
      if constexpr (MIXED) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          ci[k] = t.cen[3 * i + k];
          dc[k] = t.cen[3 * j + k] - ci[k];
        }
        if (!(ps.req & kOccTight)) {
          const double span = sqrt(dc[0] * dc[0] + dc[1] * dc[1] + dc[2] * dc[2]) + t.rad[i] + t.rad[j];
          r2_min = fmaxf(r2_min, kMinRay2 * (float)(span * span));
        }
        near = (ps.req & kOccNear) != 0;
        n_near += near && npj > 0 && lane == 0 ? 1 : 0;
        cullp = (ps.req & kOccOut) != 0;
      }
      n_pp += lane == 0 ? npi * npj : 0;
      double accd = 0.0;    // the lane's FP64 terms
      float acc32 = 0.0f;   // mixed: the FP32 terms of rays that miss the root box, in the generation's order
      const int Qc = pm < 8 ? pm : pm <= 64 ? 64 / pm : 1;  // source points q of one pass (at most 64 rays)
      for (int q0 = 0; q0 < npj; q0 += Qc) {
        const int nray = min(Qc, npj - q0) * pm;
        RayF R[2];
        double term[2];
        float k32[2];
        int st[2];          // kMiss visible, kHit blocked, kUnsure: FP64
        bool live[2];       // tested against the list
        bool in64[2];       // the term is added in FP64
        int pp[2], qq[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int r = 32 * u + lane;
          const int dq = (int)(((float)r + 0.5f) * per);
          const int p = r - dq * pm, q = q0 + dq;
          pp[u] = p;
          qq[u] = q;
          const bool lq = r < nray && p < npi;
          st[u] = kMiss;
          live[u] = false;
          term[u] = 0.0;
          k32[u] = 0.0f;
          in64[u] = !MIXED;
          if (32 * u >= nray) continue;  // warp-uniform
          bool exact = lq;
          float rx = 0.f, ry = 0.f, rz = 0.f, r2 = 0.f, wp = 0.f, wq = 0.f;
          float xo[3] = {0.f, 0.f, 0.f};
          bool cast = false;
          if constexpr (MIXED) {
            // the mixed generation's far-field arithmetic, operation for operation
            const bool far = lq && !near;
            bool graze = false;
            if (far) {
              const float4 a0 = *reinterpret_cast<const float4*>(Pi + 8 * p), a1 = *reinterpret_cast<const float4*>(Pi + 8 * p + 4);
              const float4 b0 = *reinterpret_cast<const float4*>(Pj + 8 * q), b1 = *reinterpret_cast<const float4*>(Pj + 8 * q + 4);
              const float op0 = a0.x, op1 = a0.y, op2 = a0.z, np0 = a0.w, np1 = a1.x, np2 = a1.y;
              const float oq0 = b0.x, oq1 = b0.y, oq2 = b0.z, nq0 = b0.w, nq1 = b1.x, nq2 = b1.y;
              wp = a1.z;
              wq = b1.z;
              rx = (float)dc[0] + (oq0 - op0);
              ry = (float)dc[1] + (oq1 - op1);
              rz = (float)dc[2] + (oq2 - op2);
              r2 = fmaf(rx, rx, fmaf(ry, ry, rz * rz));
              const float di = fmaf(np0, rx, fmaf(np1, ry, np2 * rz));
              const float dj = -fmaf(nq0, rx, fmaf(nq1, ry, nq2 * rz));
              graze = r2 < 1e-18f || di * di <= 1e-10f * r2 || dj * dj <= 1e-10f * r2;
              if (!graze && di > 0.0f && dj > 0.0f) k32[u] = (di * dj) * rcp_approx(3.14159265f * (r2 * r2));
              xo[0] = (float)(ci[0] + (sw ? dc[0] : 0.0)) + (sw ? oq0 : op0);
              xo[1] = (float)(ci[1] + (sw ? dc[1] : 0.0)) + (sw ? oq1 : op1);
              xo[2] = (float)(ci[2] + (sw ? dc[2] : 0.0)) + (sw ? oq2 : op2);
              cast = k32[u] > 0.0f;
              term[u] = (double)(wq * (wp * k32[u]));
              n_graze += graze ? 1 : 0;
            }
            exact = lq && (near || graze);
          }
          if (exact) {
            double xi[3], ni[3], xj[3], nj[3];
            double wi, wj;
            if constexpr (MIXED) {
#pragma unroll
              for (int k = 0; k < 3; ++k) {
                xi[k] = it[(k * pm + p) * kTile];
                ni[k] = it[((3 + k) * pm + p) * kTile];
                xj[k] = jt[(k * pm + q) * kTile];
                nj[k] = jt[((3 + k) * pm + q) * kTile];
              }
              wi = it[(6 * pm + p) * kTile];
              wj = jt[(6 * pm + q) * kTile];
            } else {
              const double2* A = reinterpret_cast<const double2*>(Pi + 8 * p);
              const double2* B2 = reinterpret_cast<const double2*>(Pj + 8 * q);
              const double2 a0 = A[0], a1 = A[1], a2 = A[2], b0 = B2[0], b1 = B2[1], b2 = B2[2];
              xi[0] = a0.x; xi[1] = a0.y; xi[2] = a1.x; ni[0] = a1.y; ni[1] = a2.x; ni[2] = a2.y;
              xj[0] = b0.x; xj[1] = b0.y; xj[2] = b1.x; nj[0] = b1.y; nj[1] = b2.x; nj[2] = b2.y;
              wi = Pi[8 * p + 6];
              wj = Pj[8 * q + 6];
            }
            const double dx = xj[0] - xi[0], dy = xj[1] - xi[1], dz = xj[2] - xi[2];
            const double d2 = (dx * dx + dy * dy) + dz * dz;
            const double K = k_fast<true>(dx, dy, dz, d2, ni, nj);
            term[u] = wj * (wi * K);
            in64[u] = true;
            cast = K > 0.0 && (d2 > 2e-30 || sqrt(d2) > 1e-15);  // make_ray's cast rule
            n_rays64 += MIXED && cast ? 1 : 0;
            rx = (float)dx;
            ry = (float)dy;
            rz = (float)dz;
            r2 = fmaf(rx, rx, fmaf(ry, ry, rz * rz));
#pragma unroll
            for (int k = 0; k < 3; ++k) xo[k] = (float)(sw ? xj[k] : xi[k]);
          }
          n_rays += cast ? 1 : 0;
          if (cast && !cullp) {
            const bool rok = r2 > (exact ? 1e-18f : r2_min) && (sw ? make_ray_f(xo, -rx, -ry, -rz, r2, delta, R[u])
                                                : make_ray_f(xo, rx, ry, rz, r2, delta, R[u]));
            if (rok) {
              const int sr = slab_f(nodesf[0], R[u]);
              if (sr != kMiss) {
                // (a ray that may miss the root box: its leaves decide, whose boxes lie in it)
                live[u] = true;
                if (MIXED && !exact) in64[u] = true;  // a ray the root box may hold
                // mixed: the rays with FP64 terms; FP64: those that pass the root box
                n_traced += (MIXED ? !exact : sr == kHit || occ_reaches64(t, i, j, p, q, sw)) ? 1 : 0;
                n_us += sr == kUnsure ? 1 : 0;
              }
            } else {
              st[u] = kUnsure;
              in64[u] = true;
              n_bad += MIXED && !exact ? 1 : 0;
              n_rays64 += MIXED && !exact ? 1 : 0;
              n_traced += !MIXED && occ_reaches64(t, i, j, p, q, sw) ? 1 : 0;
            }
          }
        }
        // the pair's list: every lane tests the same box or triangle
        bool open[2] = {live[0], live[1]}, doubt[2] = {false, false};
        for (int k = 0; !WALK && k < ps.n; ++k) {
          if (!__any_sync(kFull, open[0] || open[1])) break;
          const uint32_t e = __shfl_sync(kFull, k < 32 ? e0 : e1, k & 31);
          const NodeF box = nodesf[e >> 8];
          int sb[2];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            sb[u] = open[u] ? slab_f(box, R[u]) : kMiss;
            n_nodes += open[u] ? 1 : 0;
            n_us += sb[u] == kUnsure ? 1 : 0;
          }
          if (!__any_sync(kFull, sb[0] != kMiss || sb[1] != kMiss)) continue;
          const TriF* tri = trisf + (box.ab >> 4);
          for (uint32_t m = e & 255u; m; m &= m - 1u) {
            const TriF tr = tri[__ffs(m) - 1];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              if (sb[u] == kMiss) continue;
              ++n_prims;
              const int h = mt_f(tr, R[u], tol);
              n_up += h == kUnsure ? 1 : 0;
              if (h == kHit && sb[u] == kHit) {
                st[u] = kHit;
                open[u] = false;
                sb[u] = kMiss;
              } else if (h != kMiss) {
                doubt[u] = true;
              }
            }
          }
        }
        if constexpr (WALK) {
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            if (!__any_sync(kFull, live[u])) continue;
            const int s = occ_walk32(t, live[u], R[u], t.group[i], t.group[j],
                                     reinterpret_cast<RayBankF*>(smem)[threadIdx.x >> 5], walk_tests);
            if (live[u] && s == kHit) st[u] = kHit;
            doubt[u] = s == kUnsure;
          }
        }
        // FP64 for the uncertain rays, one after another
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if (live[u] && st[u] != kHit && doubt[u]) st[u] = kUnsure;
          for (uint32_t m = __ballot_sync(kFull, st[u] == kUnsure); m; m &= m - 1u) {
            const int src = __ffs(m) - 1;
            const Blocked64 x = occ_blocked64(t, i, j, __shfl_sync(kFull, pp[u], src), __shfl_sync(kFull, qq[u], src), sw,
                                              list, ps.n);
            n_nodes += x.nodes;
            n_prims += x.prims;
            if (lane == src) {
              ++n_unsure;
              n_rays64 += MIXED ? 1 : 0;
              st[u] = x.blocked ? kHit : kMiss;
            }
          }
          if (in64[u] && st[u] == kMiss) accd += term[u];
        }
        if constexpr (MIXED) {
          // the remaining FP32 terms: lane q sums its point's over p, then the points in order
          const float f0 = in64[0] ? 0.0f : k32[0], f1 = in64[1] ? 0.0f : k32[1];
          if (__any_sync(kFull, f0 != 0.0f || f1 != 0.0f)) {
            const int nq = min(Qc, npj - q0);
            float inner = 0.0f;
            for (int p = 0; p < npi; ++p) {
              const int r = lane * pm + p;
              const float v0 = __shfl_sync(kFull, f0, r & 31), v1 = __shfl_sync(kFull, f1, r & 31);
              inner = fmaf(Pi[8 * p + 6], (r >> 5) & 1 ? v1 : v0, inner);
            }
            const float wq = lane < nq ? Pj[8 * (q0 + lane) + 6] : 0.0f;
            for (int u = 0; u < nq; ++u)
              acc32 = fmaf(__shfl_sync(kFull, wq, u), __shfl_sync(kFull, inner, u), acc32);
          }
        }
      }
      double acc = accd;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o);
      if constexpr (MIXED) acc += (double)acc32;
      if (lane < 2) t.F[lane == 0 ? oi + oj * N : oj + oi * N] = acc / t.area[lane == 0 ? i : j];
      __syncwarp();  // before the next pair's points
    }
  }
  n_nodes += walk_tests[0];
  n_prims += walk_tests[1];
  n_us += walk_tests[2];
  n_up += walk_tests[3];
  if (B.counters) {
    // counters: 0 point pairs, 1 rays, 2 box tests, 3 triangle tests, 4 FP64 rays, 5 near pairs, 6 grazing,
    // 7 unsure rays, 8 / 9 unsure boxes / triangles, 10 unusable directions
    const uint32_t v[11] = {n_pp, n_rays, n_nodes, n_prims, n_rays64, n_near, n_graze, n_unsure, n_us, n_up, n_bad};
#pragma unroll
    for (int k = 0; k < 11; ++k) {
      const uint64_t s = warp_sum_u64(v[k]);
      if (lane == 0 && s) atomicAdd(B.counters + k, (unsigned long long)s);
    }
    const uint64_t s = warp_sum_u64(n_traced);
    if (lane == 0 && s) atomicAdd(Q.ctr + kCtrRec64, (unsigned long long)s);
  }
}

// Tasks per tile of the list kernel: a task is all of a tile's rows, a half, or
// 8 of them (one per warp).  Tiles differ in cost by two orders of magnitude,
// so a launch wants 16 tasks per resident block.
int occ_groups(int64_t n_tiles, int sm_count) {
  const int64_t want = (int64_t)16 * 3 * sm_count;
  return n_tiles >= want ? 1 : 2 * n_tiles >= want ? 2 : 4;
}

int occ_list_grid(int sm_count) { return 3 * sm_count; }

cudaError_t launch_occ(bool mixed, int pmax, const OccBatch* b, int list_grid, int sm_count, cudaStream_t st,
                       const cudaEvent_t* marks) {
  cudaError_t e =
      cudaFuncSetAttribute(k_occ_list, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(OccTile));
  if (e != cudaSuccess) return e;
  auto mark = [&](int k) {
    if (marks) cudaEventRecord(marks[k], st);
    return cudaGetLastError();
  };
  k_occ_list<<<(unsigned)list_grid, 256, sizeof(OccTile), st>>>(b);
  if ((e = mark(0)) != cudaSuccess) return e;
  if (mixed) k_occ_rest<true><<<(unsigned)(2 * sm_count), 256, 0, st>>>(b);
  else k_occ_rest<false><<<(unsigned)(2 * sm_count), 256, stage_bytes(pmax), st>>>(b);
  if ((e = mark(1)) != cudaSuccess) return e;
  auto pairs = [&](auto fn, size_t smem, int per_sm) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return;
    fn<<<(unsigned)(per_sm * sm_count), 256, smem, st>>>(b);
    e = cudaGetLastError();
  };
  // eight warps: eight values a point for two elements, and the walks' ray banks
  const size_t points = (size_t)8 * 16 * pmax * (mixed ? sizeof(float) : sizeof(double)), bank = 8 * sizeof(RayBankF);
  if (mixed) {
    pairs(k_occ_pairs<true, false>, points, 2);
    pairs(k_occ_pairs<true, true>, bank + points, 3);
  } else {
    pairs(k_occ_pairs<false, false>, points, 2);
    pairs(k_occ_pairs<false, true>, bank + points, 3);
  }
  if (e != cudaSuccess) return e;
  return mark(2);
}

}  // namespace rvf
