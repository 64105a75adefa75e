// device_segs.cuh -- segment lists of curve meshes: the obstruction segments a
// tile's rays, and a pair's, can be blocked by.  Every ray of a pair lies within
// R = max(r_i, r_j) of the segment between the elements' centres, and a segment
// farther than R + margin from that one cannot block it (margin bounds how far
// from a ray a computed hit of the reference's segment test can lie).
#pragma once

#include "device_hull.cuh"
#include "kernels.h"

namespace rvf {

struct SegScene {
  const NodeD* nodes;
  const NodeF* nodesf;
  int n_nodes;
  const SegD* segs;
  const int32_t* frontier;
  int n_frontier;
  double margin;
  float slack;  // FP32 rounding of the coordinates (2^-20 of the scene's extent)
};

constexpr int kSegs = 2048;  // segments of a tile's list
constexpr int kRowItems = 2048;  // (pair, segment) items of a row's pairs (more: its rays walk the tree)
constexpr int kFront = kTileFront;

struct SegTile {
  int seg[kSegs];    // segment
  int leaf[kSegs];   // its leaf node
  union {
    struct {
      int front[2 * kFront];
      int leaves[kTileLeaves];
    } walk;
    uint16_t item[8][kRowItems];  // per warp: the row's items, position in the tile's list << 5 | lane of the pair
  };
  double ray[8][4][32];  // per warp: a point pair's rays, from x, y to x, y
};
static_assert(kSegs <= 1 << 11, "an item keeps the position in 11 bits");

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

// The segments within reach of the tile (hull H, largest radius rmax) into T,
// by one warp; their number, or -1 when a capacity is exceeded.  Segments of the
// groups g0, g1 are left out when g_same (every ray of the tile skips them).
__device__ __forceinline__ int tile_segments(const SegScene& sc, const HullF& H, double rmax, bool g_same, int32_t gi0,
                                             int32_t gj0, SegTile& T) {
  const int lane = threadIdx.x & 31;
  const float reach = __double2float_ru(rmax + sc.margin) + sc.slack;
  // the leaves within reach, one tree level per round
  int* cur = T.walk.front;
  int* nxt = T.walk.front + kFront;
  if (lane < sc.n_frontier) cur[lane] = sc.frontier[lane];
  __syncwarp();
  int ncur = sc.n_frontier, nleaf = 0;
  bool over = false;
  while (ncur > 0 && !over) {
    int nnext = 0;
    for (int b = 0; b < ncur; b += 32) {
      const int q = b + lane;
      bool pass = false, leaf = false;
      int k = 0, right = 0;
      if (q < ncur && cur[q] < sc.n_nodes) {
        k = cur[q];
        const NodeF nd = sc.nodesf[k];
        pass = !hull2_misses(H, nd.lo[0], nd.lo[1], nd.hi[0], nd.hi[1], reach);
        leaf = (nd.ab & 15) > 0;
        if (pass && !leaf) right = sc.nodesf[k + 1].miss;
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
      const int32_t ab = sc.nodesf[leaf].ab;
      if (u8 < (ab & 15)) {
        u = (ab >> 4) + u8;
        const SegD sg = sc.segs[u];
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
  __syncwarp();
  return over || ns > kSegs ? -1 : ns;
}

// The segments the row's pairs can be blocked by (lane: row element centre A and
// radius ri, column element cj, rj) as items in T.item[warp]; their number, or -1
// (the row's rays walk the tree: too many, or no tile list).  `some`: the pairs
// with an item (all valid ones when they walk).  skip: rays skip the groups gi, gj.
// Warp-uniform call and number.
__device__ __forceinline__ int row_segments(const SegScene& sc, const HullF& H, SegTile& T, int nseg, int warp,
                                            const double* A, const double* cj, double ri, double rj, double rj_max,
                                            bool valid, bool skip, int32_t gi, int32_t gj, uint32_t& some,
                                            int limit = kRowItems) {
  const int lane = threadIdx.x & 31;
  some = 0;
  int n = 0;
  __syncwarp();  // the last row's items are read
  if (nseg > 0) {
    const double d[2] = {cj[0] - A[0], cj[1] - A[1]};
    const double L2 = d[0] * d[0] + d[1] * d[1], R = fmax(ri, rj) + sc.margin, RL = R * sqrt(L2);
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
    const float row_reach = __double2float_ru(fmax(ri, rj_max) + sc.margin) + sc.slack;
    for (int b = 0; b < nseg && n <= limit; b += 32) {
      bool keep = false;
      if (b + lane < nseg) {
        const SegD sg = sc.segs[T.seg[b + lane]];
        const float x0 = (float)sg.x0, y0 = (float)sg.y0, x1 = (float)sg.x1, y1 = (float)sg.y1;
        keep = !(skip && sg.group == gi) &&
               !hull2_misses(Hr, fminf(x0, x1), fminf(y0, y1), fmaxf(x0, x1), fmaxf(y0, y1), row_reach);
      }
      for (uint32_t m = __ballot_sync(kFull, keep); m; m &= m - 1u) {  // lanes are pairs again
        const int at = b + __ffs(m) - 1;
        const SegD sg = sc.segs[T.seg[at]];
        const double s0[2] = {sg.x0, sg.y0}, s1[2] = {sg.x1, sg.y1};
        const bool in = valid && !(skip && sg.group == gj) && !capsule2_misses(A, d, L2, RL, R, s0, s1);
        const uint32_t mi = __ballot_sync(kFull, in);
        const int pos = n + __popc(mi & lanemask_lt());
        if (in && pos < kRowItems) T.item[warp][pos] = (uint16_t)((at << 5) | lane);
        n += __popc(mi);
        some |= mi;
      }
    }
  }
  __syncwarp();
  if (nseg < 0 || n > limit) {
    some = __ballot_sync(kFull, valid);
    return -1;
  }
  return n;
}

// The lanes (of `cast`) whose ray from -> to is blocked by one of the row's n
// items, dealt out to the lanes: a lane tests another lane's ray, and the rays'
// tests of one segment share its load.  The reference tests a segment when the
// ray's bounding box overlaps its leaf's: looked at for the few hits.
// Warp-uniform call and result.
__device__ __forceinline__ uint32_t items_block(const SegScene& sc, SegTile& T, int warp, int n, uint32_t cast,
                                                const double* from, const double* to, uint32_t& n_nodes,
                                                uint32_t& n_prims) {
  const int lane = threadIdx.x & 31;
  double(*ray)[32] = T.ray[warp];
  __syncwarp();
  ray[0][lane] = from[0];
  ray[1][lane] = from[1];
  ray[2][lane] = to[0];
  ray[3][lane] = to[1];
  __syncwarp();
  uint32_t blocked = 0;
  for (int b = 0; b < n; b += 32) {
    const int item = b + lane < n ? T.item[warp][b + lane] : 0, o = item & 31, at = item >> 5;
    bool hit = false;
    if (b + lane < n && (((cast & ~blocked) >> o) & 1u)) {
      const double f[2] = {ray[0][o], ray[1][o]}, t[2] = {ray[2][o], ray[3][o]};
      ++n_prims;
      if (seg_blocks(sc.segs[T.seg[at]], f, t)) {
        const NodeD& nd = sc.nodes[T.leaf[at]];
        ++n_nodes;
        hit = !(nd.lo[0] > fmax(f[0], t[0]) || nd.hi[0] < fmin(f[0], t[0]) || nd.lo[1] > fmax(f[1], t[1]) ||
                nd.hi[1] < fmin(f[1], t[1]));
      }
    }
    if (__any_sync(kFull, hit)) blocked |= __reduce_or_sync(kFull, hit ? 1u << o : 0u);
  }
  return blocked;
}

}  // namespace rvf
