// wave_host.cpp -- host side of the wavefront pair pipeline (kernels_wave.cu):
// per-request kernel arguments, queue sizing, and chunked launches over one
// or more requests of one launch shape, optionally replayed from a CUDA graph
// captured per shape.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "kernels.h"
#include "wave_host.h"

namespace rvf {

// Ray queues of the pipeline, kept by the session and grown on demand.
// Capacity: every point pair of every tile when that is small, otherwise up
// to 2^29 records per queue (4 GiB) within the HBM budget, and never below a
// few tiles' worst case.
int ensure_wave(Session* s, bool two_queues, bool occ, bool lists, int pmax, int64_t n_tiles, WaveQ& q) {
  int rc = 0;
  if (!s->wq_ctr.ptr && (rc = s->wq_ctr.alloc(s, sizeof(unsigned long long) * kCtrCount))) return rc;
  q = WaveQ{};
  q.ctr = s->wq_ctr.as<unsigned long long>();
  q.vis_words = (pmax * pmax + 63) / 64;
  if (!occ) return 0;
  const int64_t per_tile = (int64_t)kTile * kTile * pmax * pmax;
  const int64_t want = std::min<int64_t>(n_tiles * per_tile, (int64_t)1 << 29);
  const int64_t floor_recs = std::min<int64_t>(n_tiles * per_tile, 4 * per_tile);
  const int64_t want_s = std::min<int64_t>(n_tiles * kTile * kTile, (int64_t)1 << 25);
  const int64_t floor_s = std::min<int64_t>(n_tiles * kTile * kTile, 4 * kTile * kTile);
  const int nq = two_queues ? 2 : 1;
  // pair lists: 8 B per slot and a pool of kPoolPerSlot entries per slot
  constexpr int64_t kPoolPerSlot = 24;
  const size_t slot_bytes = sizeof(PendSlot) + sizeof(unsigned long long) * q.vis_words +
                            (lists ? sizeof(PairList) + sizeof(int32_t) * kPoolPerSlot : 0);
  auto have = [&](int64_t recs, int64_t slots) {
    return s->wq_rec64.bytes >= sizeof(uint64_t) * recs &&
           (!two_queues || s->wq_rec32.bytes >= sizeof(uint64_t) * recs) &&
           s->wq_slots.bytes >= sizeof(PendSlot) * slots &&
           s->wq_vis.bytes >= sizeof(unsigned long long) * q.vis_words * slots &&
           (!lists || (s->wq_plist.bytes >= sizeof(PairList) * slots &&
                       s->wq_pool.bytes >= sizeof(int32_t) * kPoolPerSlot * slots));
  };
  int64_t recs = want, slots = want_s;
  if (!have(recs, slots)) {
    // release and size against the budget left
    s->wq_rec64.free_();
    s->wq_rec32.free_();
    s->wq_slots.free_();
    s->wq_vis.free_();
    s->wq_plist.free_();
    s->wq_pool.free_();
    const size_t left = s->budget > s->used ? s->budget - s->used : 0;
    while ((size_t)(recs * 8 * nq) + (size_t)slots * slot_bytes > left / 2 && (recs > floor_recs || slots > floor_s)) {
      recs = std::max<int64_t>(floor_recs, recs / 2);
      slots = std::max<int64_t>(floor_s, slots / 2);
    }
    if ((rc = s->wq_rec64.alloc(s, sizeof(uint64_t) * recs))) return rc;
    if (two_queues && (rc = s->wq_rec32.alloc(s, sizeof(uint64_t) * recs))) return rc;
    if ((rc = s->wq_slots.alloc(s, sizeof(PendSlot) * slots))) return rc;
    if ((rc = s->wq_vis.alloc(s, sizeof(unsigned long long) * q.vis_words * slots))) return rc;
    if (lists && (rc = s->wq_plist.alloc(s, sizeof(PairList) * slots))) return rc;
    if (lists && (rc = s->wq_pool.alloc(s, sizeof(int32_t) * kPoolPerSlot * slots))) return rc;
  }
  q.rec64 = s->wq_rec64.as<uint64_t>();
  q.rec32 = two_queues ? s->wq_rec32.as<uint64_t>() : nullptr;
  q.cap = (int64_t)(s->wq_rec64.bytes / sizeof(uint64_t));
  if (two_queues) q.cap = std::min<int64_t>(q.cap, (int64_t)(s->wq_rec32.bytes / sizeof(uint64_t)));
  q.slots = s->wq_slots.as<PendSlot>();
  q.vis = s->wq_vis.as<unsigned long long>();
  q.scap = std::min<int64_t>((int64_t)(s->wq_slots.bytes / sizeof(PendSlot)),
                             (int64_t)(s->wq_vis.bytes / (sizeof(unsigned long long) * q.vis_words)));
  q.plist = lists ? s->wq_plist.as<PairList>() : nullptr;
  q.pool = lists ? s->wq_pool.as<int32_t>() : nullptr;
  q.pool_cap = lists ? (int64_t)(s->wq_pool.bytes / sizeof(int32_t)) : 0;
  if (lists) q.scap = std::min<int64_t>(q.scap, (int64_t)(s->wq_plist.bytes / sizeof(PairList)));
  return 0;
}

// The occlusion kernels' pair queue and list pool, kept by the session: a slot
// per pair of the offered tiles, up to 2^25, and eight entries per slot, halved
// until they fit half of the budget left (chunks then hold fewer tiles); the
// list kernel's blocks may each add one tile's 1,024 pairs beyond a full queue.
static int ensure_occ(Session* s, int64_t n_tiles, OccQ& q, int& grid) {
  constexpr int64_t kPool = 8;
  int rc = 0;
  if (!s->wq_ctr.ptr && (rc = s->wq_ctr.alloc(s, sizeof(unsigned long long) * kCtrCount))) return rc;
  const int64_t per = (int64_t)kTile * kTile;
  const int64_t floor = 8 * per;
  int64_t slots = std::min<int64_t>((n_tiles + occ_list_grid(s->sm_count)) * per, (int64_t)1 << 25);
  if (s->wq_slots.bytes < sizeof(OccSlot) * slots || s->wq_pool.bytes < sizeof(uint32_t) * kPool * slots) {
    s->wq_slots.free_();
    s->wq_pool.free_();
    const size_t left = s->budget > s->used ? s->budget - s->used : 0;
    while (slots > floor && (size_t)slots * (sizeof(OccSlot) + sizeof(uint32_t) * kPool) > left / 2)
      slots = std::max<int64_t>(floor, slots / 2);
    if ((rc = s->wq_slots.alloc(s, sizeof(OccSlot) * slots))) return rc;
    if ((rc = s->wq_pool.alloc(s, sizeof(uint32_t) * kPool * slots))) return rc;
  }
  q = OccQ{};
  q.ctr = s->wq_ctr.as<unsigned long long>();
  q.slots = s->wq_slots.as<OccSlot>();
  q.scap = (int64_t)(s->wq_slots.bytes / sizeof(OccSlot));
  q.pool = s->wq_pool.as<uint32_t>();
  q.pool_cap = (int64_t)(s->wq_pool.bytes / sizeof(uint32_t));
  grid = (int)std::max<int64_t>(1, std::min<int64_t>(occ_list_grid(s->sm_count), q.scap / (2 * per)));
  return 0;
}

// Whether a surface solve's tiles with ray work run in the queue pipeline
// (kernels_wave.cu) rather than in the occlusion kernels (kernels_occ.cu).  Those
// build every pair's list from its tile's; where the obstruction is so fine that
// most tiles reach more leaves or triangles than a tile's list holds, each pair walks
// the tree itself and, in mixed precision, sums in FP64, which costs more than the
// rays of a rule of few points.  wide, lng: of the tiles with ray work, the shares
// beyond the classification's 256 leaves, and with 200 leaves (about 1,024 triangles)
// or more.  Both sides were measured over 1,232 solves (12 to 30,000 elements of
// every family, centred boxes of 12 to 10,800 triangles, rules of 1 to 64 points):
// with lists alone 131 of them were slower than the queue pipeline had been, by up
// to 1.8x; with these lines 3, by up to 1.03x.  Examples (ms, lists / queue; wide):
//   FP64, 1 point, 3,750 Quad4, 4,800 triangles (0.94): 8.5 / 4.5; 10,800 Tri3, 2,352 (0.46): 20.2 / 17.4
//   FP64, 7 points, 1,728 Tri3, 10,800 triangles (0.93): 10.9 / 9.4; 4,800 Tri3, 4,800 (0.81): 41.0 / 47.4
//   mixed, 13 points, 768 Tri3, 4,800 triangles (1.0): 6.6 / 3.8; 7 points, 30,000 Tri3, 2,352 (0.30): 198 / 232
//   FP64, 7 points, 108 Tri3, 1,200 triangles (long 1.0): 1.23 / 0.72, the rows of few tiles one after another
// loose: the margin by which rounding can move a hit (it grows with the cube of the unit)
// exceeds a tenth of the triangles' height, so that lists hold whole leaves.  4,800
// Tri3, 1,728 triangles (long 0.1) at a scale of 1,000, 1 / 3 points, mixed: 9.3 / 6.9, 19.7 / 14.6.
static bool occ_by_queue(bool mixed, bool geometric, bool loose, int pmax, int64_t n_tiles, double wide, double lng) {
  const bool few = n_tiles <= 64 && lng >= 0.9 && wide < 0.5;
  if (pmax == 1 && n_tiles <= 200) return wide >= 0.98;
  if (pmax <= 4) {
    if (few && pmax > 1) return true;
    if (n_tiles > 64 && ((loose && lng >= 0.04) || (mixed && geometric && lng >= 0.08))) return true;
    if (mixed) return n_tiles > 64 && (wide >= (geometric ? 0.15 : 0.25) || lng >= 0.35);
    return wide >= (geometric ? 0.3 : 0.4) || (geometric && n_tiles > 64 && lng >= 0.1);
  }
  if (pmax <= 8 && few) return true;
  if (!mixed) return pmax <= 8 ? wide >= 0.92 : pmax <= 16 && few && n_tiles <= 16;
  return pmax <= 16 && n_tiles >= 100 && lng >= 0.42;
}

// Whether FP32 coordinates (2^-20 of 1 + the largest coordinate) are too coarse for
// the obstruction's triangles: the occlusion kernels test rays in FP32 and again,
// one after another, in FP64 when a decision is uncertain, and lists grow with the
// allowance.  Small units or an offset from the origin make it so; the queue pipeline
// then traces FP64 rays 32 at a time.  share: of the triangles' median height.
// Measured over 240 solves (cubes of 768 to 4,800 elements, boxes of 108 to 1,728
// triangles, at scales of 1e-4 to 1e3 and offsets to 1e5), lists against the queue
// pipeline: share 0.013, 1.3 to 2.3x as fast; 0.018, 0.55 to 1.2x; 0.035, 0.14 to 0.5x;
// 0.35, 0.07 to 0.1x.  Rules of up to four points, which gain less: 0.0027, 1.1 to 1.6x;
// 0.0037, 0.8 to 0.9x.  Mixed precision with true vertices: 0.0027, 0.9 to 1.1x.
static bool fp32_too_coarse(const rvf_mesh* m, bool mixed, bool geometric, int pmax) {
  const double h = m->tri_height[geometric ? 1 : 0];
  const double share = h > 0.0 ? std::ldexp(m->extent, -20) / h : 0.0;
  return share >= (mixed && geometric ? 2.5e-3 : pmax <= 4 ? 3e-3 : 1.5e-2);
}

// Whether a mixed solve has many rays with a direction component next to zero, which
// FP32 cannot certify and the pair kernel takes to FP64 one after another, the tree's
// walk for each: structured meshes along the axes (1.5 to 12% of the pairs aligned; nodes
// displaced by 0.3 of an edge, 0.1%) under the obstruction's true vertices, where most
// pairs are blockable.  Lists against the queue pipeline, ms, 9 points: 9,600 Quad4
// 70.6 / 45.7, 5,000 Quad4 in two plates 27.4 / 18.3, 1,536 Quad8 3.48 / 2.54; 4 points,
// 25.5 / 21.1, 10.3 / 9.2 and 1.46 / 1.28; 13 points, 3,072 Tri3 14.8 / 11.5.  At 16 the
// lists win again where few rays are traced: 55.0 / 74.9 in the plates (7.1 / 6.3 for
// 1,536 Quad4 in a cube), at 25 both are equal; 600 Quad4, 4 points, 0.62 / 0.66.
static bool fp64_rays_many(const rvf_mesh* m, bool mixed, bool geometric, int pmax) {
  return mixed && geometric && pmax > 1 && pmax < 16 && m->aligned >= 0.005;
}

int wave_prepare(Session* s, rvf_mesh* m, Tables* T, const rvf_options* o, uint8_t* ray_log, WaveReq& w,
                 int64_t* n_kernels) {
  const int64_t N = m->N;
  const bool occ = o->occlusion && m->n_nodes > 0;
  w = WaveReq{};
  w.mixed = (o->precision == RVF_PREC_MIXED) && (m->dim == 2);
  w.occ = occ;
  w.dim3 = (m->dim == 2);
  w.pmax = T->pmax;
  if (o->fault_inject & RVF_FAULT_CLAIM) w.claim_retries = 0;
  w.tables = T;
  w.fast_qb = o->fast_points;
  w.fast_groups = o->fast_row_groups;  // 0: by the tile count (wave_fast)
  // Meshes with occlusion run the occlusion kernels; the queue pipeline keeps
  // ray logs (every ray's decision in a record), solves without tile classes
  // and obstructions beyond the lists' 24-bit leaf and
  // 25-bit triangle indices.
  w.occ_lists = occ && !o->disable_tile_cull && !ray_log && !(o->fault_inject & RVF_FAULT_CLAIM) &&
            m->frontier.ptr && m->n_nodes < (1 << 24) && m->n_obs < (1 << 25) &&
            !(w.dim3 && (fp32_too_coarse(m, w.mixed, o->geometric_soup != 0, w.pmax) ||
                         fp64_rays_many(m, w.mixed, o->geometric_soup != 0, w.pmax)));
  PairArgs& a = w.pa;
  a.N = N;
  a.nT = (N + kTile - 1) / kTile;
  a.n_tiles = a.nT * (a.nT + 1) / 2;
  a.pmax = T->pmax;
  a.dim3 = w.dim3;
  a.tab = T->tab.as<double>();
  a.np = T->np.as<int8_t>();
  a.area = T->area.as<double>();
  a.flat = T->flat.as<uint8_t>();
  a.nrm = T->nrm.as<double>();
  a.group = m->group.as<int32_t>();
  a.orig = m->orig.as<int32_t>();
  a.cen = T->cen.as<double>();
  a.rad = T->rad.as<double>();
  a.cull_margin = std::ldexp(m->extent, -30);
  a.plane_dist2 = 1e-8 * m->max_coord * m->max_coord;
  a.F = m->F.as<double>();
  a.nodes = occ ? m->nodes.as<NodeD>() : nullptr;
  a.n_nodes = occ ? m->n_nodes : 0;
  a.tris = occ ? (o->geometric_soup ? m->tris_geo.as<TriD>() : m->tris_ref.as<TriD>()) : nullptr;
  a.segs = occ ? m->segs.as<SegD>() : nullptr;
  a.ray_log = ray_log;
  a.log_pm = o->ray_log_pm;
  w.n_tiles = a.n_tiles;
  if (w.mixed) {
    if (!T->tabf.ptr) {
      int rc = 0;
      if ((rc = T->tabf.alloc(s, sizeof(float) * a.nT * kComp * T->pmax * kTile))) return rc;
      cudaMemsetAsync(T->tabf.ptr, 0, T->tabf.bytes, s->stream);
      PrepF32Args pf{N, T->pmax, T->tab.as<double>(), T->tabf.as<float>(), T->np.as<int8_t>(), T->cen.as<double>()};
      const cudaError_t e = launch_prep_f32(pf, s->stream);
      if (e != cudaSuccess) return cuda_err(e, "FP32 table kernel launch");
      if (n_kernels) *n_kernels += 1;
    }
    MixedArgs& x = w.ma;
    x.N = N; x.nT = a.nT; x.n_tiles = a.n_tiles; x.pmax = a.pmax;
    x.tab = a.tab; x.tabf = T->tabf.as<float>(); x.np = a.np; x.area = a.area; x.flat = a.flat; x.nrm = a.nrm;
    x.cen = T->cen.as<double>(); x.diam = T->diam.as<double>(); x.near_factor = o->near_field_factor;
    x.rad = a.rad; x.cull_margin = a.cull_margin; x.tiny_gap = std::ldexp(m->extent, -16);
    x.group = a.group; x.orig = a.orig; x.F = a.F;
    x.nodes = a.nodes; x.n_nodes = a.n_nodes;
    x.nodesf = occ ? m->nodesf.as<NodeF>() : nullptr;
    x.tris = a.tris;
    x.trisf = occ ? (o->geometric_soup ? m->trisf_geo.as<TriF>() : m->trisf_ref.as<TriF>()) : nullptr;
    x.delta = (float)std::ldexp(m->extent, -20);
    x.ray_log = a.ray_log; x.log_pm = a.log_pm;
  }
  // Tile classes: which pairs' shadow rays may be blocked, which tiles are
  // near field (kernels_cull.cu); recomputed by every solve.
  if (!o->disable_tile_cull && N > 0 && !occ && !w.mixed) {
    // no rays and no near field: every tile is quadrature only
    w.fast_all = true;
    w.n_tiles = 0;
    w.n_fast_tiles = a.n_tiles;
    w.row_end.assign((size_t)a.nT, 0);
  } else if (!o->disable_tile_cull && N > 0 && !(w.occ_lists && !w.dim3)) {  // (curves: every tile is listed)
    int rc = 0;
    const size_t nt = (size_t)a.n_tiles;
    if (T->tcls.bytes < nt && (rc = T->tcls.alloc(s, nt))) return rc;
    if (T->tmask.bytes < nt * kTile * sizeof(uint32_t) && (rc = T->tmask.alloc(s, nt * kTile * sizeof(uint32_t))))
      return rc;
    TileClassArgs c{};
    c.N = N;
    c.nT = a.nT;
    c.n_tiles = a.n_tiles;
    c.cen = a.cen;
    c.rad = a.rad;
    c.diam = T->diam.as<double>();
    c.group = a.group;
    c.near_factor = w.mixed ? o->near_field_factor : -1.0;
    c.tiny_gap = w.mixed ? std::ldexp(m->extent, -16) : -1.0;
    c.cull_margin = a.cull_margin;
    c.occ = occ;
    c.skip_groups = true;
    c.dim3 = w.dim3;
    if (occ && w.dim3) {
      c.nodesf = m->nodesf.as<NodeF>();
      c.n_nodes = m->n_nodes;
      c.frontier = m->frontier.as<int32_t>();
      c.n_frontier = m->n_frontier;
      c.leaf_of = m->leaf_of.as<int32_t>();
      c.sat = o->geometric_soup ? m->sat_geo.as<float4>() : m->sat_ref.as<float4>();
      c.sat_em = m->sat_em;
    }
    c.cls = T->tcls.as<uint8_t>();
    c.mask = w.occ_lists ? nullptr : T->tmask.as<uint32_t>();
    if (!s->fast_ctr.ptr && (rc = s->fast_ctr.alloc(s, 256))) return rc;
    c.claim = s->fast_ctr.as<unsigned long long>() + 1;
    c.counters = s->counters.as<unsigned long long>() + 13;
    const cudaError_t e = launch_tile_class(c, s->sm_count, s->stream);
    if (e != cudaSuccess) return cuda_err(e, "tile classification launch");
    if (n_kernels) *n_kernels += 1;
    a.tcls = c.cls;
    a.tmask = T->tmask.as<uint32_t>();
    w.ma.tcls = c.cls;
    w.ma.tmask = a.tmask;
    if (!ray_log) {
      // The chunked pipeline's tiles: those with ray work (or near-field /
      // nearly coincident pairs in mixed precision), in row-major order; the
      // others go to the quadrature-only kernel (wave_fast).
      const size_t list_at = (nt + 255) & ~(size_t)255;
      if ((rc = s->h_tiles.need(list_at + sizeof(int32_t) * nt))) return rc;
      const uint8_t* cls = s->h_tiles.as<uint8_t>();
      int32_t* work = reinterpret_cast<int32_t*>(s->h_tiles.as<uint8_t>() + list_at);
      cudaError_t e2 = cudaMemcpyAsync(s->h_tiles.ptr, c.cls, nt, cudaMemcpyDeviceToHost, s->stream);
      if (e2 == cudaSuccess) e2 = cudaStreamSynchronize(s->stream);
      if (e2 != cudaSuccess) return cuda_err(e2, "tile classes");
      const uint8_t need = w.mixed ? (uint8_t)(kClsSlow | kClsNear | kClsTiny) : (uint8_t)kClsSlow;
      w.row_end.assign((size_t)a.nT, 0);
      int64_t t = 0, n_work = 0, n_slow = 0, n_wide = 0, n_long = 0;
      for (int64_t bi = 0; bi < a.nT; ++bi) {
        for (int64_t bj = bi; bj < a.nT; ++bj, ++t) {
          const uint8_t k = cls[(size_t)t];
          if (k & need) work[n_work++] = (int32_t)t;
          n_slow += k & kClsSlow ? 1 : 0;
          n_wide += k & kClsWide ? 1 : 0;
          n_long += k & kClsLong ? 1 : 0;
        }
        w.row_end[(size_t)bi] = n_work;
      }
      const int geo = o->geometric_soup ? 1 : 0;
      if (w.occ_lists && n_slow > 0 &&
          occ_by_queue(w.mixed, o->geometric_soup != 0, m->tri_margin[geo] > 0.1 * m->tri_height[geo], a.pmax, a.n_tiles,
                       (double)n_wide / n_slow, (double)n_long / n_slow)) {
        // the queue pipeline, which needs the masks: the same classes again, with them
        w.occ_lists = false;
        c.mask = T->tmask.as<uint32_t>();
        e2 = cudaMemsetAsync(c.counters, 0, 3 * sizeof(unsigned long long), s->stream);
        if (e2 == cudaSuccess) e2 = launch_tile_class(c, s->sm_count, s->stream);
        if (e2 != cudaSuccess) return cuda_err(e2, "tile classification launch");
        if (n_kernels) *n_kernels += 1;
      }
      if (n_work > 0) {
        if (T->twork.bytes < sizeof(int32_t) * n_work && (rc = T->twork.alloc(s, sizeof(int32_t) * n_work))) return rc;
        // (the buffer is next written after a synchronisation of this stream)
        e2 = cudaMemcpyAsync(T->twork.ptr, work, sizeof(int32_t) * n_work, cudaMemcpyHostToDevice, s->stream);
        if (e2 != cudaSuccess) return cuda_err(e2, "tile list upload");
      }
      a.work = T->twork.as<int32_t>();
      w.ma.work = a.work;
      w.n_tiles = n_work;
      w.n_fast_tiles = a.n_tiles - w.n_tiles;
    }
  }
  TraceArgs& ta = w.ta;
  ta.N = N; ta.pmax = a.pmax; ta.dim3 = a.dim3; ta.tab = a.tab; ta.tabf = w.ma.tabf; ta.cen = a.cen;
  ta.group = a.group; ta.orig = a.orig; ta.nodes = a.nodes; ta.nodesf = occ ? m->nodesf.as<NodeF>() : nullptr; ta.n_nodes = a.n_nodes;
  ta.tris = a.tris; ta.segs = a.segs;
  ta.trisf = (occ && w.dim3) ? (o->geometric_soup ? m->trisf_geo.as<TriF>() : m->trisf_ref.as<TriF>()) : nullptr;
  ta.delta = (float)std::ldexp(m->extent, -20);
  ta.leaf_of = (occ && w.dim3 && !o->disable_pair_lists) ? m->leaf_of.as<int32_t>() : nullptr;
  ta.sat = (occ && w.dim3) ? (o->geometric_soup ? m->sat_geo.as<float4>() : m->sat_ref.as<float4>()) : nullptr;
  ta.sat_em = m->sat_em;
  ta.frontier = (occ && w.dim3) ? m->frontier.as<int32_t>() : nullptr;
  ta.n_frontier = (occ && w.dim3) ? m->n_frontier : 0;
  ta.rad = a.rad;
  ta.cull_margin = a.cull_margin;
  ta.ray_log = a.ray_log; ta.log_pm = a.log_pm;
  if (w.occ_lists) {
    OccArgs& x = w.oa;
    x.N = N; x.nT = a.nT; x.pmax = a.pmax; x.mixed = w.mixed; x.lists = !o->disable_pair_lists;
    x.tab = a.tab; x.tabf = w.ma.tabf; x.np = a.np; x.area = a.area; x.nrm = a.nrm; x.cen = a.cen;
    x.diam = T->diam.as<double>(); x.rad = a.rad; x.flat = a.flat; x.near_factor = o->near_field_factor;
    x.cull_margin = a.cull_margin; x.sat_em = m->sat_em; x.delta = ta.delta; x.group = a.group; x.orig = a.orig;
    x.F = a.F; x.nodes = a.nodes; x.nodesf = ta.nodesf; x.n_nodes = a.n_nodes; x.tris = a.tris; x.trisf = ta.trisf;
    x.sat = ta.sat; x.frontier = ta.frontier; x.n_frontier = ta.n_frontier; x.work = a.work; x.tcls = a.tcls;
    x.tmask = T->tmask.as<uint32_t>();
    x.segs = a.segs;
    if (!w.dim3) {
      int rc = 0;
      const size_t nt = (size_t)a.n_tiles;
      if (T->tcls.bytes < nt && (rc = T->tcls.alloc(s, nt))) return rc;
      if (T->tmask.bytes < nt * kTile * sizeof(uint32_t) && (rc = T->tmask.alloc(s, nt * kTile * sizeof(uint32_t))))
        return rc;
      cudaError_t e = cudaMemsetAsync(T->tcls.ptr, 0, nt, s->stream);
      if (e == cudaSuccess) e = cudaMemsetAsync(T->tmask.ptr, 0, nt * kTile * sizeof(uint32_t), s->stream);
      if (e != cudaSuccess) return cuda_err(e, "deferred tiles");
      x.deferred = T->tcls.as<uint8_t>();
      x.tmask = T->tmask.as<uint32_t>();
      // a computed hit of the reference's segment test (src/BVH.jl:265-322: |den| >= 1e-8, parameters strictly inside
      // (1e-8, 1 - 1e-8)) lies within about 2e-7 S^3 of both segments (S bounds every length)
      const double S = 2.0 * m->extent;
      x.cand_margin = 1e-5 * S * S * S + std::ldexp(S, -16);
      x.frontier = m->frontier.as<int32_t>();
      x.n_frontier = m->n_frontier;
    }
  }
  ResolveArgs& ra = w.ra;
  ra.N = N; ra.pmax = a.pmax; ra.dim3 = a.dim3; ra.tab = a.tab; ra.tabf = w.ma.tabf; ra.cen = a.cen;
  ra.diam = T->diam.as<double>(); ra.near_factor = o->near_field_factor; ra.area = a.area; ra.orig = a.orig;
  ra.F = a.F;
  w.nodes_d = a.nodes;
  w.nodes_f = w.ma.nodesf;
  return 0;
}

int fast_groups_auto(int64_t n_tiles, int sm_count) {
  const int64_t want = (int64_t)4 * 16 * std::max(sm_count, 1);  // four tasks per resident warp (16 per SM)
  int g = 1;
  while (g < 32 && n_tiles * g < want) g = g == 8 ? 32 : 2 * g;
  return g;
}

int wave_fast(Session* s, WaveReq& w, int64_t* n_kernels) {
  if ((!w.pa.tcls && !w.fast_all) || (w.pa.ray_log && !w.fast_all) || w.pa.n_tiles == 0) return 0;
  int rc = 0;
  if (!s->fast_ctr.ptr && (rc = s->fast_ctr.alloc(s, 256))) return rc;
  w.pa.fast_groups = w.ma.fast_groups =
      w.fast_groups > 0 ? w.fast_groups : fast_groups_auto(w.n_fast_tiles > 0 ? w.n_fast_tiles : w.pa.n_tiles,
                                                           s->sm_count);
  cudaError_t e = cudaMemsetAsync(s->fast_ctr.ptr, 0, sizeof(unsigned long long), s->stream);
  if (e == cudaSuccess)
    e = launch_fast(w.mixed, w.dim3, w.occ, w.fast_qb, w.pa, w.ma, s->fast_ctr.as<unsigned long long>(),
                    s->counters.as<unsigned long long>(), s->sm_count, s->stream);
  if (e != cudaSuccess) return cuda_err(e, "quadrature-only tiles launch");
  if (n_kernels) *n_kernels += 1;
  w.pa.fast_done = true;
  w.ma.fast_done = true;
  return 0;
}

// Shared-memory shape of a launch over reqs.
WaveShape wave_shape(Session* s, WaveReq* const* reqs, int n) {
  WaveShape sh{};
  sh.mixed = reqs[0]->mixed;
  sh.dim3 = reqs[0]->dim3;
  sh.occ = reqs[0]->occ;
  for (int r = 0; r < n; ++r) sh.pmax_max = std::max(sh.pmax_max, reqs[r]->pmax);
  if (n == 1 && sh.occ && !reqs[0]->occ_lists) {
    sh.n_nodes_smem = reqs[0]->pa.n_nodes;
    sh.trace64_nodes_smem = trace_smem_bytes(false, sh.n_nodes_smem) <= (size_t)72 * 1024;
    sh.trace32_nodes_smem = sh.mixed && trace_smem_bytes(true, sh.n_nodes_smem) <= (size_t)80 * 1024;
    if (!sh.trace64_nodes_smem && !sh.trace32_nodes_smem) sh.n_nodes_smem = 0;
  }
  return sh;
}

namespace {

// Launch blocks of a chunk: the batch structs at fixed offsets (a captured
// graph keeps their addresses), then the requests' arguments as many as the
// launch has; filled in page-locked memory and copied at once.
constexpr size_t kAtGen = 0, kAtTrace = 256, kAtResolve = 512, kAtOcc = 768, kAtArgs = 1024;
static_assert(sizeof(GenBatch) <= 256 && sizeof(TraceBatch) <= 256 && sizeof(ResolveBatch) <= 256 &&
                  sizeof(OccBatch) <= 256,
              "batch structs fit their places");
constexpr size_t kBlocksBytes =
    kAtArgs + 6 * 256 + sizeof(int64_t) * (kMaxBatch + 1) +
    (sizeof(PairArgs) + sizeof(MixedArgs) + sizeof(TraceArgs) + sizeof(ResolveArgs) + sizeof(OccArgs)) * kMaxBatch;

int ensure_blocks(Session* s) {
  int rc = 0;
  if (!s->wl.ptr && (rc = s->wl.alloc(s, kBlocksBytes))) return rc;
  if ((rc = s->h_wl.need(kBlocksBytes))) return rc;
  if (!s->h_ctr) {
    const cudaError_t e =
        cudaHostAlloc(reinterpret_cast<void**>(&s->h_ctr), sizeof(unsigned long long) * (kCtrCount + 1), 0);
    if (e != cudaSuccess) return cuda_err(e, "cudaHostAlloc");
  }
  return 0;
}

template <typename T>
T* block(Session* s, size_t at) {
  return reinterpret_cast<T*>(s->wl.as<unsigned char>() + at);
}

// the chunk's counters and error flags to the host
cudaError_t copy_counters(Session* s) {
  const cudaError_t e = cudaMemcpyAsync(s->h_ctr, s->wq_ctr.ptr, sizeof(unsigned long long) * kCtrCount,
                                        cudaMemcpyDeviceToHost, s->stream);
  if (e != cudaSuccess) return e;
  return cudaMemcpyAsync(s->h_ctr + kCtrCount, s->err.ptr, sizeof(int), cudaMemcpyDeviceToHost, s->stream);
}

uint64_t shape_key(const WaveShape& sh) {
  return (uint64_t)sh.mixed | ((uint64_t)sh.dim3 << 1) | ((uint64_t)sh.occ << 2) |
         ((uint64_t)sh.trace64_nodes_smem << 4) | ((uint64_t)sh.trace32_nodes_smem << 5) |
         ((uint64_t)sh.pmax_max << 8) | ((uint64_t)sh.gen_bps << 16) | ((uint64_t)sh.trace_bps << 20) |
         ((uint64_t)(sh.n_nodes_smem & 0xffffff) << 24) | ((uint64_t)sh.occ_grid << 48);
}

// The chunk's device work: counters reset, generation, traversal(s), resolve
// and the counters' copy to pinned host memory (with timing events when
// launched eagerly).
cudaError_t enqueue_chunk(Session* s, const WaveShape& sh, bool events) {
  cudaStream_t st = s->stream;
  cudaError_t e = cudaMemsetAsync(s->wq_ctr.ptr, 0, sizeof(unsigned long long) * kCtrCount, st);
  if (e != cudaSuccess) return e;
  if (events) cudaEventRecord(s->ev[0], st);
  if (sh.occ_grid > 0 && !sh.dim3) {
    if ((e = launch_occ2d(sh.pmax_max, block<OccBatch>(s, kAtOcc), s->sm_count, st)) != cudaSuccess) return e;
    for (int k = 1; events && k <= 3; ++k) cudaEventRecord(s->ev[k], st);
    return copy_counters(s);
  }
  if (sh.occ_grid > 0) {
    if ((e = launch_occ(sh.mixed, sh.pmax_max, block<OccBatch>(s, kAtOcc), sh.occ_grid, s->sm_count, st,
                        events ? &s->ev[1] : nullptr)) != cudaSuccess)
      return e;
    return copy_counters(s);
  }
  if ((e = launch_gen(sh, block<GenBatch>(s, kAtGen), s->sm_count, st)) != cudaSuccess) return e;
  if (events) cudaEventRecord(s->ev[1], st);
  if (sh.occ) {
    // the pair lists count as traversal time (the first traversal phase)
    const bool lists = sh.dim3;
    auto plist = [&]() -> cudaError_t {
      if (events) cudaEventRecord(s->ev[5], st);
      const cudaError_t el = launch_plist(block<TraceBatch>(s, kAtTrace), s->sm_count, st);
      if (events) cudaEventRecord(s->ev[6], st);
      return el;
    };
    if (lists && sh.mixed && (e = plist()) != cudaSuccess) return e;
    if (sh.mixed && (e = launch_trace(sh, block<TraceBatch>(s, kAtTrace), true, s->sm_count, st)) != cudaSuccess) return e;
    if (events) cudaEventRecord(s->ev[2], st);
    if (lists && !sh.mixed && (e = plist()) != cudaSuccess) return e;
    if ((e = launch_trace(sh, block<TraceBatch>(s, kAtTrace), false, s->sm_count, st)) != cudaSuccess) return e;
    if (events) cudaEventRecord(s->ev[3], st);
    if ((e = launch_resolve(sh, block<ResolveBatch>(s, kAtResolve), s->sm_count, st)) != cudaSuccess) return e;
    if (events) cudaEventRecord(s->ev[4], st);
  }
  return copy_counters(s);
}

}  // namespace

// The pairs of curves that the chunk's kernel deferred (tiles [t0, t0 + n) of a
// request), in the queue pipeline.
static int deferred_pairs(Session* s, const WaveReq& req, int64_t t0, int64_t n, bool use_graph, ChunkInfo* info) {
  int rc = 0;
  Tables* T = req.tables;
  const size_t list_at = ((size_t)n + 255) & ~(size_t)255;
  if ((rc = s->h_tiles.need(list_at + sizeof(int32_t) * n))) return rc;
  const uint8_t* cls = s->h_tiles.as<uint8_t>();
  int32_t* work = reinterpret_cast<int32_t*>(s->h_tiles.as<uint8_t>() + list_at);
  cudaError_t e = cudaMemcpyAsync(s->h_tiles.ptr, T->tcls.as<uint8_t>() + t0, (size_t)n, cudaMemcpyDeviceToHost, s->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
  if (e != cudaSuccess) return cuda_err(e, "deferred tiles");
  int64_t n_work = 0;
  for (int64_t t = 0; t < n; ++t)
    if (cls[t]) work[n_work++] = (int32_t)(t0 + t);
  if (n_work == 0) return 0;
  if (T->twork.bytes < sizeof(int32_t) * n_work && (rc = T->twork.alloc(s, sizeof(int32_t) * n_work))) return rc;
  if ((e = cudaMemcpyAsync(T->twork.ptr, work, sizeof(int32_t) * n_work, cudaMemcpyHostToDevice, s->stream)) != cudaSuccess)
    return cuda_err(e, "deferred tile list upload");
  WaveReq d = req;
  d.occ_lists = false;
  d.pa.tcls = T->tcls.as<uint8_t>();
  d.pa.tmask = T->tmask.as<uint32_t>();
  d.pa.work = T->twork.as<int32_t>();
  d.pa.only_masked = true;
  d.n_tiles = n_work;
  d.claimed = 0;
  WaveReq* one = &d;
  while (!d.done()) {
    const int64_t before = d.claimed;
    ChunkInfo ci;
    if ((rc = wave_chunk(s, &one, 1, use_graph, info ? &ci : nullptr))) return rc;
    if (d.claimed == before) return no_progress(s);
    if (info) {
      info->ms_gen += ci.ms_gen;
      info->ms_trace += ci.ms_trace;
      info->ms_resolve += ci.ms_resolve;
      info->rays_traced += ci.rays_traced;
      info->kernels += ci.kernels;
    }
  }
  return 0;
}

int wave_chunk(Session* s, WaveReq* const* reqs_in, int n_in, bool use_graph, ChunkInfo* info, int gen_bps,
               int trace_bps, double pp_budget, const std::function<void()>* on_launched) {
  if (n_in < 1 || n_in > kMaxBatch) return set_err(RVF_EINVAL, "batch of %d requests (1..%d)", n_in, kMaxBatch);
  int rc = 0;
  if ((rc = ensure_blocks(s))) return rc;
  // tiles offered to this launch, in request order: all that remain, or as
  // many as the point-pair budget allows (the oldest requests first)
  std::vector<WaveReq*> reqs;
  std::vector<int64_t> offer;
  double left = pp_budget > 0 ? pp_budget : 1e300;
  for (int r = 0; r < n_in && left > 0; ++r) {
    const int64_t rem = reqs_in[r]->n_tiles - reqs_in[r]->claimed;
    // one launch holds requests of one kernel: those of the oldest one's
    if (rem <= 0 || (!reqs.empty() && reqs_in[r]->occ_lists != reqs[0]->occ_lists)) continue;
    const double per = (double)kTile * kTile * reqs_in[r]->pmax * reqs_in[r]->pmax;
    const int64_t take = (left >= per * (double)rem) ? rem : std::max<int64_t>(1, (int64_t)std::ceil(left / per));
    reqs.push_back(reqs_in[r]);
    offer.push_back(take);
    left -= per * (double)take;
  }
  if (reqs.empty()) return RVF_OK;
  const int n = (int)reqs.size();
  WaveShape sh = wave_shape(s, reqs.data(), n);
  const bool fused = reqs[0]->occ_lists;
  sh.gen_bps = fused ? 0 : gen_bps;
  sh.trace_bps = fused ? 0 : trace_bps;
  std::vector<int64_t> base(n + 1, 0);
  for (int r = 0; r < n; ++r) base[r + 1] = base[r] + offer[r];
  const bool queues = sh.occ && !fused;
  WaveQ q{};
  OccBatch ob{};
  if (fused && !sh.dim3) {
    if (!s->wq_ctr.ptr && (rc = s->wq_ctr.alloc(s, sizeof(unsigned long long) * kCtrCount))) return rc;
    ob.q.ctr = s->wq_ctr.as<unsigned long long>();
    sh.occ_grid = 1;
  } else if (fused) {
    if ((rc = ensure_occ(s, base[n], ob.q, sh.occ_grid))) return rc;
  } else if ((rc = ensure_wave(s, sh.mixed && queues, queues, queues && sh.dim3, sh.pmax_max, base[n], q))) {
    return rc;
  }
  size_t at = kAtArgs;
  unsigned char* hw = s->h_wl.as<unsigned char>();
  auto place = [&](auto fill, auto* kind) {  // n arguments of one kind; their device address
    using T = std::remove_pointer_t<decltype(kind)>;
    T* h = reinterpret_cast<T*>(hw + at);
    for (int r = 0; r < n; ++r) fill(h[r] = T{}, *reqs[r]);
    T* d = block<T>(s, at);
    at = (at + sizeof(T) * n + 255) & ~(size_t)255;
    return d;
  };
  GenBatch g{};
  std::memcpy(hw + at, base.data(), sizeof(int64_t) * (n + 1));
  g.tile_base = block<int64_t>(s, at);
  at = (at + sizeof(int64_t) * (n + 1) + 255) & ~(size_t)255;
  g.reqs = place([&](PairArgs& x, WaveReq& w) { x = w.pa; x.tile0 = w.claimed; x.q = q; }, (PairArgs*)nullptr);
  if (sh.mixed)
    g.mreqs = place([&](MixedArgs& x, WaveReq& w) { x = w.ma; x.tile0 = w.claimed; x.q = q; }, (MixedArgs*)nullptr);
  g.n_req = n;
  g.pmax_max = sh.pmax_max;
  g.total_tiles = base[n];
  g.claim_retries = reqs[0]->claim_retries;
  for (int r = 1; r < n; ++r) g.claim_retries = std::min(g.claim_retries, reqs[r]->claim_retries);
  g.q = q;
  g.counters = s->counters.as<unsigned long long>();
  g.err = s->err.as<int>();
  if (fused) {
    ob.reqs = place([&](OccArgs& x, WaveReq& w) { x = w.oa; x.tile0 = w.claimed; }, (OccArgs*)nullptr);
    ob.preqs = g.reqs;
    ob.mreqs = g.mreqs;
    ob.tile_base = g.tile_base;
    ob.n_req = n;
    ob.pmax_max = sh.pmax_max;
    ob.total_tiles = base[n];
    // a tile is split into parts only when the queue holds every tile at once: a chunk then ends between tiles
    const bool all = !sh.dim3 || (base[n] + sh.occ_grid) * kTile * kTile <= ob.q.scap;
    ob.groups = all ? occ_groups(base[n], s->sm_count) : 1;
    ob.rest_parts = base[n] * 8 >= (int64_t)64 * s->sm_count ? 8 : 32;
    ob.counters = g.counters;
    std::memcpy(hw + kAtOcc, &ob, sizeof ob);
  } else {
    TraceBatch tb{};
    tb.reqs = place([&](TraceArgs& x, WaveReq& w) { x = w.ta; x.q = q; }, (TraceArgs*)nullptr);
    tb.n_req = n;
    tb.nodes64_in_smem = sh.trace64_nodes_smem;
    tb.nodes32_in_smem = sh.trace32_nodes_smem;
    tb.smem_nodes64 = reqs[0]->nodes_d;
    tb.smem_nodes32 = reqs[0]->nodes_f;
    tb.n_nodes_smem = sh.n_nodes_smem;
    tb.q = q;
    tb.counters = g.counters;
    ResolveBatch rb{};
    rb.reqs = place([&](ResolveArgs& x, WaveReq& w) { x = w.ra; }, (ResolveArgs*)nullptr);
    rb.n_req = n;
    rb.q = q;
    std::memcpy(hw + kAtGen, &g, sizeof g);
    std::memcpy(hw + kAtTrace, &tb, sizeof tb);
    std::memcpy(hw + kAtResolve, &rb, sizeof rb);
  }
  cudaStream_t st = s->stream;
  cudaError_t e = cudaMemcpyAsync(s->wl.ptr, hw, at, cudaMemcpyHostToDevice, st);
  if (e != cudaSuccess) return cuda_err(e, "launch block upload");
  bool replayed = false;
  if (use_graph) {
    const uint64_t key = shape_key(sh);
    auto it = s->graphs.find(key);
    if (it == s->graphs.end()) {
      cudaGraph_t graph = nullptr;
      cudaGraphExec_t exec = nullptr;
      if (cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
        const cudaError_t e1 = enqueue_chunk(s, sh, false);
        const cudaError_t e2 = cudaStreamEndCapture(st, &graph);
        if (e1 == cudaSuccess && e2 == cudaSuccess && graph && cudaGraphInstantiate(&exec, graph, 0) == cudaSuccess)
          it = s->graphs.emplace(key, exec).first;
        if (graph) cudaGraphDestroy(graph);
        cudaGetLastError();  // a refused capture falls back to eager launches
      }
    }
    if (it != s->graphs.end()) {
      if ((e = cudaGraphLaunch(it->second, st)) != cudaSuccess) return cuda_err(e, "graph launch");
      replayed = true;
    }
  }
  if (!replayed && (e = enqueue_chunk(s, sh, info != nullptr)) != cudaSuccess) return cuda_err(e, "pair pipeline launch");
  if (on_launched) (*on_launched)();
  if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return cuda_err(e, "pair pipeline");
  if (info) {
    *info = ChunkInfo{};
    info->graph = replayed;
    info->kernels = (fused && sh.dim3 ? 4 : 1) + (queues ? (sh.mixed ? 3 : 2) + (sh.dim3 ? 1 : 0) : 0);
    if (!replayed) {
      float t = 0.f;
      cudaEventElapsedTime(&t, s->ev[0], s->ev[1]);
      if (fused) {
        float tr = 0.f, tp = 0.f;
        cudaEventElapsedTime(&tr, s->ev[1], s->ev[2]);
        cudaEventElapsedTime(&tp, s->ev[2], s->ev[3]);
        info->ms_gen = tr;
        info->ms_trace = t + tp;
        info->ms_lists = sh.dim3 ? t : 0.0;
      } else {
        info->ms_gen = t;
      }
      if (queues) {
        float t12 = 0.f, t23 = 0.f, t34 = 0.f;
        cudaEventElapsedTime(&t12, s->ev[1], s->ev[2]);
        cudaEventElapsedTime(&t23, s->ev[2], s->ev[3]);
        cudaEventElapsedTime(&t34, s->ev[3], s->ev[4]);
        info->ms_trace = sh.mixed ? t12 : t23;
        info->ms_trace_fp64 = sh.mixed ? t23 : 0.0;
        info->ms_resolve = t34;
        if (sh.dim3) {
          float tl = 0.f;
          cudaEventElapsedTime(&tl, s->ev[5], s->ev[6]);
          info->ms_lists = tl;
        }
      }
    }
    info->rays_traced = (int64_t)(sh.mixed && !fused ? s->h_ctr[kCtrRec32] : s->h_ctr[kCtrRec64]);
  }
  // tiles are claimed in launch order: request r got min(claimed - base[r], its remaining tiles)
  const int64_t got = (int64_t)s->h_ctr[kCtrTile] / (fused ? ob.groups : 1);
  const bool deferred = fused && !sh.dim3 && s->h_ctr[kCtrWalk] > 0;
  for (int r = 0; r < n; ++r) {
    const int64_t take = std::max<int64_t>(0, std::min<int64_t>(got - base[r], base[r + 1] - base[r]));
    if (deferred && take > 0 && (rc = deferred_pairs(s, *reqs[r], reqs[r]->claimed, take, use_graph, info))) return rc;
    reqs[r]->claimed += take;
  }
  return 0;
}

}  // namespace rvf
