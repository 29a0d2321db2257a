// packet.cu — relation predicates refined inside a traversal that 32
// neighbouring probe rows share.
//
// The candidate pairs' path (lbvh.cu, refine*.cu) writes every pair of
// overlapping boxes, orders the pairs so that a warp works on one build
// geometry, refines one pair per lane and compacts.  It is bound by
// divergence (6 of 32 lanes per instruction on 2M buildings x 50k zones) and,
// for points, by the passes over the pairs.  Here a warp takes 32 probe rows
// that are neighbours in Morton order, walks the tree once for all of them,
// and meets each build row with all its lanes at once: what belongs to the
// build row is loaded once, and
//   1. the box of all 32 probes is looked up in the build ring's cell grid;
//      clean cells of one status answer for every lane;
//   2. else the edges listed in those cells are taken one per lane, and the
//      few that cut the box are shown to every lane, which tests its own
//      point (point in ring) or box (ring_isolation's test, with the side of
//      its first vertex) against them;
//   3. pairs of rings that come near each other, and rows the packet does
//      not know (multipolygons, polygons with holes on the probe side), go to
//      a queue that k_packet_open takes with one lane per pair.
// A packet keeps one record per build row, (build row, lane mask): no
// candidate pairs, permutation, flags or compaction.  k_packet_scatter turns
// the masks into pairs; records are in traversal order, so every probe row's
// pairs come in the order of the candidate pairs' path.
//
// 2M buildings x 50k zones, ST_Intersects: 40.5 -> 18.1 ms a step (refine 28.5,
// traversal 3.6, ordering and compaction of 132M pairs 4.9 before; k_packet
// 9.1, k_packet_open 6.9, k_packet_scatter 0.4 now); 2M points x 50k zones:
// 15.7 -> 5.6 ms; 300k buildings in 20k holed zones: 17.4 -> 3.8 ms.  k_packet
// is bound by its instructions (some 1,000 per packet and build row): for
// polygons from a loop body larger than the instruction cache (a quarter of a
// warp's cycles wait for instructions, as many for loads, at 24 warps per SM;
// half of the issue slots are used), for points 70 % of the slots are used.
// 64 / 80 registers measured 10 % better than 80 / 96 and 128.
#include "packet.cuh"

#include <algorithm>

#include "refine_eval.cuh"

namespace spj {
namespace {

using namespace pred;

constexpr int kPacketThreads = 128;
constexpr unsigned kAll = 0xffffffffu;
// flags of a queued pair above its lane
constexpr uint32_t kOpenNear = 32;  // two single rings, an edge near the probe's box

constexpr uint32_t kOpenIn = 64;    // (with kOpenNear) its first vertex is strictly inside ...
constexpr uint32_t kOpenOut = 128;  // ... or strictly outside the build ring

// A lane's ring against a uniform ring: strictly outside or inside with no
// edge near, or near an edge.
constexpr int kIsOut = 0, kIsIn = 1, kIsNear = 2;

__device__ __forceinline__ float warp_min(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(kAll, v, o));
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(kAll, v, o));
  return v;
}

// Status of the box U (f32 bounds of points' RN32 copies or of exact boxes) in
// ring r's cell grid: 1 / 2 when the cells that hold it (at most 4 x 4) are all
// clean and inside / outside, else 0.
__device__ __forceinline__ int box_grid_status(const GeomsView& G, uint32_t r, float4 U) {
  if (G.grid_meta == nullptr) return 0;
  const uint4 m = G.grid_meta[r];
  if (m.y == 0) return 0;
  CellRange c;
  const int found = grid_cells(G.grid_rect[r], (int)m.y, U, c);
  if (found <= 0) return found == 0 ? 2 : 0;
  if (c.i1 - c.i0 > 3 || c.j1 - c.j0 > 3) return 0;
  const uint32_t* cell = G.grid_cell + m.x;
  const uint32_t st = cell_state(cell[(uint32_t)c.j0 * m.y + (uint32_t)c.i0]);
  if (st == kCellUnknown || st >= kCellMixed || (st == kCellIn && c.past)) return 0;
  for (int j = c.j0; j <= c.j1; j++)
    for (int i = c.i0; i <= c.i1; i++)
      if (cell_state(cell[(uint32_t)j * m.y + (uint32_t)i]) != st) return 0;
  return (int)st;
}

__device__ __noinline__ bool lone_pip(const GeomsView& G, uint32_t r, double2 p, float2 p32,
                                      bool aoe, uint32_t& esc) {
  return ring_pip_fast(G, r, p, p32, aoe, esc).hit;
}
__device__ __noinline__ int lone_isolation(const GeomsView& Gr, uint32_t rr, const GeomsView& Go,
                                           uint32_t ro, uint32_t& esc) {
  return ring_isolation<true>(Gr, rr, Go, ro, esc);
}

// The functions below are called by all 32 lanes (those without work pass
// on = false): their loops run as long as any lane's and meet at the end of
// each step.  With loops of each lane's own length the lanes drift apart and
// stay apart (k_packet_open then ran 1.3 of 32 lanes at a time).

__device__ __forceinline__ bool apart32(float4 e, float x0, float y0, float x1, float y1) {
  return fmax0f(e.x, e.z) < x0 || fmin0f(e.x, e.z) > x1 || fmax0f(e.y, e.w) < y0 ||
         fmin0f(e.y, e.w) > y1;
}

constexpr int kLaneCells = 6;  // cells per axis that a lane's box may span

// A lane's single-ring probe polygon.
struct LaneRing {
  uint32_t ring;
  float4 box;   // RN32 rect
  float2 v032;  // first vertex
};

// Where the lanes' points p (RN32 copies) and boxes lie in ring r, from its
// grid: side 1 the point is strictly inside, 0 strictly outside, -1 not
// decided; near (kBox): an edge comes near the lane's box (ring_isolation's
// test; when none does, the whole box lies on its point's side).  Returns false
// when the grid does not answer.
//
// The lanes look together at the cells that hold H, a box of all their points
// and boxes: at most 8 x 4, listing at most 32 edges.  A lane takes one listed
// edge and drops it when another cell listed it too, or when all of H lies on
// one side of it.  The few edges left are shown to all lanes: an edge comes
// near a box that it does not leave on one side; and a point lies where the
// centre c of a cell does (known) unless an odd number of edges crosses the
// segment between them, which stays in the cells.  Every edge that is not
// strictly separated from that segment needs decided sides of p and c, and
// when these differ, its ends decided sides of the segment.  A decided answer
// is the exact one, and tg's: an edge that is not listed in the cells, was
// dropped or is strictly separated leaves the point clear of it (comparisons,
// or a decided side of all of H), and a decided side is some 2^24 times
// clearer than the rounding of tg's slope test (the argument of ring_isolation).
// The lane that took the edge bounds the error of every orientation that the
// other lanes evaluate with it, so that each costs them a few instructions.
template <bool kBox>
__device__ __forceinline__ bool shared_cells(const GeomsView& G, uint32_t r, bool on, float2 p,
                                             float4 box, float4 U, int lane, bool& near,
                                             int& side) {
  const uint4 m = G.grid_meta[r];
  const float4 q = G.grid_rect[r];
  CellRange c;
  near = false;
  const int found = grid_cells(q, (int)m.y, U, c);
  side = found == 0 ? 0 : -1;  // (all past the grid: outside)
  if (found <= 0) return found == 0;
  const int nx = c.i1 - c.i0 + 1, ny = c.j1 - c.j0 + 1;
  if (nx > 8 || ny > 4) return false;
  // lane t: cell (t & 7, t >> 3)
  const bool cell = (lane & 7) < nx && (lane >> 3) < ny;
  const uint32_t w =
      cell ? G.grid_cell[m.x + (uint32_t)(c.j0 + (lane >> 3)) * m.y + (uint32_t)(c.i0 + (lane & 7))]
           : kCellIn;
  if (__any_sync(kAll, cell_state(w) == kCellUnknown)) return false;
  const uint32_t n = cell && cell_state(w) >= kCellMixed ? cell_count(w) : 0u;
  const uint32_t inc = warp_inclusive_scan(n);
  const uint32_t total = __shfl_sync(kAll, inc, 31);
  if (total > 32u) return false;
  const int ref = (ny >> 1) * 8 + (nx >> 1);
  const uint32_t rs = cell_state(__shfl_sync(kAll, w, ref));
  const float2 ctr = grid_centre(q, c.i0 + (nx >> 1), c.j0 + (ny >> 1));
  // this lane's listed edge
  uint32_t at = 0;
  unsigned holders = __ballot_sync(kAll, n > 0);
  while (holders) {
    const int h = __ffs(holders) - 1;
    holders &= holders - 1;
    const uint32_t end = __shfl_sync(kAll, inc, h), wh = __shfl_sync(kAll, w, h);
    const uint32_t begin = end - cell_count(wh);
    if ((uint32_t)lane >= begin && (uint32_t)lane < end) at = cell_first(wh) + lane - begin;
  }
  float4 e = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  uint32_t id = 0x10000u + lane;
  if ((uint32_t)lane < total) {
    e = G.grid_seg[m.z + at];
    id = G.grid_edge_id[m.z + at];
  }
  const unsigned same = __match_any_sync(kAll, id);
  const float4 H = make_float4(fminf(U.x, ctr.x), fminf(U.y, ctr.y), fmaxf(U.z, ctr.x),
                               fmaxf(U.w, ctr.y));
  const float2 ma = make_float2(e.x, e.y), mb = make_float2(e.z, e.w);
  // bound of the edge's orientation of any point of H, and of the ends'
  // orientations to a segment from a point of H to c
  const float E1 = box_orient_bound(ma, mb, H);
  const float2 mo = box_orient(ma, mb, H);
  const bool keep = (uint32_t)lane < total && __ffs(same) - 1 == lane &&
                    !apart32(e, H.x, H.y, H.z, H.w) && !(mo.x > E1 || mo.y < -E1);
  unsigned todo = __ballot_sync(kAll, keep);
  bool in = rs == kCellIn || rs == kCellMixedIn, ok = true;
  if (todo) {
    const float dx = fmaxf(__fsub_ru(ctr.x, H.x), __fsub_ru(H.z, ctr.x));
    const float dy = fmaxf(__fsub_ru(ctr.y, H.y), __fsub_ru(H.w, ctr.y));
    const float px = fmaxf(fabsf(H.x), fabsf(H.z)), py = fmaxf(fabsf(H.y), fabsf(H.w));
    const float ex = fmaxf(__fsub_ru(fmaxf(H.z, fmaxf(ma.x, mb.x)), fminf(H.x, fminf(ma.x, mb.x))),
                           0.0f);
    const float ey = fmaxf(__fsub_ru(fmaxf(H.w, fmaxf(ma.y, mb.y)), fminf(H.y, fminf(ma.y, mb.y))),
                           0.0f);
    const float t1 = __fmul_ru(dx, ey), t2 = __fmul_ru(dy, ex);
    const float E2 = orient_bound(
        dx, dy, ex, ey, __fadd_ru(px, fabsf(ctr.x)), __fadd_ru(py, fabsf(ctr.y)),
        __fadd_ru(px, fmaxf(fabsf(ma.x), fabsf(mb.x))), __fadd_ru(py, fmaxf(fabsf(ma.y), fabsf(mb.y))),
        t1, t2, __fadd_ru(t1, t2));
    const float mc = __fsub_rn(__fmul_rn(__fsub_rn(mb.x, ma.x), __fsub_rn(ctr.y, ma.y)),
                               __fmul_rn(__fsub_rn(mb.y, ma.y), __fsub_rn(ctr.x, ma.x)));
    const float x0 = fmin0f(p.x, ctr.x), x1 = fmax0f(p.x, ctr.x);
    const float y0 = fmin0f(p.y, ctr.y), y1 = fmax0f(p.y, ctr.y);
    const float sx = __fsub_rn(ctr.x, p.x), sy = __fsub_rn(ctr.y, p.y);
    while (todo) {
      const int s = __ffs(todo) - 1;
      todo &= todo - 1;
      const float4 x = make_float4(__shfl_sync(kAll, e.x, s), __shfl_sync(kAll, e.y, s),
                                   __shfl_sync(kAll, e.z, s), __shfl_sync(kAll, e.w, s));
      const float F1 = __shfl_sync(kAll, E1, s), F2 = __shfl_sync(kAll, E2, s);
      const float oc = __shfl_sync(kAll, mc, s);
      const float2 a = make_float2(x.x, x.y), b = make_float2(x.z, x.w);
      if (kBox && !apart32(x, box.x, box.y, box.z, box.w)) {
        const float2 o = box_orient(a, b, box);
        if (!(o.x > F1 || o.y < -F1)) near = true;
      }
      if (!apart32(x, x0, y0, x1, y1)) {
        const float o = __fsub_rn(__fmul_rn(__fsub_rn(b.x, a.x), __fsub_rn(p.y, a.y)),
                                  __fmul_rn(__fsub_rn(b.y, a.y), __fsub_rn(p.x, a.x)));
        // sides of the line through p and c
        const float oa = __fsub_rn(__fmul_rn(sx, __fsub_rn(a.y, p.y)), __fmul_rn(sy, __fsub_rn(a.x, p.x)));
        const float ob = __fsub_rn(__fmul_rn(sx, __fsub_rn(b.y, p.y)), __fmul_rn(sy, __fsub_rn(b.x, p.x)));
        const bool sides = fabsf(o) > F1 && fabsf(oc) > F1;
        if (!sides) ok = false;
        else if ((o > 0.0f) != (oc > 0.0f)) {
          if (!(fabsf(oa) > F2 && fabsf(ob) > F2)) ok = false;
          else if ((oa > 0.0f) != (ob > 0.0f)) in = !in;
        }
      }
    }
  }
  side = ok ? (in ? 1 : 0) : -1;
  return true;
}

// The same with each lane's own cells (at most 6 x 6 that hold its box), for
// packets whose common box holds too many: a cell lists few edges, but every
// lane loads and bounds its own.  A point is compared with the centre of the
// cell that it lies in.
template <bool kBox>
__device__ __forceinline__ bool lane_cells(const GeomsView& G, uint32_t r, bool on, float2 p,
                                           float4 box, bool& near, int& side) {
  const uint4 m = G.grid_meta[r];
  const float4 q = G.grid_rect[r];
  CellRange c{0, -1, 0, -1, false};
  const int found = on ? grid_cells(q, (int)m.y, box, c) : -1;
  const int nx = c.i1 - c.i0 + 1, ny = c.j1 - c.j0 + 1;
  const bool act = found > 0 && nx <= kLaneCells && ny <= kLaneCells;
  const int cells = act ? nx * ny : 0;
  const int most = __reduce_max_sync(kAll, cells);
  bool unknown = false;
  int clean = 0;  // state of a clean cell
  near = false;
  side = found == 0 ? 0 : -1;
  int i = c.i0, j = c.j0;
  for (int t = 0; t < most; t++) {
    uint32_t w = kCellIn;
    bool vc = false;  // the point lies strictly inside this cell
    if (t < cells) {
      w = G.grid_cell[m.x + (uint32_t)j * m.y + (uint32_t)i];
      if (cell_state(w) == kCellUnknown) unknown = true;
      else if (cell_state(w) < kCellMixed) clean = (int)cell_state(w);
      vc = p.x > grid_edge(q.x, q.z, i) && p.x < grid_edge(q.x, q.z, i + 1) &&
           p.y > grid_edge(q.y, q.w, j) && p.y < grid_edge(q.y, q.w, j + 1);
    }
    const uint32_t s = cell_state(w);
    const float2 ctr = grid_centre(q, i, j);
    const float x0 = fmin0f(p.x, ctr.x), x1 = fmax0f(p.x, ctr.x);
    const float y0 = fmin0f(p.y, ctr.y), y1 = fmax0f(p.y, ctr.y);
    const int n = s >= kCellMixed && (vc || (kBox && !near)) ? (int)cell_count(w) : 0;
    const int mostn = __reduce_max_sync(kAll, n);
    const float4* seg = G.grid_seg + m.z + cell_first(w);
    bool in = s == kCellIn || s == kCellMixedIn, ok = true;
    for (int k = 0; k < mostn; k++) {
      if (k < n) {
        const float4 e = seg[k];
        const float2 a = make_float2(e.x, e.y), b = make_float2(e.z, e.w);
        if (kBox && !near && !apart32(e, box.x, box.y, box.z, box.w))
          near = box_side32(a, b, box) == 0;
        if (vc && !apart32(e, x0, y0, x1, y1)) {
          const int o = orient32(a, b, p);  // (the centre is strictly left)
          if (o <= 0) {
            const int oa = orient32(p, ctr, a), ob = orient32(p, ctr, b);
            if (o == 0 || oa == 0 || ob == 0) ok = false;
            else if (oa != ob) in = !in;
          }
        }
      }
      __syncwarp();
    }
    if (vc && s != kCellUnknown && ok) side = in ? 1 : 0;
    if (++i > c.i1) {
      i = c.i0;
      j++;
    }
  }
  if (act && side < 0 &&
      (p.x < q.x || p.y < q.y || p.x > grid_edge(q.x, q.z, (int)m.y) ||
       p.y > grid_edge(q.y, q.w, (int)m.y)))
    side = 0;  // past the grid
  if (act && !unknown && !near && side < 0 && clean != 0) side = clean == 1;
  return found == 0 || (act && !unknown);
}

// ring_pip of the lanes' points (all in U) against ring r: the cells of its
// grid, else (not decided there, or no grid) the band scan.
__device__ __forceinline__ bool packet_pip(const GeomsView& G, uint32_t r, bool on, double2 p,
                                           float2 p32, float4 U, int lane, bool aoe,
                                           uint32_t& esc) {
  int side = -1;
  bool near;
  if (G.grid_meta != nullptr && G.grid_meta[r].y != 0 &&
      !shared_cells<false>(G, r, on, p32, U, U, lane, near, side))
    lane_cells<false>(G, r, on, p32, make_float4(p32.x, p32.y, p32.x, p32.y), near, side);
  bool hit = side == 1;
  if (__any_sync(kAll, on && side < 0)) {
    if (on && side < 0) hit = lone_pip(G, r, p, p32, aoe, esc);
    __syncwarp();
  }
  return on && hit;
}

// ring_isolation of the lanes' rings (all in U) against ring r: kIsOut / kIsIn
// when no edge comes near the lane's box, else kIsNear.  v_in: 1 / 0 the first
// vertex is strictly inside / outside, -1 not known; set for near lanes too.
__device__ __forceinline__ int packet_isolation(const GeomsView& G, uint32_t r, bool on,
                                                const LaneRing& o, const GeomsView& P, float4 U,
                                                int lane, int& v_in, uint32_t& esc) {
  int iso = -1;
  v_in = -1;
  bool near = false;
  if (G.grid_meta != nullptr && G.grid_meta[r].y != 0 &&
      (shared_cells<true>(G, r, on, o.v032, o.box, U, lane, near, v_in) ||
       lane_cells<true>(G, r, on, o.v032, o.box, near, v_in)))
    iso = near ? kIsNear : v_in;
  if (__any_sync(kAll, on && iso < 0)) {
    if (on && iso < 0) {
      const int b = lone_isolation(G, r, P, o.ring, esc);
      iso = b == 1 ? kIsIn : (b == 0 ? kIsOut : kIsNear);
      if (iso != kIsNear) v_in = iso;
    }
    __syncwarp();
  }
  return iso;
}

// Result of a pair of polygons whose build rings no edge of comes near the
// probe's box, the probe lying strictly inside (in) or outside the polygon.
__device__ __forceinline__ bool isolated_result(int predicate, bool in) {
  switch (predicate) {
    case kIntersects:
    case kContains:
    case kCovers:
      return in;
    case kDisjoint:
      return !in;
    default:  // the probe neither holds the build row nor meets its boundary
      return false;
  }
}

// Packets: runs of up to 32 consecutive rows of the Morton order.  A run whose
// box is wide would meet many more build rows than its rows do (a cluster's
// thin tail, a gap of the order) and one warp would still be at it when the
// others are done, so it is cut in halves, down to one row: an aligned group of
// rows is split where its box, widened by the mean build box, is over
// kPacketGrowth times one row's and may meet over kPacketRows build rows (by
// the density that the caller gives; with fewer, splitting costs more than it
// saves).  (8,000 buildings, whose neighbours lie far apart: 1,667 us with
// packets of 4 rows and up, 1,242 with single rows; 2M alike.)
constexpr float kPacketRows = 64.0f, kPacketGrowth = 4.0f;
__global__ void __launch_bounds__(256)
    k_packets(LbvhView t, const float4* __restrict__ box, const uint32_t* __restrict__ order,
              uint32_t n, float mean_w, float mean_h, float per_area,
              uint2* __restrict__ packets, unsigned long long* __restrict__ ctrl) {
  const int lane = threadIdx.x & 31;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t g = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; g * 32 < n; g += nw) {
    const uint64_t j = g * 32 + lane;
    const uint32_t pi = j < n ? order[j] : 0u;
    const float q = __int_as_float(0x7fc00000);
    float4 b = make_float4(q, q, q, q);
    if (j < n && pi < n) b = box[pi];
    const bool live = b.x <= b.z && b.y <= b.w;
    float x0 = live ? b.x : INFINITY, y0 = live ? b.y : INFINITY;
    float x1 = live ? b.z : -INFINITY, y1 = live ? b.w : -INFINITY;
    float own = live ? (b.z - b.x + mean_w) * (b.w - b.y + mean_h) : 0.0f;
    int size = 1;  // of the group taken so far
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      x0 = fminf(x0, __shfl_xor_sync(kAll, x0, o));
      y0 = fminf(y0, __shfl_xor_sync(kAll, y0, o));
      x1 = fmaxf(x1, __shfl_xor_sync(kAll, x1, o));
      y1 = fmaxf(y1, __shfl_xor_sync(kAll, y1, o));
      own = fmaxf(own, __shfl_xor_sync(kAll, own, o));
      const float w = fmaxf(x1 - x0, 0.0f) + mean_w, h = fmaxf(y1 - y0, 0.0f) + mean_h;
      // (both halves whole; an overflow to NaN counts as wide)
      const int other = __shfl_xor_sync(kAll, size, o);
      const bool whole = size == o && other == o;
      if (whole && (w * h * per_area <= kPacketRows || w * h <= kPacketGrowth * own))
        size = 2 * o;
    }
    const bool leader = (lane & (size - 1)) == 0 && j < n;
    const unsigned lead = __ballot_sync(kAll, leader);
    unsigned long long at = 0;
    if (lane == 0) at = atomicAdd(&ctrl[3], (unsigned long long)__popc(lead));
    at = __shfl_sync(kAll, at, 0) + __popc(lead & ((1u << lane) - 1u));
    if (leader) packets[at] = make_uint2((uint32_t)j, min((uint32_t)size, n - (uint32_t)j));
  }
}

// What a packet holds of the 32 build rows it works on next (lane u: row u).
struct PacketRow {
  uint32_t b, mask;          // build row, lanes whose boxes overlap
  uint32_t hits, opens;      // lanes that meet it, lanes left open
  uint32_t near, v_in, v_out;  // of the open lanes
};

template <bool kPoints>
__global__ void __launch_bounds__(kPacketThreads, kPoints ? 8 : 6)
    k_packet(LbvhView t, GeomsView B, GeomsView P, const uint32_t* __restrict__ order,
             int predicate, uint32_t* __restrict__ counts, PacketStore A, DeviceStatus* st) {
  __shared__ int stacks[kPacketThreads / 32][kTravStack];
  __shared__ uint2 lists[kPacketThreads / 32][32];  // sorted build row, lane mask
  const int lane = threadIdx.x & 31;
  const unsigned lower = (1u << lane) - 1u;
  int* stack = stacks[threadIdx.x >> 5];
  uint2* list = lists[threadIdx.x >> 5];
  const uint32_t n = P.n;
  const uint32_t max_steps = 2u * t.nleaves + 2u;
  const uint32_t npackets = (uint32_t)A.ctrl[3];
  uint32_t esc = 0, cand = 0;
  const float nanf32 = __int_as_float(0x7fc00000);
  while (true) {
    uint32_t g = 0;
    if (lane == 0) g = (uint32_t)min(atomicAdd(&A.ctrl[2], 1ull), 0xffffffffull);
    g = __shfl_sync(kAll, g, 0);
    if (g >= npackets) break;
    const uint2 run = A.packets[g];
    bool have = (uint32_t)lane < run.y;
    const uint32_t pi = have ? order[run.x + lane] : 0u;
    if (have && pi >= n) {
      traversal_fault(t, kBadProbe, pi);
      have = false;
    }
    float4 q = make_float4(nanf32, nanf32, nanf32, nanf32);
    if (have) q = P.box[pi];
    const bool live = q.x <= q.z && q.y <= q.w && t.nprims > 0;
    // the lane's point, or its polygon when that is a single ring
    double2 p = make_double2(0.0, 0.0);
    float2 p32 = make_float2(0.0f, 0.0f);
    LaneRing o{0, make_float4(0.0f, 0.0f, 0.0f, 0.0f), p32};
    bool ring = false;
    if (live) {
      if (kPoints) {
        p = P.pt[pi];
        p32 = make_float2(q.x, q.y);
      } else if (P.kind[pi] == kPolygon) {
        const uint32_t q0 = P.row_part[pi];
        if (P.row_part[pi + 1] - q0 == 1) {
          const uint32_t r0 = P.part_ring[q0];
          if (P.part_ring[q0 + 1] - r0 == 1 && ring_npts(P, r0) >= 3 && P.ring_nsegs[r0] > 0) {
            ring = true;
            const uint32_t V = P.ring_vtx[r0];
            o = LaneRing{r0, P.ring_rect32[r0], P.xy32[V]};
          }
        }
      }
    }
    const float4 U = make_float4(warp_min(live ? q.x : INFINITY), warp_min(live ? q.y : INFINITY),
                                 warp_max(live ? q.z : -INFINITY), warp_max(live ? q.w : -INFINITY));
    uint32_t cnt = 0;  // this lane's pairs
    uint32_t nrec = 0, chunk = kNoChunk;

    int sp = 0;
    int node = t.nleaves > 1 ? 0 : ~0;
    uint32_t steps = 0;
    uint32_t k = 0, k1 = 0;  // rest of the leaf at hand
    bool more = __any_sync(kAll, live);
    while (more || k < k1) {
      // the next (up to 32) build rows that some lane's box overlaps
      uint32_t listed = 0;
      while (true) {
        for (; k < k1 && listed < 32; k++) {
          const bool on = live && box_overlap(t.sorted_box[k], q);
          const unsigned mask = __ballot_sync(kAll, on);
          if (mask == 0) continue;
          cand += on ? 1u : 0u;
          if (lane == 0) list[listed] = make_uint2(k, mask);
          listed++;
        }
        if (k < k1) break;
        if (!more) break;
        if (++steps > max_steps) {  // each node is visited at most once
          if (lane == 0) traversal_fault(t, kTooLong, g);
          more = false;
          break;
        }
        if (node < 0) {
          const uint32_t c = (uint32_t)(~node);
          if (c >= t.nleaves) {
            if (lane == 0) traversal_fault(t, kBadLeaf, c);
            more = false;
            break;
          }
          k = c * t.leaf_size;
          k1 = min(k + t.leaf_size, t.nprims);
        } else {
          if ((uint32_t)node + 1 >= t.nleaves) {
            if (lane == 0) traversal_fault(t, kBadNode, (unsigned)node);
            more = false;
            break;
          }
          const float4 lb = t.node_box[2 * node], rb = t.node_box[2 * node + 1];
          const int2 ch = t.node_child[node];
          const bool hl = __any_sync(kAll, live && box_overlap(lb, q));
          const bool hr = __any_sync(kAll, live && box_overlap(rb, q));
          if (hl && hr) {
            if (sp >= kTravStack) {  // deeper than any tree built here: record, stop
              if (lane == 0) traversal_fault(t, kStackOverflow, g);
              more = false;
              break;
            }
            if (lane == 0) stack[sp] = ch.y;
            sp++;
            node = ch.x;
            continue;
          }
          if (hl || hr) {
            node = hl ? ch.x : ch.y;
            continue;
          }
        }
        if (sp == 0) {
          more = false;  // after the leaf at hand
          continue;
        }
        sp--;
        __syncwarp();
        node = stack[sp];
        __syncwarp();
      }
      if (listed == 0) continue;

      // decided, recorded, open pairs queued
      __syncwarp();
      // lane u: build row u, its first ring and the cells that hold U
      PacketRow me{0, 0, 0, 0, 0, 0, 0};
      uint32_t r0 = 0, r1 = 0, q0 = 0, q1 = 0;
      int st_u = 0;
      bool known = false;
      uint8_t kind = kEmpty;
      if ((uint32_t)lane < listed) {
        const uint2 x = list[lane];
        me.mask = x.y;
        me.b = t.sorted_id[x.x];
        kind = B.kind[me.b];
        q0 = B.row_part[me.b];
        q1 = B.row_part[me.b + 1];
        if (kind == kPolygon && q1 - q0 == 1) {
          r0 = B.part_ring[q0];
          r1 = B.part_ring[q0 + 1];
          if (kPoints) {
            known = r1 - r0 == 1;
          } else {
            // rings without bands (or too few points) take the general code
            known = r1 > r0 && B.ring_bands != nullptr;
            for (uint32_t r = r0; r < r1 && known; r++)
              known = ring_npts(B, r) >= 3 && B.band_param[r].y >= 0.0f;
          }
          if (known) st_u = box_grid_status(B, r0, U);
          // inside the shell, the holes have to be looked at
          if (st_u == 1 && r1 - r0 > 1) st_u = 0;
        }
      }
      __syncwarp();
      const unsigned rings = __ballot_sync(kAll, ring);  // (polygons) lanes with a known ring
      if (st_u != 0) {
        const uint32_t sure = kPoints ? me.mask : me.mask & rings;
        if (isolated_result(predicate, st_u == 1)) me.hits = sure;
        me.opens = me.mask & ~sure;
      }
      unsigned todo = __ballot_sync(kAll, (uint32_t)lane < listed && st_u == 0);
      while (todo) {
        const int u = __ffs(todo) - 1;
        todo &= todo - 1;
        const unsigned mask = __shfl_sync(kAll, me.mask, u);
        const bool on = (mask >> lane) & 1u;
        const uint32_t b = __shfl_sync(kAll, me.b, u);
        const uint32_t s0 = __shfl_sync(kAll, r0, u), s1 = __shfl_sync(kAll, r1, u);
        bool hit = false, open = false;
        int near = 0, v_in = -1;
        if (kPoints) {
          const bool aoe = predicate != kContains;
          if (__shfl_sync(kAll, (int)kind, u) == kPoint) {
            hit = on && pteq(B.pt[b], p);
          } else {
            // poly_contains_point of any part
            const uint32_t a0 = __shfl_sync(kAll, q0, u), a1 = __shfl_sync(kAll, q1, u);
            for (uint32_t qa = a0; qa < a1; qa++) {
              const uint32_t t0 = B.part_ring[qa], t1 = B.part_ring[qa + 1];
              bool in = on && !hit && (t1 - t0 == 1 || ring_npts(B, t0) >= 3);
              for (uint32_t h = t0; h < t1 && __any_sync(kAll, in); h++) {
                const bool x = packet_pip(B, h, in, p, p32, U, lane, (h == t0) == aoe, esc);
                in = in && x == (h == t0);  // in the shell, in none of the holes
              }
              hit = hit || in;
            }
          }
          if (predicate == kDisjoint) hit = on && !hit;
        } else {
          open = on;
          const bool mine = on && ring;
          const bool rows = __shfl_sync(kAll, (int)known, u) != 0;
          if (predicate == kWithin || predicate == kCoveredBy || predicate == kEquals) {
            // the probe's ring contains the shell only if its rect does
            if (rows && mine) {
              const float4 h = B.ring_rect32[s0];
              if (h.x < o.box.x || h.y < o.box.y || h.z > o.box.z || h.w > o.box.w) open = false;
            }
          } else if (rows) {
            // the shell, then for lanes strictly inside it the holes
            // (strictly inside a hole is outside the polygon)
            int s = kIsIn;
            for (uint32_t h = s0; h < s1; h++) {
              const bool ask = mine && s == kIsIn;
              if (!__any_sync(kAll, ask)) break;
              int hv;
              const int hs = packet_isolation(B, h, ask, o, P, U, lane, hv, esc);
              if (h == s0) v_in = hv;
              if (ask) s = hs == kIsNear || h == s0 ? hs : (hs == kIsIn ? kIsOut : kIsIn);
            }
            if (mine && s != kIsNear) {
              open = false;
              hit = isolated_result(predicate, s == kIsIn);
            } else if (mine) {
              // a first vertex strictly outside the shell: not contained
              if (v_in == 0 && (predicate == kContains || predicate == kCovers)) open = false;
              near = 1;
              if (s1 - s0 == 1) {
                // strictly inside: they intersect (the vertex test of the
                // smaller ring, which the probe is)
                if (v_in == 1 && (predicate == kIntersects || predicate == kDisjoint) &&
                    !swap_rings<true>(B, s0, P, o.ring)) {
                  open = false;
                  hit = predicate == kIntersects;
                }
              }
            }
          }
        }
        const unsigned hits = __ballot_sync(kAll, hit), opens = __ballot_sync(kAll, open);
        const unsigned nears = __ballot_sync(kAll, open && near);
        const unsigned ins = __ballot_sync(kAll, v_in == 1), outs = __ballot_sync(kAll, v_in == 0);
        if (lane == u) {
          me.hits = hits;
          me.opens = opens;
          me.near = nears;
          me.v_in = ins;
          me.v_out = outs;
        }
      }
      // records of the rows with something to say, in order
      const unsigned say = __ballot_sync(kAll, (me.hits | me.opens) != 0);
      if (say == 0) continue;
      const uint32_t at = packet_append(A, g, lane, (say >> lane) & 1u, make_uint2(me.b, me.hits),
                                        nrec, chunk);
      for (unsigned s = say; s;) {
        const int u = __ffs(s) - 1;
        s &= s - 1;
        cnt += (__shfl_sync(kAll, me.hits, u) >> lane) & 1u;
        const unsigned opens = __shfl_sync(kAll, me.opens, u);
        if (kPoints || opens == 0) continue;
        const uint32_t b = __shfl_sync(kAll, me.b, u), rec = __shfl_sync(kAll, at, u);
        const unsigned nears = __shfl_sync(kAll, me.near, u);
        const unsigned ins = __shfl_sync(kAll, me.v_in, u), outs = __shfl_sync(kAll, me.v_out, u);
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(&A.ctrl[1], (unsigned long long)__popc(opens));
        const unsigned long long e = __shfl_sync(kAll, base, 0) + __popc(opens & lower);
        if (((opens >> lane) & 1u) && e < A.queue_cap) {
          uint32_t flags = (uint32_t)lane;
          if ((nears >> lane) & 1u) {
            flags |= kOpenNear;
            if ((ins >> lane) & 1u) flags |= kOpenIn;
            if ((outs >> lane) & 1u) flags |= kOpenOut;
          }
          A.queue[e] = make_uint4(b, pi, rec, flags);
        }
      }
    }
    __syncwarp();
    if (have) counts[pi] = cnt;
    if (lane == 0) A.nrec[g] = nrec;
  }
  flush_counters(st, esc, cand);
}

// The side of vertex v (FP64) of edge `id` of ring rr that FP32 leaves open, in
// FP64 (e: the edge's listed direction; 0 when still open).
__device__ __noinline__ int side64(const GeomsView& Gr, uint32_t rr, uint32_t id, float4 e,
                                   double2 v) {
  const uint32_t V = Gr.ring_vtx[rr] + id;
  const double2 a = Gr.xy[V], b = Gr.xy[V + 1];
  const float2 a32 = Gr.xy32[V];
  if (e.x == e.z && e.y == e.w) return 0;
  const int o = orient64(a, b, v);
  return a32.x == e.x && a32.y == e.y ? o : -o;
}

// Whether the segment from vertex V to V + 1 of Go, whose ends lie on
// different sides of an edge's line, crosses the edge (1 / 0, -1 open), in FP64.
__device__ __noinline__ int cross64(const GeomsView& Gr, uint32_t rr, uint32_t id,
                                    const GeomsView& Go, uint32_t V) {
  const uint32_t E = Gr.ring_vtx[rr] + id;
  const double2 a = Go.xy[V], b = Go.xy[V + 1];
  const int oc = orient64(a, b, Gr.xy[E]), od = orient64(a, b, Gr.xy[E + 1]);
  return oc == 0 || od == 0 ? -1 : oc != od;
}

// Two rings, per lane (all 32 lanes call, those with `on` have a pair):
// whether some edges of them properly cross (1), none meet (0), or that is not
// decided (-1).  Only edges of rr that come near ro's box matter (the others are
// strictly separated from all of ro, or all of it lies strictly on one side of
// them): those of the cells that hold it.  Every vertex of ro needs a decided
// side of such an edge (or its two neighbours' segments to be strictly
// separated from it); two neighbours on different sides cross its line, and
// then its own ends need decided sides of theirs.
//
// The lanes' edges differ in number, from none to over ten, so the warp lists
// all (pair, edge) items and takes them 32 at a time, first against the pair's
// box and, those that come near it, against its ring.  (With each lane going
// through its own edges the warp took the longest list of the 32 times the
// most vertices: 10.5 ms for 11.7M pairs, 7.0 this way.)
constexpr int kItems = 512;
struct OpenWarp {
  uint32_t item[kItems];  // lane << 27 | edge entry from the ring's first
  uint32_t near[kItems];
  float4 box[32];
  uint32_t ring[32], other[32], first[32];  // rr, ro, rr's first entry
  uint32_t flags[32];  // 1 crosses, 2 not decided
};

__device__ __forceinline__ int rings_cross32(const GeomsView& Gr, uint32_t rr, const GeomsView& Go,
                                             uint32_t ro, bool on, int lane, OpenWarp& W) {
  const uint4 m = on ? Gr.grid_meta[rr] : make_uint4(0u, 0u, 0u, 0u);
  const bool grid = m.y != 0;
  const float4 q = grid ? Gr.grid_rect[rr] : make_float4(0.0f, 0.0f, 1.0f, 1.0f);
  const float4 ob = on ? Go.ring_rect32[ro] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  CellRange r{0, -1, 0, -1, false};
  const int found = grid ? grid_cells(q, (int)m.y, ob, r) : -1;
  const int nx = r.i1 - r.i0 + 1, ny = r.j1 - r.j0 + 1;
  bool ok = found == 0 || (found > 0 && nx <= kLaneCells && ny <= kLaneCells);
  const int cells = ok && found > 0 ? nx * ny : 0;
  const int most = __reduce_max_sync(kAll, cells);
  W.box[lane] = ob;
  W.ring[lane] = rr;
  W.other[lane] = ro;
  W.first[lane] = m.z;
  W.flags[lane] = 0;
  uint32_t nitem = 0, nnear = 0;  // uniform
  // items against their pair's box
  auto sift = [&] {
    __syncwarp();
    for (uint32_t x0 = 0; x0 < nitem; x0 += 32) {
      bool near = false;
      uint32_t it = 0;
      if (x0 + lane < nitem) {
        it = W.item[x0 + lane];
        const uint32_t l = it >> 27;
        const float4 e = Gr.grid_seg[W.first[l] + (it & 0x7ffffffu)];
        const float4 b = W.box[l];
        near = !apart32(e, b.x, b.y, b.z, b.w) &&
               box_side32(make_float2(e.x, e.y), make_float2(e.z, e.w), b) == 0;
      }
      __syncwarp();
      const unsigned keep = __ballot_sync(kAll, near);
      if (near) {
        const uint32_t at = nnear + __popc(keep & ((1u << lane) - 1u));
        if (at < kItems) W.near[at] = it;
        else atomicOr(&W.flags[it >> 27], 2u);
      }
      nnear = min(nnear + (uint32_t)__popc(keep), (uint32_t)kItems);
    }
    nitem = 0;
    __syncwarp();
  };
  int i = r.i0, j = r.j0;
  for (int t = 0; t < most; t++) {
    uint32_t w = kCellIn;
    if (t < cells) w = Gr.grid_cell[m.x + (uint32_t)j * m.y + (uint32_t)i];
    if (cell_state(w) == kCellUnknown) ok = false;
    const uint32_t n = cell_state(w) >= kCellMixed ? cell_count(w) : 0u;
    const uint32_t inc = warp_inclusive_scan(n);
    const uint32_t all = __shfl_sync(kAll, inc, 31);
    if (all > (uint32_t)kItems) {
      ok = false;  // (over 16 edges a cell on average: not worth it)
    } else {
      if (nitem + all > (uint32_t)kItems) sift();
      for (uint32_t k = 0; k < n; k++)
        W.item[nitem + inc - n + k] = (uint32_t)lane << 27 | (cell_first(w) + k);
      nitem += all;
    }
    __syncwarp();
    if (++i > r.i1) {
      i = r.i0;
      j++;
    }
  }
  sift();
  // near edges against their pair's ring
  for (uint32_t x0 = 0; x0 < nnear; x0 += 32) {
    const bool mine = x0 + lane < nnear;
    const uint32_t it = mine ? W.near[x0 + lane] : 0u;
    const uint32_t l = it >> 27;
    uint32_t V = 0, at = 0;
    int ns = -1;
    float4 e = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (mine) {
      V = Go.ring_vtx[W.other[l]];
      ns = Go.ring_nsegs[W.other[l]];
      at = W.first[l] + (it & 0x7ffffffu);
      e = Gr.grid_seg[at];
    }
    const float2 c = make_float2(e.x, e.y), d = make_float2(e.z, e.w);
    const int mostv = __reduce_max_sync(kAll, ns);
    uint32_t fl = 0;
    float2 a = make_float2(0.0f, 0.0f);
    int sa = 0;
    for (int v = 0; v <= mostv; v++) {
      if (v <= ns) {
        const float2 b = Go.xy32[V + v];
        int sb = orient32(c, d, b);
        if (sb == 0) sb = side64(Gr, W.ring[l], Gr.grid_edge_id[at], e, Go.xy[V + v]);
        if (v > 0 && !apart32(e, fmin0f(a.x, b.x), fmin0f(a.y, b.y), fmax0f(a.x, b.x),
                              fmax0f(a.y, b.y))) {
          if (sa == 0 || sb == 0) {
            fl |= 2u;
          } else if (sa != sb) {
            const int oc = orient32(a, b, c), od = orient32(a, b, d);
            int x = oc != od;
            if (oc == 0 || od == 0)
              x = cross64(Gr, W.ring[l], Gr.grid_edge_id[at], Go, V + v - 1);
            fl |= x < 0 ? 2u : (uint32_t)x;
          }
        }
        a = b;
        sa = sb;
      }
      __syncwarp();
    }
    if (fl) atomicOr(&W.flags[l], fl);
    __syncwarp();
  }
  const uint32_t f = W.flags[lane];
  __syncwarp();
  return !ok || (f & 2u) ? -1 : (int)(f & 1u);
}

// An open pair in full.  near: a polygon against a single ring; when the
// polygon has no holes its edges are known to come near the ring's box.
__device__ __noinline__ int open_general(const GeomsView& B, uint32_t b, const GeomsView& P,
                                         uint32_t p, int predicate, bool near, uint32_t& esc) {
  if (near && predicate != kTouches && predicate != kWithin && predicate != kCoveredBy &&
      predicate != kEquals) {
    const uint32_t q = B.row_part[b], rb = B.part_ring[q], rp = P.part_ring[P.row_part[p]];
    if (B.part_ring[q + 1] - rb == 1) {
      if (predicate == kContains || predicate == kCovers)
        return ring_contains_ring<true, true>(B, rb, P, rp, true, esc);
      const int r = ring_intersects_ring<true, false, true>(B, rb, P, rp, esc);
      return predicate == kDisjoint ? !r : r;
    }
  }
  return eval<true>(B, b, P, p, predicate, esc);
}

// The pairs the packets left open, one lane each (neighbouring entries share
// a build row and neighbouring probes).
//
// A single probe ring whose first vertex is strictly inside or outside a build
// ring, with a decided answer to whether their edges cross (rings_cross32),
// needs no point tests: along the probe ring a vertex changes side only at a
// crossing.
//  - Some edge crosses properly.  Walking from the first vertex, the first
//    edge that crosses starts where the first vertex lies; it crosses once
//    and ends on the other side, or meets two edges.  Outside -> in: tg finds
//    a vertex in the build ring, or a segment with two hits: they intersect
//    (with and without allow_on_edge); inside -> out: a vertex out or a segment
//    that crosses: not contained.  tg's segment tests of touches agree with
//    and without edges: it is false.
//  - None does, none touches: the probe ring lies where its first vertex
//    does.  Outside, tg finds no vertex in and no hits; inside, every vertex
//    in and no segment that meets an edge.
// A polygon with holes (tg.c:4040-4136) meets the ring when its shell does and
// no hole holds it, and contains it when its shell does and no hole meets it.
__global__ void __launch_bounds__(kPacketThreads)
    k_packet_open(GeomsView B, GeomsView P, int predicate, uint32_t* __restrict__ counts,
                  PacketStore A, DeviceStatus* st) {
  __shared__ OpenWarp warps[kPacketThreads / 32];
  OpenWarp& W = warps[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  uint32_t esc = 0;
  // past a capacity the run is repeated with more room
  const uint64_t nq =
      A.ctrl[0] > A.chunks || A.ctrl[1] > A.queue_cap ? 0 : (uint64_t)A.ctrl[1];
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const bool sides = B.grid_meta != nullptr && predicate != kWithin && predicate != kCoveredBy &&
                     predicate != kEquals;
  // (whole warps: the loop's bound is that of the warp's first entry)
  for (uint64_t e0 = blockIdx.x * (uint64_t)blockDim.x + (threadIdx.x & ~31u); e0 < nq;
       e0 += stride) {
    const uint64_t e = e0 + (threadIdx.x & 31);
    const bool on = e < nq;
    const uint4 x = on ? A.queue[e] : make_uint4(0u, 0u, 0u, 0u);
    const uint32_t b = x.x, p = x.y;
    int r = -2;
    const bool ring = on && (x.w & kOpenNear);
    uint32_t rb = 0, rp = 0;
    if (ring) {
      rb = B.part_ring[B.row_part[b]];
      rp = P.part_ring[P.row_part[p]];
    }
    if (sides) {
      // ring by ring (the shell, then the holes): the side of the first
      // vertex, and whether edges cross.  tg takes the probe's ring for the
      // smaller one of each two.
      const uint32_t r0 = rb, nr = ring ? B.part_ring[B.row_part[b] + 1] - rb : 0u;
      const uint32_t most = __reduce_max_sync(kAll, nr);
      bool fit = ring && !(predicate == kTouches && nr > 1);
      bool shell_in = false, shell_cross = false, in_hole = false, meets_hole = false;
      for (uint32_t h = 0; h < most; h++) {
        const uint32_t rh = r0 + h;
        if (h < nr && fit)
          fit = B.grid_meta[rh].y != 0 &&
                (nr == 1 ? !swap_rings<true>(B, rh, P, rp) : swap_rings<true>(P, rp, B, rh));
        const bool ask = fit && h < nr;
        int side = h == 0 && (x.w & kOpenIn) ? 1 : (h == 0 && (x.w & kOpenOut) ? 0 : -1);
        if (__any_sync(kAll, ask && side < 0)) {
          const float2 v = ask ? P.xy32[P.ring_vtx[rp]] : make_float2(0.0f, 0.0f);
          bool none;
          int found;
          lane_cells<false>(B, ask ? rh : 0u, ask && side < 0, v, make_float4(v.x, v.y, v.x, v.y),
                            none, found);
          if (side < 0) side = found;
        }
        const int cross = rings_cross32(B, rh, P, rp, ask && side >= 0, lane, W);
        if (ask) {
          if (side < 0 || cross < 0) {
            fit = false;
          } else if (h == 0) {
            shell_in = side == 1;
            shell_cross = cross != 0;
          } else {
            in_hole = in_hole || (side == 1 && !cross);
            meets_hole = meets_hole || side == 1 || cross;
          }
        }
      }
      if (fit) {
        const bool meet = (shell_in || shell_cross) && !in_hole;
        if (predicate == kIntersects) r = meet;
        else if (predicate == kDisjoint) r = !meet;
        else if (predicate == kTouches) r = 0;
        else r = shell_in && !shell_cross && !meets_hole;  // kContains, kCovers
      }
    }
    if (on && r == -2) r = open_general(B, b, P, p, predicate, ring, esc);
    __syncwarp();
    if (on && r < 0) {
      status_fail(st, kUnsupported, e);
    } else if (on && r) {
      atomicOr(&A.rec[x.z].y, 1u << (x.w & 31u));
      atomicAdd(&counts[p], 1u);
    }
  }
  __syncwarp();
  flush_counters(st, esc, 0);
}

// Lane l's bit i of the result: lane i's bit l of x (five exchanges of halves).
__device__ __forceinline__ uint32_t transpose32(uint32_t x, int lane) {
  uint32_t m = 0x0000ffffu;
#pragma unroll
  for (int j = 16; j; j >>= 1, m ^= m << j) {
    const uint32_t y = __shfl_xor_sync(kAll, x, j);
    x = (lane & j) ? (x & ~m) | ((y & ~m) >> j) : (x & m) | ((y & m) << j);
  }
  return x;
}

// A warp per packet: 64 records at a time, two per lane, whose lane masks are
// transposed into each probe's mask of records; then for each probe the lanes
// whose record has it write its next pairs, side by side.  Bound by its
// instructions (98M pairs of 4M points: 629 us with 32 records at a time, a
// ballot for each probe and 64-bit positions, 532 this way; Pos: 32 bits
// where the output has fewer places).  A block takes 4 packets and the next
// block the next ones, as a dense packet has many times another's records.
template <class Pos>
__global__ void __launch_bounds__(128)
    k_packet_scatter(uint32_t n, const uint32_t* __restrict__ order,
                     const uint64_t* __restrict__ offs, uint32_t probe_base, PacketStore A,
                     uint32_t* __restrict__ out_build, uint32_t* __restrict__ out_probe,
                     Pos cap) {
  const int lane = threadIdx.x & 31;
  const uint32_t lower = (1u << lane) - 1u;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint64_t npackets = A.ctrl[3];
  for (uint64_t g = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; g < npackets; g += nw) {
    const uint2 run = A.packets[g];
    const uint32_t pi = (uint32_t)lane < run.y ? order[run.x + lane] : n;
    // (past the output: at its end)
    Pos pos = pi < n ? (Pos)min(offs[pi], (uint64_t)cap) : cap;
    const uint32_t nrec = A.nrec[g];
    uint32_t chunk = nrec ? A.head[g] : kNoChunk;
    for (uint32_t r0 = 0; r0 < nrec && chunk < A.chunks; r0 += 64) {
      uint2 ra = make_uint2(0u, 0u), rb = ra;
      if (r0 + lane < nrec) ra = A.rec[(uint64_t)chunk * 32 + lane];
      if (r0 + 32 < nrec) {
        chunk = A.next[chunk];
        if (chunk >= A.chunks) break;
        if (r0 + 32 + lane < nrec) rb = A.rec[(uint64_t)chunk * 32 + lane];
        if (r0 + 64 < nrec) chunk = A.next[chunk];
      }
      const uint32_t ma = transpose32(ra.y, lane), mb = transpose32(rb.y, lane);
      for (unsigned rows = __ballot_sync(kAll, (ma | mb) != 0); rows; rows &= rows - 1) {
        const int l = __ffs(rows) - 1;
        const uint32_t ba = __shfl_sync(kAll, ma, l), bb = __shfl_sync(kAll, mb, l);
        const Pos at = __shfl_sync(kAll, pos, l);
        const uint32_t row = __shfl_sync(kAll, pi, l) + probe_base;
        const Pos pa = at + __popc(ba & lower), pb = at + __popc(ba) + __popc(bb & lower);
        if ((ra.y >> l) & 1u && pa < cap) {
          out_build[pa] = ra.x;
          out_probe[pa] = row;
        }
        if ((rb.y >> l) & 1u && pb < cap) {
          out_build[pb] = rb.x;
          out_probe[pb] = row;
        }
      }
      pos = min(pos, cap) + (Pos)(__popc(ma) + __popc(mb));  // (never far past the output)
    }
  }
}

}  // namespace

static uint64_t most_packets(uint32_t n) { return ((uint64_t)n + 31) / 32 * 32; }

bool PacketBufs::reserve(uint32_t n, uint64_t chunks, uint64_t queued, cudaStream_t s) {
  const uint64_t most = most_packets(n);
  chunks = std::max(chunk_cap, chunks);
  queued = std::max(queue_cap, queued);
  SPJ_CHECK(chunks <= kPacketMaxChunks && queued <= kPacketMaxQueue,
            "packet records exceed their limit");
  try {
    rec.reserve(chunks * 32 * sizeof(uint2), s);
    next.reserve(chunks * 4, s);
    queue.reserve((queued + 1) * sizeof(uint4), s);
    heads.reserve((most + 1) * 16, s);
    ctrl.reserve(kPacketCtrlBytes, s);
  } catch (const Error&) {
    (void)cudaGetLastError();  // (the next launch's check is not to find it)
    release();
    return false;
  }
  chunk_cap = chunks;
  queue_cap = queued;
  return true;
}

PacketStore PacketBufs::store(uint32_t n) const {
  PacketStore a;
  a.rec = rec.as<uint2>();
  a.next = next.as<uint32_t>();
  a.chunks = (uint32_t)chunk_cap;
  a.packets = heads.as<uint2>();
  a.head = heads.as<uint32_t>() + 2 * most_packets(n);
  a.nrec = a.head + most_packets(n);
  a.queue = queue.as<uint4>();
  a.queue_cap = (uint32_t)queue_cap;
  a.ctrl = ctrl.as<unsigned long long>();
  return a;
}

void PacketBufs::release() {
  for (DevBuf* b : {&rec, &next, &heads, &queue, &ctrl}) b->release();
  chunk_cap = queue_cap = 0;
}

bool packet_takes(int predicate, bool points) {
  // a point probe neither covers nor touches a polygon's inside
  return !points || predicate == kIntersects || predicate == kContains || predicate == kCovers ||
         predicate == kDisjoint;
}

float mean_density(const LbvhView& t) {
  return t.extent_area > 0.0f ? (float)t.nprims / t.extent_area : 0.0f;
}

void packet_runs(const LbvhView& t, const float4* box, const uint32_t* order, uint32_t n,
                 float density, const PacketStore& a, cudaStream_t s) {
  SPJ_CUDA(cudaMemsetAsync(a.ctrl, 0, kPacketCtrlBytes, s));
  if (n == 0) return;
  k_packets<<<grid_for(n, 256, kNumSMs * 8), 256, 0, s>>>(t, box, order, n, t.mean_w, t.mean_h,
                                                          density, a.packets, a.ctrl);
  SPJ_CUDA(cudaGetLastError());
}

void packet_join(const LbvhView& t, const GeomsView& build, const GeomsView& probe, bool points,
                 const uint32_t* order, int predicate, uint32_t* counts, const PacketStore& a,
                 DeviceStatus* st, cudaStream_t s) {
  packet_runs(t, probe.box, order, probe.n, mean_density(t), a, s);
  if (probe.n == 0) return;
  // (a warp per packet, and a packet may hold one row)
  const int g = grid_for((int64_t)probe.n * 32, kPacketThreads, kNumSMs * 8);
  if (points) {
    k_packet<true><<<g, kPacketThreads, 0, s>>>(t, build, probe, order, predicate, counts, a, st);
  } else {
    k_packet<false><<<g, kPacketThreads, 0, s>>>(t, build, probe, order, predicate, counts, a, st);
    k_packet_open<<<kNumSMs * 16, kPacketThreads, 0, s>>>(build, probe, predicate, counts, a, st);
  }
  SPJ_CUDA(cudaGetLastError());
}

void packet_scatter(uint32_t n, const uint32_t* order, const uint64_t* offs, uint32_t probe_base,
                    const PacketStore& a, uint32_t* out_build,
                    uint32_t* out_probe, uint64_t cap, cudaStream_t s) {
  if (n == 0) return;
  const int g = grid_for(n, 128, 1 << 24);
  // (32-bit positions: at most 64 past the output's end)
  if (cap < 0xffffffffull - 0x01000000ull)
    k_packet_scatter<uint32_t><<<g, 128, 0, s>>>(n, order, offs, probe_base, a, out_build,
                                                 out_probe, (uint32_t)cap);
  else
    k_packet_scatter<uint64_t><<<g, 128, 0, s>>>(n, order, offs, probe_base, a, out_build,
                                                 out_probe, cap);
  SPJ_CUDA(cudaGetLastError());
}

}  // namespace spj
