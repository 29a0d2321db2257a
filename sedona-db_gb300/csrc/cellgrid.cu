// cellgrid.cu — per-ring cell grids for the FP32 refine.
//
// A ring with at least kGridMinSegs segments gets a G x G grid over its
// outward f32 rect.  An edge touches a cell unless it provably does not, on
// f32 values: its RN32 bbox strictly separated from the closed cell (a strict
// comparison of RN values proves the exact one), or all four cell corners
// strictly on one side of it (box_side32, whose static bound covers the
// rounding of the edge's coordinates).  A cell that no edge touches is clean:
// every point of it has the same tg answer (the isolation-exit argument in
// predicates.cuh).  The other cells list the edges that touch them.  Each cell
// stores the answer at its centre, from the regular point-in-ring code, and
// each listed edge runs so that the centre is strictly left of it (a cell
// with an edge whose side of the centre is not decided is not answered).
//
// Every edge visits the cells of its bbox (6 or 7 for the zones' rings of 145
// vertices and 26 x 26 cells), twice: to count and to fill, 0.46 + 1.97 ms for
// 50k zones.  (4.47 when each cell scanned the some 50 edges of the bands that
// it spans.)  A packet (packet.cu) reads the 2 or 3 edges of a mixed cell where
// the y-band scan of a point reads some 10, and of a box some 20.
#include "geoms.cuh"
#include "predicates.cuh"
#include "prims.cuh"

#include <cmath>

namespace spj {
namespace {

using namespace pred;

__device__ __forceinline__ uint32_t grid_dim(int nsegs) {
  if (nsegs < kGridMinSegs) return 0;
  uint32_t g = 2u * (uint32_t)ceilf(sqrtf((float)nsegs));
  return g < 8u ? 8u : (g > 32u ? 32u : g);
}

__global__ void k_grid_count(uint32_t nr, const int32_t* __restrict__ nsegs,
                             uint32_t* __restrict__ cells) {
  for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < nr; r += gridDim.x * blockDim.x) {
    const uint32_t g = grid_dim(nsegs[r]);
    cells[r] = g * g;
  }
}

// Outward f32 origin / step of one axis: [lo, lo + n step] covers [a, b].
__device__ __forceinline__ bool grid_axis(double a, double b, int n, float& o, float& step) {
  float lo = __double2float_rd(a), hi = __double2float_ru(b);
  if (!(hi > lo) || !isfinite(lo) || !isfinite(hi)) return false;
  step = __fdiv_ru(__fsub_ru(hi, lo), (float)n);
  if (!(step > 0.0f) || !isfinite(step)) return false;
  o = lo;
  for (int t = 0; t < 64 && grid_edge(o, step, n) < hi; t++) step = next_upf(step);
  return grid_edge(o, step, n) >= hi;
}

constexpr int kMaxCells = 1024;  // grid_dim <= 32
constexpr int kCellThreads = 128;

// The ring's grid (false: none).  meta: the grid's (first cell, G, 0, 0).
__device__ __forceinline__ bool ring_grid(const GeomsView& G, uint32_t r, int& g, float4& q) {
  g = (int)grid_dim(G.ring_nsegs[r]);
  q = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  const Rect64 R = G.ring_rect[r];
  return g > 0 && G.ring_bands != nullptr && G.band_param[r].y >= 0.0f &&
         grid_axis(R.x, R.z, g, q.x, q.z) && grid_axis(R.y, R.w, g, q.y, q.w);
}

// Calls f(cell) for the cells that edge (a, b) touches.
template <class F>
__device__ __forceinline__ void edge_cells(float4 q, int g, float2 a, float2 b, F&& f) {
  const float xmin = fmin0f(a.x, b.x), xmax = fmax0f(a.x, b.x);
  const float ymin = fmin0f(a.y, b.y), ymax = fmax0f(a.y, b.y);
  // closed cells that the bbox is not strictly separated from
  auto lo = [g](float o, float step, float v) {
    int i = (int)fminf(fmaxf(__fdividef(v - o, step), 0.0f), (float)(g - 1));
    while (i < g - 1 && grid_edge(o, step, i + 1) < v) i++;
    while (i > 0 && !(grid_edge(o, step, i) < v)) i--;
    return i;
  };
  auto hi = [g](float o, float step, float v) {
    int i = (int)fminf(fmaxf(__fdividef(v - o, step), 0.0f), (float)(g - 1));
    while (i > 0 && v < grid_edge(o, step, i)) i--;
    while (i < g - 1 && !(v < grid_edge(o, step, i + 1))) i++;
    return i;
  };
  const int i0 = lo(q.x, q.z, xmin), i1 = hi(q.x, q.z, xmax);
  const int j0 = lo(q.y, q.w, ymin), j1 = hi(q.y, q.w, ymax);
  for (int j = j0; j <= j1; j++) {
    const float y0 = grid_edge(q.y, q.w, j), y1 = grid_edge(q.y, q.w, j + 1);
    for (int i = i0; i <= i1; i++) {
      const float x0 = grid_edge(q.x, q.z, i), x1 = grid_edge(q.x, q.z, i + 1);
      if (xmax < x0 || xmin > x1 || ymax < y0 || ymin > y1) continue;
      if (box_side32(a, b, make_float4(x0, y0, x1, y1)) == 0) f(j * g + i);
    }
  }
}

// One block per ring (grid-stride over rings), threads over the edges:
// cell[] receives each cell's edge count, entries[r] their sum.
__global__ void __launch_bounds__(kCellThreads)
    k_cell_count(GeomsView G, const uint64_t* __restrict__ cell_off, uint4* __restrict__ meta,
                 float4* __restrict__ rect, uint32_t* __restrict__ cell,
                 uint32_t* __restrict__ entries) {
  __shared__ uint32_t cnt[kMaxCells];
  __shared__ uint32_t total;
  for (uint32_t r = blockIdx.x; r < G.nrings; r += gridDim.x) {
    int g;
    float4 q;
    const bool ok = ring_grid(G, r, g, q);
    if (threadIdx.x == 0) {
      meta[r] = make_uint4((uint32_t)cell_off[r], ok ? (uint32_t)g : 0u, 0u, 0u);
      rect[r] = q;
      total = 0;
    }
    for (int c = threadIdx.x; c < g * g; c += blockDim.x) cnt[c] = 0;
    __syncthreads();
    uint32_t mine = 0;
    if (ok) {
      const uint32_t V = G.ring_vtx[r];
      const int ns = G.ring_nsegs[r];
      for (int e = threadIdx.x; e < ns; e += blockDim.x)
        edge_cells(q, g, G.xy32[V + e], G.xy32[V + e + 1], [&](int c) {
          atomicAdd(&cnt[c], 1u);
          mine++;
        });
    }
    for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
    if ((threadIdx.x & 31) == 0 && mine) atomicAdd(&total, mine);
    __syncthreads();
    for (int c = threadIdx.x; c < g * g; c += blockDim.x) cell[cell_off[r] + c] = cnt[c];
    if (threadIdx.x == 0) entries[r] = total;
    __syncthreads();
  }
}

// The cells' words from their counts, and their edges: first = the ring's
// first entry.
//
// Where the centres lie is known without point tests.  The horizontal through
// the centres of a row of cells starts left of the ring, outside; each of its
// halves, from a cell's left border to its centre and on to the right border,
// stays in that cell, so only the cell's edges can cross it, and each thread
// that lists an edge there toggles the halves that it crosses (the edge's
// ends strictly above and below the horizontal, the half's ends on decided
// sides of it).  One thread per row then goes along it.  A half with an
// undecided edge ends that: the next centre is asked of the point-in-ring
// code (as all of them once were: 3.36 ms for 50k zones, 1.97 now).
constexpr uint32_t kOddLeft = 1, kOddRight = 2, kOpenLeft = 4, kOpenRight = 8, kOpenCell = 16;
__global__ void __launch_bounds__(kCellThreads)
    k_cell_fill(GeomsView G, const uint64_t* __restrict__ first, uint4* __restrict__ meta,
                const float4* __restrict__ rect, uint32_t* __restrict__ cell,
                float4* __restrict__ seg, uint16_t* __restrict__ edge_id) {
  __shared__ uint32_t start[kMaxCells], at[kMaxCells], flag[kMaxCells];
  __shared__ uint32_t warp_sum[kCellThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint32_t r = blockIdx.x; r < G.nrings; r += gridDim.x) {
    const uint4 m = meta[r];
    const int g = (int)m.y, cells = g * g;
    if (g == 0) continue;
    const float4 q = rect[r];
    const uint64_t base = first[r];
    uint32_t* word = cell + m.x;
    // exclusive scan of the counts, each thread a run of cells
    const int per = (cells + kCellThreads - 1) / kCellThreads;
    const int c0 = min((int)threadIdx.x * per, cells), c1 = min(c0 + per, cells);
    uint32_t sum = 0;
    for (int c = c0; c < c1; c++) sum += word[c];
    uint32_t inc = warp_inclusive_scan(sum);
    if (lane == 31) warp_sum[warp] = inc;
    __syncthreads();
    uint32_t run = inc - sum;
    for (int w = 0; w < warp; w++) run += warp_sum[w];
    for (int c = c0; c < c1; c++) {
      start[c] = at[c] = run;
      flag[c] = 0;
      run += word[c];
    }
    __syncthreads();
    const uint32_t V = G.ring_vtx[r];
    const int ns = G.ring_nsegs[r];
    for (int e = threadIdx.x; e < ns; e += blockDim.x) {
      const float2 a = G.xy32[V + e], b = G.xy32[V + e + 1];
      edge_cells(q, g, a, b, [&](int c) {
        const int i = c % g;
        const float2 p = grid_centre(q, i, c / g);
        const int o = orient32(a, b, p);
        uint32_t f = o == 0 ? kOpenCell | kOpenLeft | kOpenRight : 0u;
        const bool above = a.y > p.y && b.y > p.y, below = a.y < p.y && b.y < p.y;
        if (o != 0 && !above && !below) {
          const int ol = orient32(a, b, make_float2(grid_edge(q.x, q.z, i), p.y));
          const int orr = orient32(a, b, make_float2(grid_edge(q.x, q.z, i + 1), p.y));
          const bool ends = a.y == p.y || b.y == p.y;  // an end on the horizontal
          if (ends || ol == 0) f |= kOpenLeft;
          else if (ol != o) f |= kOddLeft;
          if (ends || orr == 0) f |= kOpenRight;
          else if (orr != o) f |= kOddRight;
        }
        if (f & (kOddLeft | kOddRight)) atomicXor(&flag[c], f & (kOddLeft | kOddRight));
        if (f & ~(kOddLeft | kOddRight)) atomicOr(&flag[c], f & ~(kOddLeft | kOddRight));
        const uint32_t k = atomicAdd(&at[c], 1u);
        edge_id[base + k] = (uint16_t)e;
        seg[base + k] = o < 0 ? make_float4(b.x, b.y, a.x, a.y) : make_float4(a.x, a.y, b.x, b.y);
      });
    }
    __syncthreads();
    for (int j = threadIdx.x; j < g; j += blockDim.x) {
      bool in = false, known = true;  // at the cell's left border
      for (int i = 0; i < g; i++) {
        const int c = j * g + i;
        const uint32_t f = flag[c], n = at[c] - start[c];
        bool centre = in != ((f & kOddLeft) != 0);
        uint32_t w = kCellUnknown;
        if (!(f & kOpenCell)) {
          if (!known || (f & kOpenLeft)) {
            const float2 p = grid_centre(q, i, j);
            uint32_t esc = 0;
            centre = ring_pip_fast(G, r, make_double2((double)p.x, (double)p.y), p, true, esc).hit;
          }
          if (n <= 255u && start[c] < (1u << 21))
            w = (n ? (centre ? kCellMixedIn : kCellMixedOut) : (centre ? kCellIn : kCellOut)) |
                n << 3 | start[c] << 11;
        }
        word[c] = w;
        known = !(f & (kOpenCell | kOpenRight));
        in = centre != ((f & kOddRight) != 0);
      }
    }
    if (threadIdx.x == 0) meta[r].z = (uint32_t)base;
    __syncthreads();
  }
}

}  // namespace

void build_cell_grid(DeviceGeoms& g, DecodeScratch& sc, cudaStream_t s) {
  const uint32_t nr = g.nrings;
  g.has_grid = false;
  if (nr == 0 || !g.has_bands) return;
  g.grid_meta.reserve(((size_t)nr + 1) * sizeof(uint4), s);
  g.grid_rect.reserve(((size_t)nr + 1) * sizeof(float4), s);
  sc.counts.reserve(((size_t)nr + 1) * 4, s);
  sc.scans.reserve(((size_t)nr + 1) * 8, s);
  k_grid_count<<<grid_for(nr, 256), 256, 0, s>>>(nr, g.ring_nsegs.as<int32_t>(),
                                                 sc.counts.as<uint32_t>());
  scan_u32_u64(sc.counts.as<uint32_t>(), sc.scans.as<uint64_t>(), nr, sc.tmp, s);
  uint64_t total = 0;
  SPJ_CUDA(cudaMemcpyAsync(&total, sc.scans.as<uint64_t>() + nr, 8, cudaMemcpyDeviceToHost, s));
  SPJ_CUDA(cudaStreamSynchronize(s));
  SPJ_CHECK(total < 0xFFFFFFFFull, "cell grid too large");
  g.grid_cell.reserve((total + 1) * 4, s);
  // the grid is built with the point-in-ring code of a view without a grid
  const GeomsView v = g.view();
  const int blocks = grid_for(nr, 1, kNumSMs * 16);
  k_cell_count<<<blocks, kCellThreads, 0, s>>>(v, sc.scans.as<uint64_t>(), g.grid_meta.as<uint4>(),
                                               g.grid_rect.as<float4>(),
                                               g.grid_cell.as<uint32_t>(),
                                               sc.counts.as<uint32_t>());
  scan_u32_u64(sc.counts.as<uint32_t>(), sc.scans.as<uint64_t>(), nr, sc.tmp, s);
  SPJ_CUDA(cudaMemcpyAsync(&total, sc.scans.as<uint64_t>() + nr, 8, cudaMemcpyDeviceToHost, s));
  SPJ_CUDA(cudaStreamSynchronize(s));
  if (total >= 0xFFFFFFFFull) return;  // (more entries than 32 bits count: no grid)
  g.grid_seg.reserve((total + 1) * sizeof(float4), s);
  g.grid_edge_id.reserve((total + 1) * sizeof(uint16_t), s);
  k_cell_fill<<<blocks, kCellThreads, 0, s>>>(v, sc.scans.as<uint64_t>(), g.grid_meta.as<uint4>(),
                                              g.grid_rect.as<float4>(),
                                              g.grid_cell.as<uint32_t>(),
                                              g.grid_seg.as<float4>(),
                                              g.grid_edge_id.as<uint16_t>());
  SPJ_CUDA(cudaGetLastError());
  SPJ_CUDA(cudaStreamSynchronize(s));
  g.has_grid = true;
}

}  // namespace spj
