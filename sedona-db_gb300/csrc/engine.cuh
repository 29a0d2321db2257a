// engine.cuh — the join engine behind the C ABI: a decoded, indexed build
// side resident in HBM and a probe pipeline
//   decode probe WKB -> f32 filter boxes -> LBVH count / scan / scatter ->
//   refine (tg semantics or DWithin) -> scan / compact
// whose results stay on the device.  This is the GB300 counterpart of the
// reference's GPUSpatialIndex::query_batch
// (rust/sedona-spatial-join-gpu/src/index/gpu_spatial_index.rs:163-229), which
// runs RTSpatialIndex::Probe and RTSpatialRefiner::Refine back to back with
// host round trips in between.
#pragma once
#include <atomic>
#include <mutex>

#include "geoms.cuh"
#include "dwithin.cuh"
#include "lbvh.cuh"
#include "packet.cuh"
#include "refine.cuh"

namespace spj {

constexpr int kPredDWithin = 100;  // ST_DWithin(build, probe, distance)

struct EngineConfig {
  // LBVH leaf size; 0 = by build side: 16 for point columns (ST_DWithin and
  // equality traversals test cheap points), 4 otherwise
  uint32_t leaf_size = 0;
  int refine_form = kFastF32;
  bool profile = false;  // time each phase with CUDA events on the engine stream
  // traversal order of the probe rows: 0 = Morton order from kOrderMinRows
  // rows up, and of fewer where packets take them (packet_pays), 1 = always
  // Morton order, -1 = row order
  int probe_order = 0;
  // point build and probe sides: decide ST_DWithin inside the traversal
  // (FAST_F32 form); otherwise filter, refine and compact
  bool fuse_dwithin = true;
  // fused ST_DWithin: build ids kept per probe by the counting pass (0 = none)
  uint32_t dwithin_slots = 64;
  // fused ST_DWithin: results past the slots go to an overflow arena of the
  // slots' size, so the scatter pass traverses only the probes the arena
  // could not hold (the 24 % of 20M GMM probes with over 64 neighbours hold
  // 80 % of the pairs).  0 off, 1 on, 2 auto: on when the probes are not in
  // Morton order.  20M x 1M GMM points: in row order 297 -> 139 ms per step;
  // in Morton order the counting pass slowed from 38 to 103 ms with it (the
  // scatter pass fell from 33 to 9 ms), so auto leaves it off there.  (Slots and
  // arena are of the traversal per probe; ordered probes take packets unless
  // one of them is set)
  int dwithin_arena = 2;
  // (candidate_order, order_tiles, refine_min_blocks and refine_split are of the
  // candidate pairs' path and their figures are its; ordered probe rows take the
  // packet kernels where these pay unless one of them is set: 2M x 50k polygons
  // 18.1 ms)
  // refine order of the candidates: 0 as listed (by probe row), 2 by build
  // row then probe Morton rank (a warp then tests one build geometry's edges
  // against neighbouring probes: shared loads and similar trip counts; 2M x
  // 50k polygons: 77 vs 104 ms per step), 3 auto: 2 for relation predicates
  // over a build side that is not all points, from kBuildMajorMin candidates
  // up, else 0.  (The probes' Morton order and a band-and-x order inside the
  // build ring measured slower on every workload and were removed.)
  int candidate_order = 3;
  // build-major order within tiles of the probes' Morton-ordered candidate
  // list: -1 auto (tiles of kOrderTileCandidates), n >= 0: 2^n tiles.  A
  // tile's probe rows stay in cache while the refine passes its build rows
  // (2M x 50k polygons: 45.4 ms per step in one tile, 41.8 with 64 tiles,
  // 40.9 with 256-1024)
  int order_tiles = -1;
  // FP32 refine compiled for this many resident 256-thread blocks per SM
  // (4 or 6), or 0 auto: 6 for ST_Intersects / ST_Disjoint in build-major
  // candidate order (a warp's pairs share one build geometry, and more
  // resident warps hide its load latency better than registers do: 2M x
  // 50k polygons 41.0 vs 43.4 ms), else 4 (the containment and touch tests'
  // deeper calls want the registers: ST_Contains on the same inputs 77.1 vs
  // 78.3 ms; 10M points x 50k zones: 96.7 vs 99.4 ms with 6)
  int refine_min_blocks = 0;
  // per-ring cell grids on the build side (clean cells answer point-in-ring
  // tests in O(1)); set before the build
  bool cell_grid = true;
  // ring-ring and ring-in-ring tests answer from the build ring's clean cells
  // when the probe ring's box lies in them (2M buildings x 50k star zones:
  // 63.0 ms per step with it, 52.7 without: the zones' spiky edges leave few
  // buildings inside clean cells, and the lookup costs every pair)
  bool grid_rings = false;
  // FP32 refine in two passes: a cheap pass (isolation exit, first vertex)
  // over every pair queues the pairs it leaves open, a full pass takes the
  // queue (a warp's lanes then hold pairs of similar cost).  0 off, 1 on,
  // 2 auto: on unless the candidates are in build-major order, where a
  // warp's pairs already share one build geometry (2M x 50k polygons: 59.0
  // ms one pass vs 61.0 split in build-major order; 78.0 vs 63.3 as listed);
  // 3 on, with the open pairs' queue sorted back into candidate order
  int refine_split = 2;
  // host probes (SpjJoinProbeHost): 0 auto (2 slices from 524,288 rows up),
  // 1 one call, n > 1 that many slices
  int host_slices = 0;
  // most memory of the packet kernels' records, and as much again of the pairs
  // that they leave open; joins that need more, or whose memory is not there,
  // take the candidate pairs (ST_DWithin: a traversal per probe).  0: none
  uint64_t packet_bytes = 1ull << 34;
};
constexpr uint32_t kOrderMinRows = 1u << 16;
// When the packet kernels are taken (packet_pays).  A packet's warp goes
// through its build rows one after the other, so with few packets the longest
// takes longer than the candidate pairs spread over all threads; and where 32
// neighbouring rows lie far apart against the build rows, their packet walks
// the tree for each of them in turn.  Both show in how many probe rows a build
// row's box holds (share * rows, the rows spread as the build rows are; a probe
// row meets share * nprims build rows).  Packets against pairs, us per call:
//  - points in 50k zones: 66k rows (84 held) 1,460 / 1,097, 140k (180)
//    1,649 / 1,674, 200k 1,962 / 2,008; in 10k zones 100k (128) 515 / 510, 140k
//    558 / 629: from 90 held, and 1.3 for each build row that one meets;
//  - points in small build rows, where the packets save launches and no more:
//    10k stars 1M rows 490 / 537; 50k stars 130k rows 360 / 335, 500k 558 / 587;
//    5k clustered buildings 250k rows 277 / 301, 50k of them 610 / 354;
//  - buildings intersecting 50k zones: 49k rows (63) 2,315 / 2,150, 66k (84)
//    2,289 / 2,498; 50k stars, 1M rows (31) 2,180 / 1,847, 10k 130k rows 467 / 496,
//    500 131k rows (with the copies of a host batch) 549 / 589;
//  - containment (dearer pairs): 50k zones 16k rows (21) 2,063 / 1,662, 24k (31)
//    1,895 / 2,275; with holes 8k (10) 2,301 / 2,245, 12k (15) 2,500 / 2,987;
//    20k stars 250k rows 652 / 650, 1M 1,301 / 1,431;
//  - touches (the dearest): 50k zones 8k rows 1,987 / 2,575, 5k stars 452 / 524,
//    50k clustered buildings (0.02 met) 647 / 568;
//  - within, covered by, equals: 5k zones (6.4 met) 16k rows 246 / 239, 50k 472 / 586;
//  - ST_DWithin, by how many points of a middling leaf's density the square of
//    twice the distance holds (crowd): 400k points, 16k rows: 5 m 510 / 456, 10 m
//    (0.8) 582 / 528, 20 m (3) 690 / 821; 4k rows at 10 m 490 / 523; 200k points,
//    16k rows: 5 m 411 / 427; 5k points, 20k rows 200 / 172.
constexpr uint32_t kPacketRowsDWithin = 1u << 11;
constexpr uint32_t kPacketRowsFull = 1u << 13;
struct PacketTree {
  uint64_t nprims = 0;
  double share = 0;    // of the build rows' extent that the mean box covers
  bool holes = false;  // some build polygon has holes
  double crowd = 0;
};
bool packet_pays(int predicate, bool points, uint64_t rows, const PacketTree& t);
constexpr uint64_t kBuildMajorMin = 1ull << 22;  // candidates before build-major order pays
constexpr uint64_t kOrderTileCandidates = 1ull << 19;  // auto order_tiles: candidates per tile

// order_tiles as configured, resolved to a tile count for m candidates
inline uint64_t order_tile_count(int configured, uint64_t m) {
  if (configured >= 0) return 1ull << configured;
  return m / kOrderTileCandidates > 1 ? m / kOrderTileCandidates : 1;
}

// refine_min_blocks as configured, with 0 (auto) resolved by the candidate order and
// the predicate (intersects: ST_Intersects or ST_Disjoint)
inline int refine_blocks(int configured, bool build_major, bool intersects = true) {
  return configured ? configured : (build_major && intersects ? 6 : 4);
}
constexpr uint64_t kMaxSlotBytes = 8ull << 30;  // cap of the fused ST_DWithin slot buffer

// Per-phase device time (CUDA events on the launching stream) and counters.
struct JoinStats {
  double ms_decode = 0, ms_filter = 0, ms_refine = 0, ms_compact = 0;
  uint64_t calls = 0;
  uint64_t probe_rows = 0;
  uint64_t candidates = 0;
  uint64_t results = 0;
  uint64_t escalations = 0;  // segment / distance tests decided in FP64
  uint64_t pairs_evaluated = 0;
  uint64_t kernel_launches = 0;
  uint64_t probe_bytes = 0;  // WKB + offsets bytes of the probe columns
};

// Per-call scratch; one per concurrent caller.
struct Workspace {
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  DeviceGeoms probe;
  DecodeScratch dsc;
  ProbeScratch psc;
  DevBuf boxes_tmp, cand_build, cand_probe, flags, out_build, out_probe, scan_tmp, status;
  DevBuf slots;   // fused ST_DWithin result slots
  DevBuf arena;   // fused ST_DWithin overflow arena: cursor, heads, chunks
  DevBuf rqueue;  // pairs left open by the refine's cheap pass, then its count
  DevBuf wkb_data, wkb_offsets, wkb_validity;  // H2D staging of host columns
  PacketBufs packet;  // records and open pairs of the packet refine
  // pinned words that a probe reads back: the decode's status, the filter's
  // counts, the refine's status and counts
  struct Readback {
    DeviceStatus decode;
    uint64_t filter[2];
    DeviceStatus st;
    uint64_t total, ctrl[4];
    unsigned fault[2];
  };
  PinnedBuf host;
  Readback* back() const { return host.as<Readback>(); }
  cudaEvent_t ev[6] = {};
  bool last_probe_points = true;
  Workspace();
  ~Workspace();
};

class JoinEngine {
 public:
  JoinEngine(int device, EngineConfig cfg);
  ~JoinEngine();

  int device() const { return device_; }
  EngineConfig& config() { return cfg_; }

  // Build side from a device WKB column (decoded, boxed, indexed, banded),
  // on the engine's own stream; the column must be complete on the device
  // (the caller has synchronized whatever stream wrote it).
  void build(const WkbDeviceColumn& col);
  bool built() const { return built_; }
  // Rebuild the LBVH over the decoded build boxes with another leaf size.
  void reindex(uint32_t leaf_size);
  const DeviceGeoms& build_geoms() const { return bg_; }
  void set_grid_rings(bool on) { bg_.grid_rings = on; }
  const Lbvh& lbvh() const { return bvh_; }

  // Probe with a device WKB column.  Results (device pointers owned by the
  // workspace, valid until its next call) are grouped by probe row in
  // ascending probe order; probe ids are offset by probe_base.
  // d_row (device, one per probe row): ST_DWithin distances per row; a
  // negative or NaN distance matches nothing.
  uint64_t probe(Workspace& ws, const WkbDeviceColumn& col, int predicate, double distance,
                 uint32_t probe_base, const uint32_t** d_build, const uint32_t** d_probe,
                 const double* d_row = nullptr);

  // Refine caller-supplied candidate pairs (device arrays) against an
  // already decoded probe column; output compacted into ws.out_*.
  uint64_t refine_pairs(Workspace& ws, const GeomsView& probe, const uint32_t* cb,
                        const uint32_t* cp, uint64_t m, int predicate, double distance);

  // Whether probes in Morton order take the packet kernels (packet.cuh).
  bool packet_path(int predicate, bool points) const;
  bool packet_dwithin() const;
  // What packet_pays goes by.
  PacketTree packet_tree(double distance) const;
  uint64_t packet_calls() const { return packet_calls_; }

  JoinStats stats();
  void reset_stats();

 private:
  void split_points();
  bool packet_probe(Workspace& ws, int predicate, double distance, const double* d_row,
                    const float4* boxes, uint32_t probe_base, const uint32_t* order,
                    DeviceStatus& hst, uint64_t& launches, uint64_t& total);
  int device_;
  std::atomic<uint64_t> packet_calls_{0};
  EngineConfig cfg_;
  DeviceGeoms bg_;
  DecodeScratch bsc_;
  Lbvh bvh_;
  PointSplit bsplit_;  // point build sides: ST_DWithin decided in the traversal
  cudaStream_t bs_ = nullptr;  // build stream; owns the frees of bg_/bsc_/bvh_
  bool built_ = false;
  std::mutex stats_mu_;
  JoinStats stats_;
};

// Host Arrow binary column view (after the Arrow C data interface is parsed).
struct HostWkbColumn {
  int64_t n = 0;
  const void* offsets = nullptr;  // int32 or int64, n+1 entries (absolute into data)
  bool offsets64 = false;
  const uint8_t* data = nullptr;
  const uint8_t* validity = nullptr;
  int64_t validity_offset = 0;
};

// Copies a host column into the workspace staging buffers (H2D on ws.stream)
// and returns the device view.  Returns the bytes copied in *bytes.
WkbDeviceColumn stage_column(Workspace& ws, const HostWkbColumn& col, uint64_t* bytes);

}  // namespace spj
