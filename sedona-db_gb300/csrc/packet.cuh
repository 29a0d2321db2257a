// packet.cuh — filter and refine of relation predicates in one traversal per
// warp (a packet) of 32 probe rows that are neighbours in Morton order.
#pragma once
#include "geoms.cuh"
#include "lbvh.cuh"
#include "refine.cuh"

namespace spj {

// The hits of a packet: one record per build row that some of its 32 probes
// may meet (build row, lane mask of the probes that do), in traversal order,
// kept in chunks of 32 records linked per packet.  Pairs that the packet
// leaves open wait in a queue, with the place of their bit.
struct PacketStore {
  uint2* rec = nullptr;        // chunks * 32 records
  uint32_t* next = nullptr;    // chunks: the packet's next chunk
  uint32_t chunks = 0;
  uint2* packets = nullptr;    // per packet: first place in the probe order, rows
  uint32_t* head = nullptr;    // per packet: first chunk
  uint32_t* nrec = nullptr;    // per packet: records
  uint4* queue = nullptr;      // (build row, probe row, record, lane | flags)
  uint32_t queue_cap = 0;
  // [0] chunks taken, [1] pairs queued, [2] packets started, [3] packets; past
  // a capacity the counts go on (the caller makes room and runs again)
  unsigned long long* ctrl = nullptr;
};
constexpr size_t kPacketCtrlBytes = 4 * sizeof(unsigned long long);

// Adds the records of the lanes with `say` (in lane order) to packet g's list
// (nrec records so far, the last of them in `chunk`); all 32 lanes call.
// Returns where the lane's record lies, written only within the store's room.
constexpr uint32_t kNoChunk = 0xffffffffu;
#ifdef __CUDACC__
__device__ __forceinline__ uint32_t packet_append(const PacketStore& A, uint32_t g, int lane,
                                                  bool say, uint2 rec, uint32_t& nrec,
                                                  uint32_t& chunk) {
  const unsigned all = 0xffffffffu;
  const unsigned who = __ballot_sync(all, say);
  const uint32_t n = (uint32_t)__popc(who);
  if (n == 0) return 0;
  const uint32_t room = (32u - (nrec & 31u)) & 31u;  // in the current chunk
  uint32_t fresh = kNoChunk;
  if (n > room) {
    if (lane == 0) {
      fresh = (uint32_t)min(atomicAdd(&A.ctrl[0], 1ull), (unsigned long long)kNoChunk);
      if (nrec == 0) A.head[g] = fresh;
      else if (chunk < A.chunks) A.next[chunk] = fresh;
    }
    fresh = __shfl_sync(all, fresh, 0);
  }
  const uint32_t rank = (uint32_t)__popc(who & ((1u << lane) - 1u));
  const uint32_t into = rank < room ? chunk : fresh;
  const uint32_t at = into * 32u + ((nrec + rank) & 31u);
  if (say && into < A.chunks) A.rec[at] = rec;
  nrec += n;
  if (n > room) chunk = fresh;
  return at;
}
#endif

// Most chunks and queued pairs a join keeps (at most 16 GB each); one that needs
// more, or whose memory is not there, takes the candidate pairs' path, which has
// no records.
constexpr uint64_t kPacketMaxChunks = 1ull << 26, kPacketMaxQueue = 1ull << 30;
struct PacketLimits {
  uint64_t chunks, queue;
  // as many as `bytes` of records and `bytes` of queued pairs hold
  explicit PacketLimits(uint64_t bytes)
      : chunks(bytes / (32 * sizeof(uint2)) < kPacketMaxChunks ? bytes / (32 * sizeof(uint2))
                                                               : kPacketMaxChunks),
        queue(bytes / sizeof(uint4) < kPacketMaxQueue ? bytes / sizeof(uint4) : kPacketMaxQueue) {}
};

struct PacketBufs {
  DevBuf rec, next, heads, queue, ctrl;
  uint64_t chunk_cap = 0, queue_cap = 0;  // what the buffers hold
  // Makes room for n probe rows and at least the given chunks / pairs.  False
  // when the memory is not there: nothing is kept then.
  bool reserve(uint32_t n, uint64_t chunks, uint64_t queued, cudaStream_t s);
  PacketStore store(uint32_t n) const;
  void release();
};

// Whether the packet kernels answer this predicate for probe rows that are
// all points (else any rows): the others take the candidate pairs' path.
bool packet_takes(int predicate, bool points);

// counts[row] = pairs of each probe row and the packets' records in `a`;
// order: the probe rows in Morton order (n entries).  st: counters[0] += FP64
// escalations, [1] += candidate pairs (overlapping boxes).
void packet_join(const LbvhView& t, const GeomsView& build, const GeomsView& probe, bool points,
                 const uint32_t* order, int predicate, uint32_t* counts, const PacketStore& a,
                 DeviceStatus* st, cudaStream_t s);

// Cuts the n probe rows' Morton order into packets (a.packets, a.ctrl[3]) and
// clears a's counts.  density: build rows per area, by which it judges how many
// a packet may meet (mean_density: over the whole extent).
void packet_runs(const LbvhView& t, const float4* box, const uint32_t* order, uint32_t n,
                 float density, const PacketStore& a, cudaStream_t s);
float mean_density(const LbvhView& t);

// The pairs of the n probe rows, grouped by probe row in ascending order (offs:
// exclusive scan of counts), writes bounded by cap.
void packet_scatter(uint32_t n, const uint32_t* order, const uint64_t* offs,
                    uint32_t probe_base, const PacketStore& a, uint32_t* out_build,
                    uint32_t* out_probe, uint64_t cap, cudaStream_t s);

}  // namespace spj
