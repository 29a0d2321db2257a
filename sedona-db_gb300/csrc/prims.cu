// prims.cu — device-wide scans and an 8-bit LSD radix sort.
//
// Scan: reduce-then-scan over 4096-element tiles (256 threads x 16 items);
// the tile sums are scanned by one 1024-thread block that walks them in
// chunks, then each tile is rescanned with its prefix.  Two reads of the
// input plus one write of the output: the scan is HBM-bound.  Up to 16,384
// elements one block does it all (below).
//
// Radix sort: per 8-bit digit, (1) a per-tile 256-bin histogram, (2) a scan of
// the digit-major histogram table, (3) a stable block-local ranking of the
// tile by digit (ballots and per-warp digit counters), a reorder in shared
// memory, then a scatter whose runs of equal digits land on consecutive
// addresses.  With segments, the table is segment-major, so the same passes
// sort each segment of consecutive tiles in place.
//
// Compaction of candidate pairs by 0/1 flags: per-tile counts and their
// scan, then each tile gathers its survivors in shared memory and writes
// them as one run (no per-element position array).
#include "prims.cuh"

namespace spj {

namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 16;
constexpr int kScanTile = kScanThreads * kScanItems;
static_assert(kScanTile == 4096, "compact_tiles (prims.cuh) counts tiles of 4096 flags");

// Several arrays of one length are scanned by the same launches: array y
// (blockIdx.y) lies y * in_step / y * out_step elements on, its tile sums
// y * sums_step on, and totals (where given) gets its total at [y].
template <class Tin, class Tout>
struct ScanArgs {
  const Tin* in;
  Tout* out;
  Tout* sums;
  Tout* totals;
  int64_t n, in_step, out_step, sums_step;
};

template <class Tin, class Tout>
__global__ void k_tile_reduce(ScanArgs<Tin, Tout> a) {
  __shared__ Tout sm[9];
  const Tin* in = a.in + blockIdx.y * a.in_step;
  const int64_t base = (int64_t)blockIdx.x * kScanTile;
  Tout acc = 0;
#pragma unroll
  for (int j = 0; j < kScanItems; j++) {
    int64_t i = base + j * kScanThreads + threadIdx.x;
    if (i < a.n) acc += (Tout)in[i];
  }
  Tout total;
  block_exclusive_scan_256<Tout>(acc, sm, &total);
  if (threadIdx.x == 0) a.sums[blockIdx.y * a.sums_step + blockIdx.x] = total;
}

// One block of 1024 threads per array scans its nt tile sums in place
// (exclusive); total_out + y * out_step and totals[y] get the total.
template <class T>
__global__ void k_scan_sums(T* __restrict__ sums, int64_t nt, T* __restrict__ total_out,
                            int64_t sums_step, int64_t out_step, T* __restrict__ totals) {
  __shared__ T warp_tot[32];
  __shared__ T carry;
  sums += blockIdx.y * sums_step;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int64_t b = 0; b < nt; b += blockDim.x) {
    int64_t i = b + threadIdx.x;
    T v = i < nt ? sums[i] : T(0);
    T inc = warp_inclusive_scan(v);
    if (lane == 31) warp_tot[warp] = inc;
    __syncthreads();
    if (warp == 0) {
      T w = warp_tot[lane];
      T wi = warp_inclusive_scan(w);
      warp_tot[lane] = wi - w;
    }
    __syncthreads();
    T ex = carry + warp_tot[warp] + inc - v;
    if (i < nt) sums[i] = ex;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry = ex + v;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    total_out[blockIdx.y * out_step] = carry;
    if (totals) totals[blockIdx.y] = carry;
  }
}

// The exclusive prefixes within a warp's 32 * kItems elements (lane l of round
// j: element 32 j + l), in place; returns their sum.
template <class T, int kItems>
__device__ __forceinline__ T scan_rounds(T* v) {
  T run = 0;
#pragma unroll
  for (int j = 0; j < kItems; j++) {
    const T inc = warp_inclusive_scan(v[j]);
    v[j] = run + inc - v[j];
    run += __shfl_sync(0xffffffffu, inc, 31);
  }
  return run;
}

// Scans one tile of 32 * kItems elements per warp from `base` on; a warp's
// elements are consecutive and its loads and stores coalesced.  (With 16
// consecutive elements per thread each store touched 32 sectors: 4M counts
// 27 us, 9.4 this way.)  The shuffles bound a block of 32 warps (one a clock
// per SM), so sums that fit are added in 32 bits.
template <class Tin, class Tout, int kWarps, int kItems>
__device__ __forceinline__ Tout scan_tile(const Tin* __restrict__ in, int64_t base, int64_t n,
                                          Tout start, Tout* __restrict__ out) {
  __shared__ Tout warp_sum[kWarps + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t i0 = base + (int64_t)warp * (32 * kItems) + lane;
  uint32_t v[kItems], most = 0;
#pragma unroll
  for (int j = 0; j < kItems; j++) {
    v[j] = i0 + j * 32 < n ? (uint32_t)in[i0 + j * 32] : 0u;
    most |= v[j];
  }
  Tout ex[kItems];
  Tout run;
  constexpr uint32_t kFits = 0xffffffffu / (32 * kItems);
  if (sizeof(Tout) == 4 || !__any_sync(0xffffffffu, most > kFits)) {
    run = (Tout)scan_rounds<uint32_t, kItems>(v);
#pragma unroll
    for (int j = 0; j < kItems; j++) ex[j] = (Tout)v[j];
  } else {
#pragma unroll
    for (int j = 0; j < kItems; j++) ex[j] = (Tout)v[j];
    run = scan_rounds<Tout, kItems>(ex);
  }
  if (lane == 0) warp_sum[warp] = run;
  __syncthreads();
  if (warp == 0) {
    const Tout w = lane < kWarps ? warp_sum[lane] : Tout(0);
    const Tout wi = warp_inclusive_scan(w);
    if (lane < kWarps) warp_sum[lane] = wi - w;
    if (lane == kWarps - 1) warp_sum[kWarps] = wi;
  }
  __syncthreads();
  start += warp_sum[warp];
#pragma unroll
  for (int j = 0; j < kItems; j++)
    if (i0 + j * 32 < n) out[i0 + j * 32] = start + ex[j];
  return warp_sum[kWarps];
}

template <class Tin, class Tout>
__global__ void __launch_bounds__(kScanThreads) k_tile_scan(ScanArgs<Tin, Tout> a) {
  scan_tile<Tin, Tout, kScanThreads / 32, kScanItems>(
      a.in + blockIdx.y * a.in_step, (int64_t)blockIdx.x * kScanTile, a.n,
      a.sums[blockIdx.y * a.sums_step + blockIdx.x], a.out + blockIdx.y * a.out_step);
}

// The whole scan of up to kScanOne elements by one block per array: a small
// call is bound by its launches (three of them with their gaps took 14 us for
// 8,192 counts, this one 3.7), and no tile sums are needed.
constexpr int kScanOneThreads = 1024;
constexpr int64_t kScanOne = kScanOneThreads * kScanItems;
template <class Tin, class Tout, int kItems>
__global__ void __launch_bounds__(kScanOneThreads) k_scan_one(ScanArgs<Tin, Tout> a) {
  Tout* out = a.out + blockIdx.y * a.out_step;
  const Tout total = scan_tile<Tin, Tout, kScanOneThreads / 32, kItems>(
      a.in + blockIdx.y * a.in_step, 0, a.n, Tout(0), out);
  if (threadIdx.x == 0) {
    out[a.n] = total;
    if (a.totals) a.totals[blockIdx.y] = total;
  }
}

// Stream compaction of candidate pairs by 0/1 flags, per 4096-flag tile:
// the tile's flags (16 per thread, one 16-byte load when aligned), a block
// scan of their counts, the survivors gathered in shared memory, then
// written as one coalesced run at the tile's offset (sums: exclusive tile
// offsets).  No per-element position array is written or read.
__global__ void __launch_bounds__(kScanThreads)
    k_compact_tile(const uint32_t* __restrict__ cb, const uint32_t* __restrict__ cp,
                   const uint8_t* __restrict__ flags, int64_t n,
                   const uint64_t* __restrict__ sums, uint32_t* __restrict__ ob,
                   uint32_t* __restrict__ op, uint64_t out_cap) {
  __shared__ uint32_t sb[kScanTile], sp[kScanTile];
  __shared__ uint32_t sm[9];
  const int64_t mybase = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
  uint32_t f = 0;  // bit j: flag of item mybase + j
  if (mybase + kScanItems <= n && (reinterpret_cast<uintptr_t>(flags + mybase) & 15) == 0) {
    const uint4 v = *reinterpret_cast<const uint4*>(flags + mybase);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < kScanItems; j++)
      f |= (uint32_t)(((w[j >> 2] >> (8 * (j & 3))) & 0xffu) != 0) << j;
  } else {
#pragma unroll
    for (int j = 0; j < kScanItems; j++)
      if (mybase + j < n && flags[mybase + j]) f |= 1u << j;
  }
  uint32_t total;
  uint32_t lo = block_exclusive_scan_256<uint32_t>((uint32_t)__popc(f), sm, &total);
#pragma unroll
  for (int j = 0; j < kScanItems; j++)
    if ((f >> j) & 1u) {
      sb[lo] = cb[mybase + j];
      sp[lo] = cp[mybase + j];
      lo++;
    }
  __syncthreads();
  const uint64_t tb = sums[blockIdx.x];
  for (uint32_t k = threadIdx.x; k < total; k += kScanThreads) {
    const uint64_t o = tb + k;
    if (o < out_cap) {  // bounded by the output capacity
      ob[o] = sb[k];
      op[o] = sp[k];
    }
  }
}

// Scans of `count` arrays with caller-owned tile sums (sums_step entries of
// Tout for each).
template <class Tin, class Tout>
void scan_launch(const ScanArgs<Tin, Tout>& a, unsigned count, cudaStream_t s) {
  const dim3 one(1, count);
  if (a.n <= kScanOne / 4) {
    k_scan_one<Tin, Tout, kScanItems / 4><<<one, kScanOneThreads, 0, s>>>(a);
  } else if (a.n <= kScanOne / 2) {
    k_scan_one<Tin, Tout, kScanItems / 2><<<one, kScanOneThreads, 0, s>>>(a);
  } else if (a.n <= kScanOne) {
    k_scan_one<Tin, Tout, kScanItems><<<one, kScanOneThreads, 0, s>>>(a);
  } else {
    const int64_t nt = (a.n + kScanTile - 1) / kScanTile;
    const dim3 g((unsigned)nt, count);
    k_tile_reduce<Tin, Tout><<<g, kScanThreads, 0, s>>>(a);
    k_scan_sums<Tout><<<dim3(1, count), 1024, 0, s>>>(a.sums, nt, a.out + a.n, a.sums_step,
                                                      a.out_step, a.totals);
    k_tile_scan<Tin, Tout><<<g, kScanThreads, 0, s>>>(a);
  }
  SPJ_CUDA(cudaGetLastError());
}

template <class Tin, class Tout>
void scan_into_impl(const Tin* in, Tout* out, int64_t n, Tout* sums, cudaStream_t s) {
  scan_launch<Tin, Tout>({in, out, sums, nullptr, n, 0, 0, 0}, 1, s);
}

template <class Tin, class Tout>
void scan_impl(const Tin* in, Tout* out, int64_t n, DevBuf& tmp, cudaStream_t s) {
  tmp.reserve(scan_tile_sums_bytes(n), s);
  scan_into_impl<Tin, Tout>(in, out, n, tmp.as<Tout>(), s);
}

// ---------------------------------------------------------------------------
// radix sort

constexpr int kSortThreads = 256;
constexpr int kSortItems = 8;
constexpr int kSortTile = kSortThreads * kSortItems;

// Place of (digit d, tile b) in the histogram table.  The tiles form
// segments of seg_tiles consecutive tiles (the last may be shorter); the
// table is segment-major, then digit-major, so its scan gives every item a
// place inside its own segment's range and a pass sorts each segment alone.
// seg_tiles = ntiles: one segment, the plain digit-major table.
__device__ __forceinline__ int64_t hist_slot(uint32_t d, int64_t b, int64_t ntiles,
                                             int64_t seg_tiles) {
  const int64_t b0 = b / seg_tiles * seg_tiles;
  const int64_t nb = min(seg_tiles, ntiles - b0);
  return b0 * 256 + (int64_t)d * nb + (b - b0);
}

__global__ void k_digit_hist(const uint32_t* __restrict__ keys, int64_t n, int shift,
                             uint32_t* __restrict__ hist, int64_t ntiles, int64_t seg_tiles) {
  __shared__ uint32_t h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kSortTile;
#pragma unroll
  for (int j = 0; j < kSortItems; j++) {
    int64_t i = base + j * kSortThreads + threadIdx.x;
    if (i < n) atomicAdd(&h[(keys[i] >> shift) & 0xFF], 1u);
  }
  __syncthreads();
  hist[hist_slot(threadIdx.x, blockIdx.x, ntiles, seg_tiles)] = h[threadIdx.x];
}

// The lanes whose digit (8 bits) is the lane's own; all 32 lanes call.  Eight
// ballots: one __match_any_sync took as long as some 70 instructions and held
// up the other warps of its SM (1M pairs: 22.3 us a pass of k_digit_scatter
// with it, 9.7 this way).
__device__ __forceinline__ unsigned same_digit(uint32_t d) {
  unsigned peers = 0xffffffffu;
#pragma unroll
  for (int b = 0; b < 8; b++) {
    const bool on = (d >> b) & 1u;
    const unsigned who = __ballot_sync(0xffffffffu, on);
    peers &= on ? who : ~who;
  }
  return peers;
}

// One 8-bit LSD pass over a tile of kSortTile items: stable local ranking by
// digit (warp w ranks its 256 items in 8 rounds of 32 with same_digit
// and per-warp digit counters; a scan over warps and digits gives each item
// its place in the tile's digit-sorted order), a reorder in shared memory,
// and a write of each digit run to its global offset (scan of the tile
// histograms, hist_slot).  Pads (past n) carry key 0xFFFFFFFF, so they rank
// last in digit 255 and land past the tile's valid items, which are all
// written.
__global__ void __launch_bounds__(kSortThreads)
    k_digit_scatter(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ vals,
                    int64_t n, int shift, const uint32_t* __restrict__ offs, int64_t ntiles,
                    int64_t seg_tiles, uint32_t* __restrict__ okeys,
                    uint32_t* __restrict__ ovals) {
  constexpr int kWarps = kSortThreads / 32;
  __shared__ uint32_t sk[kSortTile];
  __shared__ uint32_t sv[kSortTile];
  __shared__ uint32_t wcnt[kWarps][256];
  __shared__ uint32_t doff[256];
  __shared__ uint32_t gbase[256];
  __shared__ uint32_t scan_sm[9];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int t = threadIdx.x; t < kWarps * 256; t += kSortThreads) (&wcnt[0][0])[t] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kSortTile;
  const int cnt = (int)min((int64_t)kSortTile, n - base);
  uint32_t k[kSortItems], v[kSortItems], pos[kSortItems];
#pragma unroll
  for (int j = 0; j < kSortItems; j++) {
    const int li = w * (32 * kSortItems) + j * 32 + lane;  // warp-contiguous chunk
    const bool valid = li < cnt;
    k[j] = valid ? keys[base + li] : 0xFFFFFFFFu;
    v[j] = valid ? vals[base + li] : 0u;
    const uint32_t d = (k[j] >> shift) & 0xFFu;
    const unsigned peers = same_digit(d);
    const int leader = __ffs(peers) - 1;
    const uint32_t b = wcnt[w][d];
    __syncwarp();
    if (lane == leader) wcnt[w][d] = b + (uint32_t)__popc(peers);
    pos[j] = b + (uint32_t)__popc(peers & ((1u << lane) - 1u));
    __syncwarp();  // the counters' updates before the next round reads them
  }
  __syncthreads();
  {
    // thread t owns digit t: offsets of each warp's run inside the digit,
    // then the digit's offset inside the tile
    const int d = threadIdx.x;
    uint32_t run = 0;
#pragma unroll
    for (int ww = 0; ww < kWarps; ww++) {
      const uint32_t c = wcnt[ww][d];
      wcnt[ww][d] = run;
      run += c;
    }
    uint32_t total;
    doff[d] = block_exclusive_scan_256<uint32_t>(run, scan_sm, &total);
    gbase[d] = offs[hist_slot(d, blockIdx.x, ntiles, seg_tiles)];
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kSortItems; j++) {
    const uint32_t d = (k[j] >> shift) & 0xFFu;
    const uint32_t lp = doff[d] + wcnt[w][d] + pos[j];
    sk[lp] = k[j];
    sv[lp] = v[j];
  }
  __syncthreads();
  for (int li = threadIdx.x; li < cnt; li += kSortThreads) {
    const uint32_t key = sk[li];
    const uint32_t d = (key >> shift) & 0xFFu;
    const uint64_t dst = (uint64_t)gbase[d] + (uint32_t)(li - doff[d]);
    if (okeys) okeys[dst] = key;  // (null: the last pass of a sort whose keys are not kept)
    ovals[dst] = sv[li];
  }
}

// The whole sort of up to 1024 * kItems pairs by one block: keys and values
// stay in shared memory and registers over all passes (ranked per pass as in
// k_digit_scatter, 32 warps of 32 * kItems consecutive items).  A small sort
// is bound by its launches: 4,096 pairs took 5 of them and 29 us a pass, 3.8
// us this way.  Up to kSortOne pairs, where one SM's shared memory ends and so
// does the gain: 16,384 pairs take 12.3 us a pass, by tiles 14.
constexpr int kSortOneThreads = 1024;
constexpr int64_t kSortOne = 16 * kSortOneThreads;
constexpr size_t sort_one_smem(int items) {
  return (size_t)kSortOneThreads * items * 8 + 32 * 256 * 2 + 256 * 4;
}
template <int kItems>
__global__ void __launch_bounds__(kSortOneThreads)
    k_sort_one(uint32_t* __restrict__ keys, uint32_t* __restrict__ vals, int n, int key_bits,
               bool keys_out) {
  extern __shared__ __align__(16) uint32_t sort_smem[];
  uint32_t* sk = sort_smem;
  uint32_t* sv = sk + kSortOneThreads * kItems;
  uint32_t* doff = sv + kSortOneThreads * kItems;
  uint16_t* wcnt = reinterpret_cast<uint16_t*>(doff + 256);  // [warp][digit]
  __shared__ uint32_t scan_sm[9];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i0 = w * (32 * kItems) + lane;
  uint32_t k[kItems], v[kItems], pos[kItems];
#pragma unroll
  for (int j = 0; j < kItems; j++) {
    const int i = i0 + j * 32;
    k[j] = i < n ? keys[i] : 0xFFFFFFFFu;  // (pads stay behind every key)
    v[j] = i < n ? vals[i] : 0u;
  }
  for (int shift = 0; shift < key_bits; shift += 8) {
    uint32_t* zero = reinterpret_cast<uint32_t*>(wcnt);
    for (int t = threadIdx.x; t < 32 * 256 / 2; t += kSortOneThreads) zero[t] = 0;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kItems; j++) {
      const uint32_t d = (k[j] >> shift) & 0xFFu;
      const unsigned peers = same_digit(d);
      const uint32_t b = wcnt[w * 256 + d];
      __syncwarp();
      if (lane == __ffs(peers) - 1) wcnt[w * 256 + d] = (uint16_t)(b + __popc(peers));
      pos[j] = b + (uint32_t)__popc(peers & ((1u << lane) - 1u));
      __syncwarp();  // the counters' updates before the next round reads them
    }
    __syncthreads();
    uint32_t run = 0;
    if (threadIdx.x < 256) {
#pragma unroll
      for (int ww = 0; ww < 32; ww++) {
        const uint32_t c = wcnt[ww * 256 + threadIdx.x];
        wcnt[ww * 256 + threadIdx.x] = (uint16_t)run;
        run += c;
      }
      const uint32_t inc = warp_inclusive_scan(run);
      if (lane == 31) scan_sm[w] = inc;
      run = inc - run;
    }
    __syncthreads();
    if (threadIdx.x < 256) {
      for (int ww = 0; ww < w; ww++) run += scan_sm[ww];
      doff[threadIdx.x] = run;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kItems; j++) {
      const uint32_t d = (k[j] >> shift) & 0xFFu;
      const uint32_t to = doff[d] + wcnt[w * 256 + d] + pos[j];
      sk[to] = k[j];
      sv[to] = v[j];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kItems; j++) {
      k[j] = sk[i0 + j * 32];
      v[j] = sv[i0 + j * 32];
    }
  }
#pragma unroll
  for (int j = 0; j < kItems; j++) {
    const int i = i0 + j * 32;
    if (i < n) {
      if (keys_out) keys[i] = k[j];
      vals[i] = v[j];
    }
  }
}

template <int kItems>
void sort_one(uint32_t* keys, uint32_t* vals, int64_t n, int key_bits, bool keys_out,
              cudaStream_t s) {
  constexpr size_t smem = sort_one_smem(kItems);
  SPJ_CUDA(cudaFuncSetAttribute(k_sort_one<kItems>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)smem));
  k_sort_one<kItems><<<1, kSortOneThreads, smem, s>>>(keys, vals, (int)n, key_bits, keys_out);
  SPJ_CUDA(cudaGetLastError());
}

}  // namespace

void scan_u32_u64_many(const uint32_t* in, int64_t in_step, uint64_t* out, int64_t out_step,
                       int64_t n, int count, uint64_t* totals, DevBuf& tmp, cudaStream_t s) {
  const int64_t step = (int64_t)(scan_tile_sums_bytes(n) / sizeof(uint64_t));
  tmp.reserve((size_t)count * step * sizeof(uint64_t), s);
  scan_launch<uint32_t, uint64_t>({in, out, tmp.as<uint64_t>(), totals, n, in_step, out_step, step},
                                  (unsigned)count, s);
}
void scan_u32_u64(const uint32_t* in, uint64_t* out, int64_t n, DevBuf& tmp, cudaStream_t s) {
  scan_impl<uint32_t, uint64_t>(in, out, n, tmp, s);
}
void scan_u8_u64(const uint8_t* in, uint64_t* out, int64_t n, DevBuf& tmp, cudaStream_t s) {
  scan_impl<uint8_t, uint64_t>(in, out, n, tmp, s);
}
size_t scan_tile_sums_bytes(int64_t n) {
  int64_t nt = (n + kScanTile - 1) / kScanTile;
  return (size_t)((nt < 1 ? 1 : nt) + 1) * sizeof(uint64_t);
}

void scan_u32_u64_into(const uint32_t* in, uint64_t* out, int64_t n, uint64_t* sums,
                       cudaStream_t s) {
  scan_into_impl<uint32_t, uint64_t>(in, out, n, sums, s);
}

void scan_u32_u32(const uint32_t* in, uint32_t* out, int64_t n, DevBuf& tmp, cudaStream_t s) {
  scan_impl<uint32_t, uint32_t>(in, out, n, tmp, s);
}

size_t compact_sums_bytes(int64_t n) {
  const int64_t nt = (n + kScanTile - 1) / kScanTile;
  return (size_t)((nt < 1 ? 1 : nt) + 1) * sizeof(uint64_t);
}

void compact_count(const uint8_t* flags, int64_t n, uint64_t* sums, cudaStream_t s) {
  if (n <= 0) {
    SPJ_CUDA(cudaMemsetAsync(sums, 0, sizeof(uint64_t), s));
    return;
  }
  const int64_t nt = (n + kScanTile - 1) / kScanTile;
  k_tile_reduce<uint8_t, uint64_t>
      <<<(unsigned)nt, kScanThreads, 0, s>>>({flags, nullptr, sums, nullptr, n, 0, 0, 0});
  k_scan_sums<uint64_t><<<1, 1024, 0, s>>>(sums, nt, sums + nt, 0, 0, nullptr);
  SPJ_CUDA(cudaGetLastError());
}

void compact_pairs_tiles(const uint32_t* cb, const uint32_t* cp, const uint8_t* flags, int64_t n,
                         const uint64_t* sums, uint32_t* ob, uint32_t* op, uint64_t out_cap,
                         cudaStream_t s) {
  if (n <= 0) return;
  const int64_t nt = (n + kScanTile - 1) / kScanTile;
  k_compact_tile<<<(unsigned)nt, kScanThreads, 0, s>>>(cb, cp, flags, n, sums, ob, op, out_cap);
  SPJ_CUDA(cudaGetLastError());
}

int scan_launches(int64_t n) { return n <= kScanOne ? 1 : 3; }

int radix_sort_launches(int64_t n, int key_bits) {
  if (n <= kSortOne) return 1;
  return (key_bits + 7) / 8 * (2 + scan_launches((n + kSortTile - 1) / kSortTile * 256));
}

size_t radix_sort_tmp_bytes(int64_t n) {
  const int64_t ntiles = (n + kSortTile - 1) / kSortTile;
  const int64_t nh = 256 * (ntiles < 1 ? 1 : ntiles);
  const int64_t nt = (nh + kScanTile - 1) / kScanTile;
  return (size_t)(2 * nh + 1 + nt + 1) * sizeof(uint32_t);
}

void radix_sort_pairs(uint32_t* keys, uint32_t* vals, uint32_t* alt_keys, uint32_t* alt_vals,
                      int64_t n, int key_bits, DevBuf& tmp, cudaStream_t s, int64_t segments,
                      bool keys_out) {
  if (n <= 1) return;
  SPJ_CHECK(n < (int64_t)0xFFFFFFFF, "radix sort: too many keys");
  if (n <= kSortOne && segments <= 1) {
    if (n <= 4 * kSortOneThreads) sort_one<4>(keys, vals, n, key_bits, keys_out, s);
    else if (n <= 8 * kSortOneThreads) sort_one<8>(keys, vals, n, key_bits, keys_out, s);
    else sort_one<16>(keys, vals, n, key_bits, keys_out, s);
    return;
  }
  const int64_t ntiles = (n + kSortTile - 1) / kSortTile;
  const int64_t seg_tiles =
      segments > 1 ? (ntiles + segments - 1) / segments : ntiles;
  const int64_t nh = 256 * ntiles;
  // histogram table, its scan, and the scan's tile sums, all in tmp (no
  // allocation when tmp already holds radix_sort_tmp_bytes(n): graph capture)
  tmp.reserve(radix_sort_tmp_bytes(n), s);
  uint32_t* hist = tmp.as<uint32_t>();
  uint32_t* offs = hist + nh;
  uint32_t* sums = offs + nh + 1;
  uint32_t *ik = keys, *iv = vals, *ok = alt_keys, *ov = alt_vals;
  int passes = 0;
  for (int shift = 0; shift < key_bits; shift += 8) {
    const bool last = shift + 8 >= key_bits;
    k_digit_hist<<<(unsigned)ntiles, kSortThreads, 0, s>>>(ik, n, shift, hist, ntiles,
                                                           seg_tiles);
    scan_into_impl<uint32_t, uint32_t>(hist, offs, nh, sums, s);
    k_digit_scatter<<<(unsigned)ntiles, kSortThreads, 0, s>>>(
        ik, iv, n, shift, offs, ntiles, seg_tiles, last && !keys_out ? nullptr : ok, ov);
    SPJ_CUDA(cudaGetLastError());
    std::swap(ik, ok);
    std::swap(iv, ov);
    passes++;
  }
  if (passes & 1) {
    if (keys_out) SPJ_CUDA(cudaMemcpyAsync(keys, ik, n * 4, cudaMemcpyDeviceToDevice, s));
    SPJ_CUDA(cudaMemcpyAsync(vals, iv, n * 4, cudaMemcpyDeviceToDevice, s));
  }
}

const char* status_message(uint32_t code) {
  switch (code) {
    case kOk: return "ok";
    case kWkbTruncated: return "invalid WKB (truncated)";
    case kWkbByteOrder: return "invalid WKB (byte order)";
    case kWkbType: return "unsupported WKB geometry type";
    case kWkbDims: return "only 2D WKB geometries are supported";
    case kWkbCount: return "invalid WKB (count)";
    case kOverflow: return "output capacity exceeded";
    case kUnsupported: return "predicate not supported for these geometry types";
  }
  return "unknown device error";
}

}  // namespace spj
