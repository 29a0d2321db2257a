// materialize.cu — result materialisation on the device: the column gathers
// that build the joined batch from the refined pairs (the reference's
// build_batch_from_indices / assemble_partial_build_batch on the host,
// rust/sedona-spatial-join/src/stream.rs:1466-1580, an Arrow take per
// column), and the build side's visited bitmap of outer, semi and anti joins
// (rust/sedona-spatial-join/src/utils/join_utils.rs:53-62,
// SpatialIndex::visited_build_side).  Indices equal to SPJ_NULL_INDEX
// produce a null row (the unmatched side of an outer join).
//
// All HBM-bound: a gathered fixed-width value reads its width once and writes
// it once (the index 4 B); a binary value reads and writes its bytes once,
// with a length pass, a scan and a copy pass (a lane group per value, the
// destination written as whole 4-byte words whatever the alignments).
// SpjGatherColumns takes the columns of a batch together: one launch for all
// values, lengths and validity words, and one wait for all sizes.
#include <errno.h>

#include <algorithm>
#include <string>
#include <vector>

#include "../../include/spj_gb300.h"
#include "common.cuh"
#include "materialize.cuh"
#include "prims.cuh"

namespace spj {
namespace {

thread_local std::string g_error;

int fail(const std::exception& e) {
  g_error = e.what();
  return EINVAL;
}

// One column of a gather.  Fixed width: values -> out; binary (width 0): the
// rows' lengths -> len; validity words -> out_valid and the count of null rows
// -> *nulls, where asked for.
struct GatherCol {
  const uint32_t* idx = nullptr;
  uint64_t n = 0;
  const void* values = nullptr;  // fixed width: the values; binary: the offsets
  uint64_t n_values = 0;
  uint32_t width = 0;
  int off64 = 0;
  void* out = nullptr;
  uint32_t* len = nullptr;
  const uint8_t* valid = nullptr;
  int64_t voff = 0;
  uint64_t n_valid = 0;
  uint32_t* out_valid = nullptr;
  unsigned long long* nulls = nullptr;
};
constexpr uint32_t kGatherCols = 8;
template <uint32_t kCols>
struct GatherCols {
  GatherCol c[kCols];
};
constexpr int kGatherRows = 4;  // rows of a lane in flight

template <class T>
__device__ __forceinline__ void gather_rows(const GatherCol& c, const uint32_t* j, uint64_t i) {
  T v[kGatherRows];
#pragma unroll
  for (int u = 0; u < kGatherRows; u++) {
    v[u] = T{};
    if (j[u] != SPJ_NULL_INDEX && j[u] < c.n_values) v[u] = static_cast<const T*>(c.values)[j[u]];
  }
#pragma unroll
  for (int u = 0; u < kGatherRows; u++)
    if (i + u * 32 < c.n) static_cast<T*>(c.out)[i + u * 32] = v[u];
}

template <bool kOff64>
__device__ __forceinline__ void bin_range(const void* off, uint32_t j, uint64_t& s, uint64_t& e) {
  if (kOff64) {
    const int64_t* o = static_cast<const int64_t*>(off);
    s = (uint64_t)o[j];
    e = (uint64_t)o[j + 1];
  } else {
    const int32_t* o = static_cast<const int32_t*>(off);
    s = (uint64_t)(uint32_t)o[j];
    e = (uint64_t)(uint32_t)o[j + 1];
  }
}

template <bool kOff64>
__device__ __forceinline__ void gather_lengths(const GatherCol& c, const uint32_t* j, uint64_t i) {
  uint32_t l[kGatherRows];
#pragma unroll
  for (int u = 0; u < kGatherRows; u++) {
    uint64_t s = 0, e = 0;
    if (j[u] != SPJ_NULL_INDEX && j[u] < c.n_values) bin_range<kOff64>(c.values, j[u], s, e);
    l[u] = e > s ? (uint32_t)(e - s) : 0;
  }
#pragma unroll
  for (int u = 0; u < kGatherRows; u++)
    if (i + u * 32 < c.n) c.len[i + u * 32] = l[u];
}

// Column blockIdx.y: a warp takes 128 rows at a time, a lane 4 of them 32
// apart, so the index, the output and the validity word (a ballot of 32 rows)
// are coalesced and 4 gathered values are in flight.  Bound by L2 and HBM: 4M
// rows, 5 columns with validity, 171 us in passes of their own (32 rows per
// thread for the validity words), 63 this way.
template <uint32_t kCols>
__global__ void __launch_bounds__(256)
    k_gather_columns(const __grid_constant__ GatherCols<kCols> cols) {
  const GatherCol& c = cols.c[blockIdx.y];
  const int lane = threadIdx.x & 31;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  uint32_t nulls = 0;
  for (uint64_t i0 = ((blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5) * (32 * kGatherRows);
       i0 < c.n; i0 += nwarps * (32 * kGatherRows)) {
    const uint64_t i = i0 + lane;
    uint32_t j[kGatherRows];
#pragma unroll
    for (int u = 0; u < kGatherRows; u++)
      j[u] = i + u * 32 < c.n ? c.idx[i + u * 32] : SPJ_NULL_INDEX;
    if (c.out) {
      switch (c.width) {
        case 1: gather_rows<uint8_t>(c, j, i); break;
        case 2: gather_rows<uint16_t>(c, j, i); break;
        case 4: gather_rows<uint32_t>(c, j, i); break;
        case 8: gather_rows<uint64_t>(c, j, i); break;
        default: gather_rows<uint4>(c, j, i); break;
      }
    } else if (c.len) {
      if (c.off64) gather_lengths<true>(c, j, i);
      else gather_lengths<false>(c, j, i);
    }
    if (c.out_valid) {
#pragma unroll
      for (int u = 0; u < kGatherRows; u++) {
        const bool row = i + u * 32 < c.n;
        bool ok = j[u] != SPJ_NULL_INDEX && j[u] < c.n_valid;
        if (ok && c.valid) {
          const uint64_t bit = (uint64_t)c.voff + j[u];
          ok = (c.valid[bit >> 3] >> (bit & 7)) & 1;
        }
        const uint32_t word = __ballot_sync(0xffffffffu, ok);
        nulls += row && !ok ? 1u : 0u;
        if (lane == 0 && row) c.out_valid[(i >> 5) + u] = word;
      }
    }
  }
  if (c.out_valid) {
    for (int o = 16; o > 0; o >>= 1) nulls += __shfl_xor_sync(0xffffffffu, nulls, o);
    if (lane == 0 && nulls) atomicAdd(c.nulls, (unsigned long long)nulls);
  }
}

template <uint32_t kCols>
void launch_gather(const GatherCol* c, unsigned m, cudaStream_t s) {
  GatherCols<kCols> a;
  uint64_t most = 0;
  for (unsigned q = 0; q < m; q++) {
    a.c[q] = c[q];
    most = std::max(most, c[q].n);
  }
  if (most == 0) return;
  const int g = grid_for((int64_t)(most + kGatherRows - 1) / kGatherRows, 256, kNumSMs * 8);
  k_gather_columns<kCols><<<dim3((unsigned)g, m), 256, 0, s>>>(a);
  SPJ_CUDA(cudaGetLastError());
}

// (a column alone is launched without the parameters of eight, which cost a
// short call 2 of 30 us)
void gather_columns(const GatherCol* c, size_t count, cudaStream_t s) {
  if (count == 1) return launch_gather<1>(c, 1, s);
  for (size_t k = 0; k < count; k += kGatherCols)
    launch_gather<kGatherCols>(c + k, (unsigned)std::min<size_t>(kGatherCols, count - k), s);
}

// A warp takes 32 values: lane k reads value k's index, source range and
// output position (one memory latency for all 32), then lane groups of G
// copy a value each (group_copy_once: whole destination words, any alignment).
// Bound by the requests to L1 and the latency of each value; two or four
// values of a group in flight cost more in registers than they hid (4M WKB
// values of 157 bytes: 220 and 403 us), as did the warp's run of the output in
// 16-byte blocks (346 us).
template <bool kOff64, int G, int U>
__global__ void __launch_bounds__(256)
    k_bin_copy(const void* __restrict__ off, const uint8_t* __restrict__ data,
               const uint32_t* __restrict__ idx, uint64_t n, uint64_t nsrc,
               const int64_t* __restrict__ pos, uint8_t* __restrict__ out, uint64_t cap) {
  const int lane = threadIdx.x & 31, grp = lane / G, gl = lane % G;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t i0 = (((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32; i0 < n;
       i0 += nwarps * 32) {
    const uint64_t i = i0 + lane;
    uint64_t s = 0, d = 0;
    uint32_t l = 0;
    if (i < n) {
      const uint32_t j = idx[i];
      if (j != SPJ_NULL_INDEX && j < nsrc) {
        uint64_t e;
        bin_range<kOff64>(off, j, s, e);
        d = (uint64_t)pos[i];
        l = e > s ? (uint32_t)(e - s) : 0;
        if (d + l > cap) l = 0;  // bounded by the output buffer
      }
    }
    for (int k = 0; k < 32; k += 32 / G) {
      const uint64_t vs = __shfl_sync(0xffffffffu, s, k + grp);
      const uint64_t vd = __shfl_sync(0xffffffffu, d, k + grp);
      const uint32_t vl = __shfl_sync(0xffffffffu, l, k + grp);
      if (vl) group_copy_once<G, U>(data + vs, out + vd, vl, gl);
    }
  }
}

// Copies the gathered values of n rows to out (positions: the output offsets;
// total bytes, at most cap of them written).  Values of up to 32 bytes on
// average by groups of 4 lanes, which take 32 bytes in one go, longer ones by
// groups of 8, which take 224: 4M names of 14 bytes 73 and 143 us, 4M WKB
// values of 157 bytes 267 and 196 us.
void copy_values(const void* off, bool off64, const uint8_t* data, uint64_t n_values,
                 const uint32_t* idx, uint64_t n, const int64_t* pos, uint64_t total, uint8_t* out,
                 uint64_t cap, cudaStream_t s) {
  if (!n || !total) return;
  const int g = grid_for((int64_t)n, 256, kNumSMs * 16);
  const auto copy = total <= n * 32 ? (off64 ? k_bin_copy<true, 4, 2> : k_bin_copy<false, 4, 2>)
                                    : (off64 ? k_bin_copy<true, 8, 7> : k_bin_copy<false, 8, 7>);
  copy<<<g, 256, 0, s>>>(off, data, idx, n, n_values, pos, out, cap);
  SPJ_CUDA(cudaGetLastError());
}

__global__ void k_mark(uint32_t* __restrict__ bits, uint64_t nbuild,
                       const uint32_t* __restrict__ ids, uint64_t n) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t b = ids[i];
    if (b >= nbuild) continue;
    const uint32_t w = b >> 5, m = 1u << (b & 31);
    if (!(bits[w] & m)) atomicOr(&bits[w], m);  // read first: most marks repeat
  }
}

// rows whose bit equals want, in ascending order: per 32-row word a count,
// a scan, then the rows
__global__ void k_bits_count(const uint32_t* __restrict__ bits, uint64_t nbuild, uint32_t want,
                             uint32_t* __restrict__ cnt) {
  const uint64_t nw = (nbuild + 31) / 32;
  for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < nw;
       w += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t v = want ? bits[w] : ~bits[w];
    const uint64_t rem = nbuild - w * 32;
    if (rem < 32) v &= (1u << rem) - 1u;
    cnt[w] = __popc(v);
  }
}

__global__ void k_bits_rows(const uint32_t* __restrict__ bits, uint64_t nbuild, uint32_t want,
                            const uint64_t* __restrict__ pos, uint32_t* __restrict__ out,
                            uint64_t cap) {
  const uint64_t nw = (nbuild + 31) / 32;
  for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < nw;
       w += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t v = want ? bits[w] : ~bits[w];
    const uint64_t rem = nbuild - w * 32;
    if (rem < 32) v &= (1u << rem) - 1u;
    uint64_t p = pos[w];
    while (v) {
      const int b = __ffs(v) - 1;
      v &= v - 1;
      if (p < cap) out[p] = (uint32_t)(w * 32 + b);
      p++;
    }
  }
}

cudaStream_t as_stream(void* s) { return static_cast<cudaStream_t>(s); }

bool aligned(const void* p, size_t a) { return reinterpret_cast<uintptr_t>(p) % a == 0; }

}  // namespace

uint64_t gather_binary(const WkbDeviceColumn& col, const uint32_t* d_idx, uint64_t n,
                       DevBuf& out_off, DevBuf& out_data, DevBuf& scratch_len, DevBuf& scan_tmp,
                       cudaStream_t s) {
  scratch_len.reserve(((size_t)n + 1) * 4, s);
  out_off.reserve(((size_t)n + 1) * 8, s);
  GatherCol c;
  c.idx = d_idx;
  c.n = n;
  c.values = col.offsets;
  c.n_values = (uint64_t)col.n;
  c.off64 = col.offsets64;
  c.len = scratch_len.as<uint32_t>();
  gather_columns(&c, 1, s);
  scan_u32_u64(c.len, out_off.as<uint64_t>(), (int64_t)n, scan_tmp, s);
  uint64_t total = 0;
  SPJ_CUDA(cudaMemcpyAsync(&total, out_off.as<uint64_t>() + n, 8, cudaMemcpyDeviceToHost, s));
  SPJ_CUDA(cudaStreamSynchronize(s));
  out_data.reserve(total + 16, s);
  copy_values(col.offsets, col.offsets64, col.data, (uint64_t)col.n, d_idx, n,
              out_off.as<int64_t>(), total, out_data.as<uint8_t>(), total, s);
  SPJ_CUDA(cudaStreamSynchronize(s));
  return total;
}

void gather_u64(const uint64_t* values, uint64_t n_values, const uint32_t* d_idx, uint64_t n,
                uint64_t* out, cudaStream_t s) {
  GatherCol c;
  c.idx = d_idx;
  c.n = n;
  c.values = values;
  c.n_values = n_values;
  c.width = 8;
  c.out = out;
  gather_columns(&c, 1, s);
}

}  // namespace spj

using namespace spj;

extern "C" const char* SpjMaterializeLastError(void) { return g_error.c_str(); }

extern "C" int SpjGatherFixed(const void* d_values, uint32_t width, uint64_t n_values,
                              const uint32_t* d_idx, uint64_t n, void* d_out, void* stream) {
  try {
    SPJ_CHECK(n == 0 || (d_idx && d_out && (d_values || n_values == 0)), "null buffer");
    SPJ_CHECK(width == 1 || width == 2 || width == 4 || width == 8 || width == 16,
              "width must be 1, 2, 4, 8 or 16 bytes");
    SPJ_CHECK(aligned(d_values, width) && aligned(d_out, width) && aligned(d_idx, 4),
              "values and output must be aligned to the width, indices to 4 bytes");
    const cudaStream_t s = as_stream(stream);
    GatherCol c;
    c.idx = d_idx;
    c.n = n;
    c.values = d_values;
    c.n_values = n_values;
    c.width = width;
    c.out = d_out;
    gather_columns(&c, 1, s);
    SPJ_CUDA(cudaStreamSynchronize(s));
    g_error.clear();
    return 0;
  } catch (const std::exception& e) {
    return fail(e);
  }
}

extern "C" int SpjGatherValidity(const uint8_t* d_validity, int64_t validity_offset,
                                 uint64_t n_values, const uint32_t* d_idx, uint64_t n,
                                 uint8_t* d_out_bitmap, uint64_t* null_count, void* stream) {
  try {
    SPJ_CHECK(null_count != nullptr, "null null_count");
    SPJ_CHECK(n == 0 || (d_idx && d_out_bitmap), "null buffer");
    SPJ_CHECK(aligned(d_out_bitmap, 4) && aligned(d_idx, 4),
              "the output bitmap (written as 32-bit words) and the indices must be 4-byte "
              "aligned");
    const cudaStream_t s = as_stream(stream);
    DevBuf cnt(8, s);
    SPJ_CUDA(cudaMemsetAsync(cnt.get(), 0, 8, s));
    GatherCol c;
    c.idx = d_idx;
    c.n = n;
    c.valid = d_validity;
    c.voff = validity_offset;
    c.n_valid = n_values;
    c.out_valid = reinterpret_cast<uint32_t*>(d_out_bitmap);
    c.nulls = cnt.as<unsigned long long>();
    gather_columns(&c, 1, s);
    unsigned long long h = 0;
    SPJ_CUDA(cudaMemcpyAsync(&h, cnt.get(), 8, cudaMemcpyDeviceToHost, s));
    SPJ_CUDA(cudaStreamSynchronize(s));
    *null_count = h;
    g_error.clear();
    return 0;
  } catch (const std::exception& e) {
    return fail(e);
  }
}

extern "C" int SpjGatherBinary(const void* d_offsets, int32_t offsets_are_64bit,
                               const uint8_t* d_data, uint64_t n_values, const uint32_t* d_idx,
                               uint64_t n, int64_t* d_out_offsets, uint8_t* d_out_data,
                               uint64_t capacity, uint64_t* out_bytes, void* stream) {
  try {
    SPJ_CHECK(out_bytes != nullptr, "null out_bytes");
    SPJ_CHECK(d_out_offsets != nullptr && d_offsets != nullptr && (n == 0 || d_idx),
              "null buffer");
    SPJ_CHECK(aligned(d_offsets, offsets_are_64bit ? 8 : 4) && aligned(d_out_offsets, 8) &&
                  aligned(d_idx, 4),
              "offsets and indices must be aligned to their element size");
    const cudaStream_t s = as_stream(stream);
    DevBuf len(((size_t)n + 1) * 4, s), tmp;
    GatherCol c;
    c.idx = d_idx;
    c.n = n;
    c.values = d_offsets;
    c.n_values = n_values;
    c.off64 = offsets_are_64bit != 0;
    c.len = len.as<uint32_t>();
    gather_columns(&c, 1, s);
    scan_u32_u64(c.len, reinterpret_cast<uint64_t*>(d_out_offsets), (int64_t)n, tmp, s);
    uint64_t total = 0;
    SPJ_CUDA(cudaMemcpyAsync(&total, d_out_offsets + n, 8, cudaMemcpyDeviceToHost, s));
    SPJ_CUDA(cudaStreamSynchronize(s));
    *out_bytes = total;
    if (total > capacity) {
      g_error = "output capacity " + std::to_string(capacity) + " < " + std::to_string(total) +
                " bytes";
      return ENOSPC;
    }
    if (n && total) {
      SPJ_CHECK(d_out_data != nullptr && d_data != nullptr, "null data buffer");
      copy_values(d_offsets, offsets_are_64bit != 0, d_data, n_values, d_idx, n, d_out_offsets,
                  total, d_out_data, capacity, s);
    }
    SPJ_CUDA(cudaStreamSynchronize(s));
    g_error.clear();
    return 0;
  } catch (const std::exception& e) {
    return fail(e);
  }
}

extern "C" int SpjGatherColumns(SpjGatherColumn* cols, uint32_t n_cols, void* stream) {
  try {
    SPJ_CHECK(n_cols == 0 || cols != nullptr, "null columns");
    const cudaStream_t s = as_stream(stream);
    uint64_t lens = 0;
    for (uint32_t k = 0; k < n_cols; k++) {
      const SpjGatherColumn& c = cols[k];
      SPJ_CHECK(c.n == 0 || (c.d_idx && c.d_out_validity), "null buffer");
      SPJ_CHECK(aligned(c.d_out_validity, 4) && aligned(c.d_idx, 4),
                "the output bitmap (written as 32-bit words) and the indices must be 4-byte "
                "aligned");
      if (c.d_offsets) {
        SPJ_CHECK(c.d_out_offsets != nullptr, "null buffer");
        SPJ_CHECK(aligned(c.d_offsets, c.offsets_are_64bit ? 8 : 4) && aligned(c.d_out_offsets, 8),
                  "offsets and indices must be aligned to their element size");
        lens += c.n + 1;
      } else {
        SPJ_CHECK(c.n == 0 || (c.d_out_values && (c.d_values || c.n_values == 0)), "null buffer");
        SPJ_CHECK(c.width == 1 || c.width == 2 || c.width == 4 || c.width == 8 || c.width == 16,
                  "width must be 1, 2, 4, 8 or 16 bytes");
        SPJ_CHECK(aligned(c.d_values, c.width) && aligned(c.d_out_values, c.width),
                  "values and output must be aligned to the width, indices to 4 bytes");
      }
    }
    // per column: null rows, then data bytes
    std::vector<unsigned long long> h(2 * (size_t)n_cols + 1);
    DevBuf cnt(h.size() * 8, s), len(lens * 4, s), tmp;
    SPJ_CUDA(cudaMemsetAsync(cnt.get(), 0, h.size() * 8, s));
    std::vector<GatherCol> g(n_cols);
    uint64_t at = 0;
    for (uint32_t k = 0; k < n_cols; k++) {
      const SpjGatherColumn& c = cols[k];
      g[k].idx = c.d_idx;
      g[k].n = c.n;
      g[k].n_values = c.n_values;
      if (c.d_offsets) {
        g[k].values = c.d_offsets;
        g[k].off64 = c.offsets_are_64bit != 0;
        g[k].len = len.as<uint32_t>() + at;
        at += c.n + 1;
      } else {
        g[k].values = c.d_values;
        g[k].width = c.width;
        g[k].out = c.d_out_values;
      }
      g[k].valid = c.d_validity;
      g[k].voff = c.validity_offset;
      g[k].n_valid = c.n_validity;
      g[k].out_valid = reinterpret_cast<uint32_t*>(c.d_out_validity);
      g[k].nulls = cnt.as<unsigned long long>() + 2 * k;
    }
    gather_columns(g.data(), n_cols, s);
    for (uint32_t k = 0; k < n_cols; k++)
      if (g[k].len)
        scan_u32_u64_many(g[k].len, 0, reinterpret_cast<uint64_t*>(cols[k].d_out_offsets), 0,
                          (int64_t)g[k].n, 1, cnt.as<uint64_t>() + 2 * k + 1, tmp, s);
    SPJ_CUDA(cudaMemcpyAsync(h.data(), cnt.get(), h.size() * 8, cudaMemcpyDeviceToHost, s));
    SPJ_CUDA(cudaStreamSynchronize(s));
    for (uint32_t k = 0; k < n_cols; k++) {
      cols[k].null_count = h[2 * k];
      cols[k].out_bytes = h[2 * k + 1];
    }
    g_error.clear();
    return 0;
  } catch (const std::exception& e) {
    return fail(e);
  }
}

extern "C" int SpjGatherColumnsData(const SpjGatherColumn* cols, uint32_t n_cols, void* stream) {
  try {
    SPJ_CHECK(n_cols == 0 || cols != nullptr, "null columns");
    const cudaStream_t s = as_stream(stream);
    for (uint32_t k = 0; k < n_cols; k++) {
      const SpjGatherColumn& c = cols[k];
      if (!c.d_offsets || !c.n || !c.out_bytes) continue;
      SPJ_CHECK(c.d_out_data != nullptr && c.d_data != nullptr, "null data buffer");
      copy_values(c.d_offsets, c.offsets_are_64bit != 0, c.d_data, c.n_values, c.d_idx, c.n,
                  c.d_out_offsets, c.out_bytes, c.d_out_data, c.out_bytes, s);
    }
    SPJ_CUDA(cudaStreamSynchronize(s));
    g_error.clear();
    return 0;
  } catch (const std::exception& e) {
    return fail(e);
  }
}

extern "C" int SpjVisitedMark(uint32_t* d_bitmap, uint64_t n_build, const uint32_t* d_build_idx,
                              uint64_t n, void* stream) {
  try {
    SPJ_CHECK(n == 0 || n_build == 0 || (d_bitmap && d_build_idx), "null buffer");
    SPJ_CHECK(aligned(d_bitmap, 4) && aligned(d_build_idx, 4), "buffers must be 4-byte aligned");
    const cudaStream_t s = as_stream(stream);
    if (n && n_build)
      k_mark<<<grid_for((int64_t)n, 256, kNumSMs * 16), 256, 0, s>>>(d_bitmap, n_build,
                                                                      d_build_idx, n);
    SPJ_CUDA(cudaGetLastError());
    SPJ_CUDA(cudaStreamSynchronize(s));
    g_error.clear();
    return 0;
  } catch (const std::exception& e) {
    return fail(e);
  }
}

extern "C" int SpjVisitedCollect(const uint32_t* d_bitmap, uint64_t n_build, int32_t visited,
                                 uint32_t* d_out_idx, uint64_t capacity, uint64_t* count,
                                 void* stream) {
  try {
    SPJ_CHECK(count != nullptr, "null count");
    SPJ_CHECK(aligned(d_bitmap, 4) && aligned(d_out_idx, 4), "buffers must be 4-byte aligned");
    const cudaStream_t s = as_stream(stream);
    const uint64_t nw = (n_build + 31) / 32;
    DevBuf cnt((nw + 1) * 4, s), pos((nw + 1) * 8, s), tmp;
    const int g = grid_for((int64_t)nw, 256, kNumSMs * 16);
    if (nw) {
      SPJ_CHECK(d_bitmap != nullptr, "null bitmap");
      k_bits_count<<<g, 256, 0, s>>>(d_bitmap, n_build, visited ? 1u : 0u, cnt.as<uint32_t>());
    }
    scan_u32_u64(cnt.as<uint32_t>(), pos.as<uint64_t>(), (int64_t)nw, tmp, s);
    uint64_t total = 0;
    SPJ_CUDA(cudaMemcpyAsync(&total, pos.as<uint64_t>() + nw, 8, cudaMemcpyDeviceToHost, s));
    SPJ_CUDA(cudaStreamSynchronize(s));
    *count = total;
    if (total > capacity) {
      g_error = "output capacity " + std::to_string(capacity) + " < " + std::to_string(total) +
                " rows";
      return ENOSPC;
    }
    if (nw && total) {
      SPJ_CHECK(d_out_idx != nullptr, "null output");
      k_bits_rows<<<g, 256, 0, s>>>(d_bitmap, n_build, visited ? 1u : 0u, pos.as<uint64_t>(),
                                    d_out_idx, capacity);
    }
    SPJ_CUDA(cudaGetLastError());
    SPJ_CUDA(cudaStreamSynchronize(s));
    g_error.clear();
    return 0;
  } catch (const std::exception& e) {
    return fail(e);
  }
}
