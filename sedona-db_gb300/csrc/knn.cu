// knn.cu — KNN join: LBVH over the build points, depth-first traversal
// nearest child first, a register-resident best list per probe thread,
// probes taken in Morton order of their coordinates (one traversal per probe,
// or one per 32 neighbouring probes where these are dense enough).
//
// Ranking key: the exact squared distance dx^2 + dy^2 of the FP64 deltas
// dx = RN(b.x - p.x), dy = RN(b.y - p.y) (the deltas the reference's
// Euclidean distance forms), held as a normalized double-double (hi, lo) and
// compared lexicographically, then by build id.  Exact duplicates tie on the
// key and fall back to the build id, as in the reference ground truth.
//
// Chosen form (k <= 16): every coordinate is split into an FP32 pair
// hi = RN32(v), lo = RN32(v - hi), and the traversal ranks points by the FP32
// squared distance of (b.hi - q.hi) + (b.lo - q.lo), whose error is a few
// ulps of the distance itself plus 2^-44 of the coordinate magnitude (the
// bound is derived at kSplitRel below).  It keeps the k+1 best; when the
// (k+1)-th is provably farther than each of the first k (their error
// intervals are disjoint), the k-set is exact, and only those k points get
// the FP64 key that orders them.  Probes whose k-set is not proven this way
// (near ties at rank k, exact duplicates) are queued for the exact kernel.
// Plain form: every visited point gets the FP64 key.
#include "knn.cuh"
#include "prims.cuh"

#include <cmath>
#include <vector>

namespace spj {
namespace {

constexpr int kKnnThreads = 128;
constexpr int kKnnStack = 64;

// |true distance - sqrt(d2)| <= kSplitRel * sqrt(d2) + cerr, cerr =
// 2^-44 (max|b.x|+|b.y| + |q.x|+|q.y|) + 2^-120, for the split FP32 distance
// d2.  Per axis, with u = 2^-24: b = hi + lo + e, |e| <= 2^-48 |b|; the three
// FP32 roundings give |dx - (b - q).x| <= 2u |dx| (1 + 2u) + 3 * 2^-48 (|b.x| +
// |q.x|); the two axes add to <= 2^-22 * |d| + 2^-46 (..); squaring, summing
// and the square root add 2^-23 relative.  kSplitRel = 2^-20 covers the
// relative part twice over, 2^-44 the absolute part four times over, and
// 2^-120 the absolute error of FP32 results below the normal range.
constexpr float kSplitUp = 1.00000095367431640625f;    // 1 + 2^-20
constexpr float kSplitDown = 0.99999904632568359375f;  // 1 - 2^-20
constexpr float kTwoM44 = 5.684341886080801486968994140625e-14f;
constexpr float kTwoM120 = 7.5231638452626400509999138382223723380394595633413601376560e-37f;
// coordinates up to this magnitude keep every split FP32 square finite
constexpr double kSplitMaxCoord = 1e18;

__device__ __forceinline__ void two_sum(double a, double b, double& s, double& e) {
  s = __dadd_rn(a, b);
  const double bb = __dsub_rn(s, a);
  e = __dadd_rn(__dsub_rn(a, __dsub_rn(s, bb)), __dsub_rn(b, bb));
}

// exact dx^2 + dy^2 as a normalized double-double
__device__ __forceinline__ void sq_dist_dd(double2 b, double2 p, double& hi, double& lo) {
  const double dx = __dsub_rn(b.x, p.x), dy = __dsub_rn(b.y, p.y);
  const double a1 = __dmul_rn(dx, dx), a2 = __fma_rn(dx, dx, -a1);
  const double b1 = __dmul_rn(dy, dy), b2 = __fma_rn(dy, dy, -b1);
  double s, e;
  two_sum(a1, b1, s, e);
  e = __dadd_rn(e, __dadd_rn(a2, b2));
  two_sum(s, e, hi, lo);
}

__device__ __forceinline__ bool key_less(double h1, double l1, uint32_t i1, double h2, double l2,
                                         uint32_t i2) {
  if (h1 != h2) return h1 < h2;
  if (l1 != l2) return l1 < l2;
  return i1 < i2;
}

// lower bound of the FP32 distance from q to box b (0 inside)
__device__ __forceinline__ float box_dist(float2 q, float4 b) {
  const float dx = fmaxf(fmaxf(b.x - q.x, q.x - b.z), 0.0f);
  const float dy = fmaxf(fmaxf(b.y - q.y, q.y - b.w), 0.0f);
  return __fsqrt_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)));
}

__device__ __forceinline__ void write_empty(uint32_t* out_idx, double* out_dist, uint64_t qi,
                                            uint32_t k) {
  for (uint32_t j = 0; j < k; j++) {
    out_idx[qi * k + j] = 0xFFFFFFFFu;
    out_dist[qi * k + j] = INFINITY;
  }
}

// Exact kernel.  With `order`, thread slot j serves probe order[j]; with
// n_dev, the slot count is read from device memory (the queue the split
// kernel filled).
template <int K, bool kFast>
__global__ void __launch_bounds__(kKnnThreads)
    k_knn(LbvhView t, const double2* __restrict__ bxy, const double2* __restrict__ probe,
          uint64_t n, const uint32_t* __restrict__ order, const uint32_t* __restrict__ n_dev,
          uint32_t k, float slack, uint32_t* __restrict__ out_idx, double* __restrict__ out_dist,
          unsigned long long* __restrict__ exact_evals) {
  __shared__ int stack[kKnnStack * kKnnThreads];
  const uint64_t max_steps = 2ull * t.nleaves + 2;
  uint32_t evals = 0;
  const uint64_t nn = n_dev ? (uint64_t)*n_dev : n;
  for (uint64_t j = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; j < nn;
       j += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t qi = order ? (uint64_t)order[j] : j;
    if (qi >= n) {
      traversal_fault(t, kBadProbe, (unsigned)qi);
      continue;
    }
    const double2 q = probe[qi];
    const float2 q32 = make_float2(__double2float_rn(q.x), __double2float_rn(q.y));
    // |q - q32| bound, plus the build-side bound
    const float qs = __fadd_ru(__fmul_ru(fabsf(q32.x) + fabsf(q32.y), 1.1920929e-07f), slack);
    double kh[K], kl[K];
    uint32_t ki[K];
#pragma unroll
    for (int c = 0; c < K; c++) {
      kh[c] = INFINITY;
      kl[c] = 0;
      ki[c] = 0xFFFFFFFFu;
    }
    uint32_t have = 0;
    float bound = INFINITY;  // FP32 upper bound of the k-th best distance
    const bool valid = !(isnan(q.x) || isnan(q.y)) && t.nprims > 0;
    int sp = 0;
    int node = valid ? (t.nleaves > 1 ? 0 : ~0) : 0;
    bool done = !valid;
    uint64_t steps = 0;
    while (!done) {
      if (++steps > max_steps) {  // each node is visited at most once
        traversal_fault(t, kTooLong, (unsigned)qi);
        break;
      }
      if (node < 0) {
        const uint32_t c = (uint32_t)(~node);
        if (c >= t.nleaves) {
          traversal_fault(t, kBadLeaf, c);
          break;
        }
        const uint32_t b0 = c * t.leaf_size, b1 = min(b0 + t.leaf_size, t.nprims);
        for (uint32_t pi = b0; pi < b1; pi++) {
          const double2 b = bxy[pi];
          if (kFast && have >= k) {
            const float4 pb = t.sorted_box[pi];  // RN32 of the point
            const float fx = __fsub_rn(pb.x, q32.x), fy = __fsub_rn(pb.y, q32.y);
            const float d32 = __fsqrt_rn(__fadd_rn(__fmul_rn(fx, fx), __fmul_rn(fy, fy)));
            const float mag = fabsf(pb.x) + fabsf(q32.x) + fabsf(pb.y) + fabsf(q32.y) +
                              fabsf(fx) + fabsf(fy);
            const float err = __fadd_ru(__fmul_ru(mag, 2.384185791015625e-07f),
                                        __fmul_ru(d32, 4.76837158203125e-07f));
            if (__fsub_rd(d32, err) > bound) continue;  // provably farther than the k-th
          }
          double h, l;
          sq_dist_dd(b, q, h, l);
          evals++;
          const uint32_t id = t.sorted_id[pi];
          if (have >= k && !key_less(h, l, id, kh[K - 1], kl[K - 1], ki[K - 1])) continue;
          // insert into the sorted register list
          bool placed = false;
#pragma unroll
          for (int c2 = K - 1; c2 > 0; c2--) {
            if (!placed) {
              if (key_less(h, l, id, kh[c2 - 1], kl[c2 - 1], ki[c2 - 1])) {
                kh[c2] = kh[c2 - 1];
                kl[c2] = kl[c2 - 1];
                ki[c2] = ki[c2 - 1];
              } else {
                kh[c2] = h;
                kl[c2] = l;
                ki[c2] = id;
                placed = true;
              }
            }
          }
          if (!placed) {
            kh[0] = h;
            kl[0] = l;
            ki[0] = id;
          }
          if (have < k) have++;
          if (have >= k) {
            // k-th entry of the list sits at index k-1 (k <= K)
            double kth = kh[K - 1];
#pragma unroll
            for (int c2 = 0; c2 < K; c2++)
              if (c2 == (int)k - 1) kth = __dadd_rn(kh[c2], kl[c2]);
            bound = __double2float_ru(sqrt(kth) * (1.0 + 1e-12));
          }
        }
      } else {
        if ((uint32_t)node + 1 >= t.nleaves) {
          traversal_fault(t, kBadNode, (unsigned)node);
          break;
        }
        const float4 lb = t.node_box[2 * node], rb = t.node_box[2 * node + 1];
        const int2 ch = t.node_child[node];
        // conservative lower bounds of the true distance
        const float dl = __fsub_rd(__fmul_rd(box_dist(q32, lb), 0.99999905f), qs);
        const float dr = __fsub_rd(__fmul_rd(box_dist(q32, rb), 0.99999905f), qs);
        const bool vl = dl <= bound, vr = dr <= bound;
        if (vl && vr) {
          const int nearc = dl <= dr ? ch.x : ch.y;
          const int farc = dl <= dr ? ch.y : ch.x;
          if (sp >= kKnnStack) {  // deeper than any tree built here: record, stop
            traversal_fault(t, kStackOverflow, (unsigned)qi);
            break;
          }
          stack[sp * kKnnThreads + threadIdx.x] = farc;
          sp++;
          node = nearc;
          continue;
        }
        if (vl) {
          node = ch.x;
          continue;
        }
        if (vr) {
          node = ch.y;
          continue;
        }
      }
      // pop, skipping subtrees the bound now excludes is left to the next
      // visit (the node test re-checks the bound)
      if (sp == 0) break;
      sp--;
      node = stack[sp * kKnnThreads + threadIdx.x];
    }
    for (uint32_t c = 0; c < k; c++) {
      uint32_t id = 0xFFFFFFFFu;
      double d = INFINITY;
#pragma unroll
      for (int cc = 0; cc < K; cc++)
        if (cc == (int)c && cc < (int)have) {
          id = ki[cc];
          d = sqrt(__dadd_rn(kh[cc], kl[cc]));
        }
      out_idx[qi * k + c] = id;
      out_dist[qi * k + c] = d;
    }
  }
  for (int o = 16; o > 0; o >>= 1) evals += __shfl_xor_sync(0xffffffffu, evals, o);
  if ((threadIdx.x & 31) == 0 && evals) atomicAdd(exact_evals, (unsigned long long)evals);
}

// A probe point split for the FP32 tier (see kSplitRel): its (hi, lo) pair,
// the slack of a box test against the build boxes, and the absolute part of
// the distance error.
struct SplitProbe {
  double2 q;
  float hx, hy, lx, ly;
  float qs, cerr;
  __device__ __forceinline__ void set(double2 p, float slack, float bmag) {
    q = p;
    hx = __double2float_rn(p.x);
    hy = __double2float_rn(p.y);
    // p - RN32(p) is exact in FP64
    lx = __double2float_rn(__dsub_rn(p.x, (double)hx));
    ly = __double2float_rn(__dsub_rn(p.y, (double)hy));
    qs = __fadd_ru(__fmul_ru(fabsf(hx) + fabsf(hy), 1.1920929e-07f), slack);
    cerr = __fadd_ru(__fmul_ru(__fadd_ru(bmag, __fadd_ru(fabsf(hx), fabsf(hy))), kTwoM44),
                     kTwoM120);
  }
  __device__ __forceinline__ float dist2(float4 h) const {
    const float dx = __fadd_rn(__fsub_rn(h.x, hx), __fsub_rn(h.z, lx));
    const float dy = __fadd_rn(__fsub_rn(h.y, hy), __fsub_rn(h.w, ly));
    return __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
  }
  // upper bound of the true distance whose split distance squared is d2
  __device__ __forceinline__ float upper(float d2) const {
    return __fadd_ru(__fmul_ru(__fsqrt_ru(d2), kSplitUp), cerr);
  }
  __device__ __forceinline__ float lower(float d2) const {
    return __fsub_rd(__fmul_rd(__fsqrt_rd(d2), kSplitDown), cerr);
  }
};

// Puts (d2, pi) into the K+1 smallest split distances seen (ascending, after
// equal ones).  No branches: every lane of a warp runs the same selects, and
// a distance past the list's end changes nothing.
template <int K>
__device__ __forceinline__ void list_insert(float (&ld)[K + 1], uint32_t (&lp)[K + 1], float d2,
                                            uint32_t pi) {
  bool below = d2 < ld[K];
#pragma unroll
  for (int c = K; c > 0; c--) {
    const bool next = d2 < ld[c - 1];  // implies below
    lp[c] = next ? lp[c - 1] : (below ? pi : lp[c]);
    ld[c] = next ? ld[c - 1] : (below ? d2 : ld[c]);
    below = next;
  }
  lp[0] = below ? pi : lp[0];
  ld[0] = below ? d2 : ld[0];
}

template <int K>
__device__ __forceinline__ float list_at(const float (&ld)[K + 1], uint32_t i) {
  float v = ld[0];
#pragma unroll
  for (int c = 1; c <= K; c++)
    if (c == (int)i) v = ld[c];
  return v;
}

// A probe's place in the queue of another kernel: its row and, for the exact one
// (else null), an upper bound of its k-th distance.
struct KnnQueue {
  uint32_t* rows;
  float* bound;
  uint32_t* count;
  __device__ __forceinline__ void push(uint64_t qi, float b) const {
    const uint32_t at = atomicAdd(count, 1u);
    rows[at] = (uint32_t)qi;
    if (bound) bound[at] = b;
  }
};

// Insertion sort of kk sorted-point positions by (exact key, build id);
// returns the number of exact keys computed.
__device__ __noinline__ uint32_t sort_by_key(const LbvhView& t, const double2* bxy, double2 q,
                                             uint32_t* pos, uint32_t kk) {
  uint32_t evals = 0;
  for (uint32_t i = 1; i < kk; i++) {
    const uint32_t p = pos[i], id = t.sorted_id[p];
    double h, l;
    sq_dist_dd(bxy[p], q, h, l);
    evals++;
    uint32_t j = i;
    for (; j > 0; j--) {
      const uint32_t o = pos[j - 1];
      double oh, ol;
      sq_dist_dd(bxy[o], q, oh, ol);
      evals++;
      if (!key_less(h, l, id, oh, ol, t.sorted_id[o])) break;
      pos[j] = o;
    }
    pos[j] = p;
  }
  return evals;
}

// The end of a split probe: the k-set is proven or queued, ordered by the
// exact keys and written.  have: list entries, capped at k + 1.
template <int K>
__device__ __forceinline__ void split_finish(const LbvhView& t, const double2* __restrict__ bxy,
                                             const SplitProbe& sp, float (&ld)[K + 1],
                                             uint32_t (&lp)[K + 1], uint32_t have, uint32_t k,
                                             uint64_t qi, uint32_t* __restrict__ out_idx,
                                             double* __restrict__ out_dist,
                                             const KnnQueue& queue, uint32_t& evals) {
  // With fewer than k+1 entries the bound never closed, so every build
  // point was visited and listed.  Otherwise the k-set is proven when the
  // (k+1)-th entry's lower bound exceeds the k-th entry's upper bound (the
  // list is ascending, so the k-th bounds the first k).
  if (have > k) {
    const float up = sp.upper(list_at<K>(ld, k - 1)), dk1 = list_at<K>(ld, k);
    if (!(sp.lower(dk1) > up)) {
      queue.push(qi, up);
      return;
    }
  }
  // Order of the proven set by (exact key, build id).  The list is already
  // ascending in the split distance; when the error intervals of neighbours
  // are all disjoint that is the exact order.  Else (near ties, duplicates)
  // the list is sorted by its exact keys.  (That sort is a loop out of line:
  // unrolled into a transposition network it was K^2/2 copies of the exact
  // arithmetic: 4M probes x 400k points with k_knn_packet, k = 16: 21.3 ms,
  // 6.3 with the loop; k = 8: 4.3 and 3.9.)
  const uint32_t kk = min(k, have);
  bool ordered = true;
#pragma unroll
  for (int c = 0; c + 1 < K; c++)
    if (c + 1 < (int)kk && !(sp.upper(ld[c]) < sp.lower(ld[c + 1]))) ordered = false;
  if (!ordered) {
    uint32_t pos[K];
#pragma unroll
    for (int c = 0; c < K; c++) pos[c] = lp[c];
    evals += sort_by_key(t, bxy, sp.q, pos, kk);
#pragma unroll
    for (int c = 0; c < K; c++) lp[c] = pos[c];
  }
  // distances in FP64 from the reference's deltas (within a few ulps of
  // the exact value; the order above is exact)
#pragma unroll
  for (int c = 0; c < K; c++) {
    if (c >= (int)k) continue;
    uint32_t id = 0xFFFFFFFFu;
    double dist = INFINITY;
    if (c < (int)kk) {
      id = t.sorted_id[lp[c]];
      const double2 b = bxy[lp[c]];
      const double dx = __dsub_rn(b.x, sp.q.x), dy = __dsub_rn(b.y, sp.q.y);
      dist = __dsqrt_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)));
    }
    out_idx[qi * k + c] = id;
    out_dist[qi * k + c] = dist;
  }
}

// Split-FP32 kernel (chosen form): see the file comment.  hl[pi] holds the
// sorted build point pi as (hi.x, hi.y, lo.x, lo.y); bmag bounds |b.x|+|b.y|
// over the build side.  Probes whose k-set is not proven are queued for
// k_knn_queued, those past the split range (big) for k_knn, their outputs
// left to them.  With n_dev, the slot count is read from device memory (the
// rows that k_knn_packet passed on).
template <int K>
__global__ void __launch_bounds__(kKnnThreads)
    k_knn_split(LbvhView t, const float4* __restrict__ hl, const double2* __restrict__ bxy,
                const double2* __restrict__ probe, uint64_t n, const uint32_t* __restrict__ order,
                const uint32_t* __restrict__ n_dev, uint32_t k, float slack, float bmag,
                uint32_t* __restrict__ out_idx, double* __restrict__ out_dist, KnnQueue queue,
                KnnQueue big, unsigned long long* __restrict__ exact_evals) {
  __shared__ int stack[kKnnStack * kKnnThreads];
  const uint64_t max_steps = 2ull * t.nleaves + 2;
  const uint64_t nn = n_dev ? min((uint64_t)*n_dev, n) : n;
  uint32_t evals = 0;
  for (uint64_t j = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; j < nn;
       j += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t qi = order ? (uint64_t)order[j] : j;
    if (qi >= n) {
      traversal_fault(t, kBadProbe, (unsigned)qi);
      continue;
    }
    const double2 q = probe[qi];
    if (isnan(q.x) || isnan(q.y) || t.nprims == 0) {
      write_empty(out_idx, out_dist, qi, k);
      continue;
    }
    if (!(fabs(q.x) <= kSplitMaxCoord && fabs(q.y) <= kSplitMaxCoord)) {
      big.push(qi, INFINITY);
      continue;
    }
    SplitProbe s;
    s.set(q, slack, bmag);
    const float2 q32 = make_float2(s.hx, s.hy);
    // the K+1 smallest split distances seen, ascending
    float ld[K + 1];
    uint32_t lp[K + 1];
#pragma unroll
    for (int c = 0; c <= K; c++) {
      ld[c] = INFINITY;
      lp[c] = 0xFFFFFFFFu;
    }
    uint32_t have = 0;       // list entries, capped at k + 1
    float bound = INFINITY;  // upper bound of the true distance of the (k+1)-th entry
    int sp = 0;
    int node = t.nleaves > 1 ? 0 : ~0;
    uint64_t steps = 0;
    while (true) {
      if (++steps > max_steps) {  // each node is visited at most once
        traversal_fault(t, kTooLong, (unsigned)qi);
        break;
      }
      if (node < 0) {
        const uint32_t c = (uint32_t)(~node);
        if (c >= t.nleaves) {
          traversal_fault(t, kBadLeaf, c);
          break;
        }
        const uint32_t b0 = c * t.leaf_size, b1 = min(b0 + t.leaf_size, t.nprims);
        for (uint32_t pi = b0; pi < b1; pi++) {
          const float d2 = s.dist2(hl[pi]);
          if (!(d2 < ld[K])) continue;
          list_insert<K>(ld, lp, d2, pi);
          if (have <= k) have++;
          if (have > k) bound = s.upper(list_at<K>(ld, k));
        }
      } else {
        if ((uint32_t)node + 1 >= t.nleaves) {
          traversal_fault(t, kBadNode, (unsigned)node);
          break;
        }
        const float4 lb = t.node_box[2 * node], rb = t.node_box[2 * node + 1];
        const int2 ch = t.node_child[node];
        const float dl = __fsub_rd(__fmul_rd(box_dist(q32, lb), 0.99999905f), s.qs);
        const float dr = __fsub_rd(__fmul_rd(box_dist(q32, rb), 0.99999905f), s.qs);
        const bool vl = dl <= bound, vr = dr <= bound;
        if (vl && vr) {
          const int nearc = dl <= dr ? ch.x : ch.y;
          const int farc = dl <= dr ? ch.y : ch.x;
          if (sp >= kKnnStack) {  // deeper than any tree built here: record, stop
            traversal_fault(t, kStackOverflow, (unsigned)qi);
            break;
          }
          stack[sp * kKnnThreads + threadIdx.x] = farc;
          sp++;
          node = nearc;
          continue;
        }
        if (vl) {
          node = ch.x;
          continue;
        }
        if (vr) {
          node = ch.y;
          continue;
        }
      }
      if (sp == 0) break;
      sp--;
      node = stack[sp * kKnnThreads + threadIdx.x];
    }
    split_finish<K>(t, bxy, s, ld, lp, have, k, qi, out_idx, out_dist, queue, evals);
  }
  for (int o = 16; o > 0; o >>= 1) evals += __shfl_xor_sync(0xffffffffu, evals, o);
  if ((threadIdx.x & 31) == 0 && evals) atomicAdd(exact_evals, (unsigned long long)evals);
}

// The same with one traversal per warp: 32 probes that are neighbours in the
// Morton order walk the tree together.  A node is opened when any of them
// wants it, boxes and points are loaded once for all, and every lane keeps
// its own list and bound, so the results are those of k_knn_split.  The
// union of the 32 searches is a little larger than one of them where the
// probes are about as dense as the build points, and no lane idles (one
// traversal per thread is bound by divergence and by the latency of its own
// node loads).  Times of a query of 4M / 1M / 400k / 100k probes x 400k
// clustered points, k = 8: 3.7 / 1.75 / 1.26 / 1.01 ms against 6.9 / 2.7 /
// 1.39 / 0.81 with k_knn_split; k = 16: 7.0 / 3.1 / 2.2 / 1.8 against 12.6 /
// 4.8 / 2.5 / 1.6; k = 1: 1.93 / 0.88 / 0.66 / 0.54 against 3.5 / 1.28 / 0.73 /
// 0.44.  So queries take it from as many probes as build points on.
//
// A warp whose 32 probes lie apart (across a gap of the Morton order, in a
// cluster's thin tail) would walk the union of unlike searches while the
// rest of the grid has finished: past most_steps nodes its probes go to the
// wide queue and k_knn_split takes them one by one.  k = 8, 400k probes:
// 1.98 ms without that limit, 1.26 with 256, 1.38 with 128 and 768.
constexpr uint32_t kPacketSteps = 256;
template <int K>
__global__ void __launch_bounds__(kKnnThreads)
    k_knn_packet(LbvhView t, const float4* __restrict__ hl, const double2* __restrict__ bxy,
                 const double2* __restrict__ probe, uint64_t n,
                 const uint32_t* __restrict__ order, uint32_t k, float slack, float bmag,
                 uint32_t* __restrict__ out_idx, double* __restrict__ out_dist, KnnQueue queue,
                 KnnQueue big, KnnQueue wide, uint32_t most_steps,
                 unsigned long long* __restrict__ exact_evals) {
  __shared__ int stacks[kKnnThreads / 32][kKnnStack];
  const unsigned all = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  int* stack = stacks[threadIdx.x >> 5];
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  uint32_t evals = 0;
  for (uint64_t w = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; w * 32 < n;
       w += nwarps) {
    const uint64_t j = w * 32 + lane;
    uint64_t qi = j < n ? (uint64_t)order[j] : n;
    if (j < n && qi >= n) traversal_fault(t, kBadProbe, (unsigned)qi);
    bool act = qi < n;
    double2 q = make_double2(0.0, 0.0);
    if (act) {
      q = probe[qi];
      if (isnan(q.x) || isnan(q.y) || t.nprims == 0) {
        write_empty(out_idx, out_dist, qi, k);
        act = false;
      } else if (!(fabs(q.x) <= kSplitMaxCoord && fabs(q.y) <= kSplitMaxCoord)) {
        big.push(qi, INFINITY);
        act = false;
      }
    }
    if (!__any_sync(all, act)) continue;
    SplitProbe s;
    s.set(act ? q : make_double2(0.0, 0.0), slack, bmag);
    if (!act) s.hx = __int_as_float(0x7fc00000);  // distances of NaN: nothing is listed
    float ld[K + 1];
    uint32_t lp[K + 1];
#pragma unroll
    for (int c = 0; c <= K; c++) {
      ld[c] = INFINITY;
      lp[c] = 0xFFFFFFFFu;
    }
    uint32_t have = 0;
    // a box is wanted while its FP32 distance squared is at most reach: the
    // test dist * (1 - 2^-20) - qs <= bound of k_knn_split, rounded up
    float reach = act ? INFINITY : -1.0f;
    const float hx = act ? s.hx : 0.0f, hy = s.hy;
    auto gap2 = [&](const float4 b) {
      const float dx = fmaxf(fmaxf(b.x - hx, hx - b.z), 0.0f);
      const float dy = fmaxf(fmaxf(b.y - hy, hy - b.w), 0.0f);
      return __fadd_rd(__fmul_rd(dx, dx), __fmul_rd(dy, dy));
    };
    int sp = 0;
    int node = t.nleaves > 1 ? 0 : ~0;
    uint32_t steps = 0;
    bool apart = false;
    while (true) {
      if (++steps > most_steps) {
        apart = true;
        break;
      }
      if (node < 0) {
        const uint32_t c = (uint32_t)(~node);
        if (c >= t.nleaves) {
          if (lane == 0) traversal_fault(t, kBadLeaf, c);
          break;
        }
        const uint32_t b0 = c * t.leaf_size, b1 = min(b0 + t.leaf_size, t.nprims);
        uint32_t listed = 0;
        for (uint32_t p0 = b0; p0 < b1; p0 += 4) {
          float4 h[4];
#pragma unroll
          for (int u = 0; u < 4; u++) h[u] = hl[min(p0 + u, b1 - 1)];
#pragma unroll
          for (int u = 0; u < 4; u++) {
            const float d2 = s.dist2(h[u]);
            const bool put = p0 + u < b1 && d2 < ld[K];
            if (__any_sync(all, put)) {
              list_insert<K>(ld, lp, put ? d2 : INFINITY, p0 + u);
              listed += put ? 1u : 0u;
            }
          }
        }
        if (listed) {
          have = min(have + listed, k + 1);
          if (have > k) {
            const float bound = s.upper(list_at<K>(ld, k));
            const float r = __fmul_ru(__fadd_ru(bound, s.qs), 1.000002f);
            reach = __fmul_ru(r, r);
          }
        }
      } else {
        if ((uint32_t)node + 1 >= t.nleaves) {
          if (lane == 0) traversal_fault(t, kBadNode, (unsigned)node);
          break;
        }
        const float4 lb = t.node_box[2 * node], rb = t.node_box[2 * node + 1];
        const int2 ch = t.node_child[node];
        const float dl = gap2(lb), dr = gap2(rb);
        const unsigned vl = __ballot_sync(all, dl <= reach);
        const unsigned vr = __ballot_sync(all, dr <= reach);
        if (vl && vr) {
          // the child that is nearer for more lanes first
          const unsigned ln = __ballot_sync(all, act && dl <= dr);
          const unsigned rn = __ballot_sync(all, act && dr < dl);
          const bool left = __popc(ln) >= __popc(rn);
          if (sp >= kKnnStack) {  // deeper than any tree built here: record, stop
            if (lane == 0) traversal_fault(t, kStackOverflow, (unsigned)w);
            break;
          }
          if (lane == 0) stack[sp] = left ? ch.y : ch.x;
          sp++;
          node = left ? ch.x : ch.y;
          continue;
        }
        if (vl | vr) {
          node = vl ? ch.x : ch.y;
          continue;
        }
      }
      // next node that a lane still wants (a leaf is tested against its box;
      // an inner node's children are, once it is opened)
      bool more = false;
      while (sp > 0) {
        __syncwarp();
        sp--;
        node = stack[sp];
        if (node >= 0 || (uint32_t)(~node) >= t.nleaves ||
            __any_sync(all, gap2(t.leaf_box[~node]) <= reach)) {
          more = true;
          break;
        }
      }
      __syncwarp();
      if (!more) break;
    }
    if (act) {
      if (apart)
        wide.push(qi, INFINITY);
      else
        split_finish<K>(t, bxy, s, ld, lp, have, k, qi, out_idx, out_dist, queue, evals);
    }
    __syncwarp();
  }
  for (int o = 16; o > 0; o >>= 1) evals += __shfl_xor_sync(all, evals, o);
  if (lane == 0 && evals) atomicAdd(exact_evals, (unsigned long long)evals);
}

// Exact kernel for the queued probes, a warp each: the lanes take up to 32
// open nodes at a time from the warp's stack, each keeps the best of the
// points it sees, and the 32 lists are merged at the end.  The split pass's
// upper bound of the k-th distance prunes from the start.  Such a probe sits
// on near ties, often thousands of equal points; one thread alone walked
// them one after the other while the rest of the GPU had finished (4M probes
// x 400k points, k = 8, some 150 queued: 2.3 ms, now under 0.1).
constexpr int kQueueStack = 1024;

template <int K>
__global__ void __launch_bounds__(kKnnThreads)
    k_knn_queued(LbvhView t, const double2* __restrict__ bxy, const double2* __restrict__ probe,
                 uint64_t n, KnnQueue queue, uint32_t k, float slack,
                 uint32_t* __restrict__ out_idx, double* __restrict__ out_dist,
                 unsigned long long* __restrict__ exact_evals) {
  __shared__ int stacks[kKnnThreads / 32][kQueueStack];
  const unsigned all = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  int* stack = stacks[threadIdx.x >> 5];
  const uint64_t max_steps = 2ull * t.nleaves + 2;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint64_t nq = min((uint64_t)*queue.count, n);
  uint32_t evals = 0;
  for (uint64_t w = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; w < nq; w += nwarps) {
    const uint64_t qi = queue.rows[w];
    if (qi >= n) {
      if (lane == 0) traversal_fault(t, kBadProbe, (unsigned)qi);
      continue;
    }
    const double2 q = probe[qi];
    const float2 q32 = make_float2(__double2float_rn(q.x), __double2float_rn(q.y));
    const float qs = __fadd_ru(__fmul_ru(fabsf(q32.x) + fabsf(q32.y), 1.1920929e-07f), slack);
    float bound = queue.bound[w];
    double kh[K], kl[K];
    uint32_t ki[K];
#pragma unroll
    for (int c = 0; c < K; c++) {
      kh[c] = INFINITY;
      kl[c] = 0;
      ki[c] = 0xFFFFFFFFu;
    }
    uint32_t have = 0;
    int sp = 1;
    if (lane == 0) stack[0] = t.nleaves > 1 ? 0 : ~0;
    __syncwarp();
    uint64_t steps = 0;
    bool bad = false;
    while (sp > 0 && !bad) {
      if (++steps > max_steps) {  // every step takes at least one node
        if (lane == 0) traversal_fault(t, kTooLong, (unsigned)qi);
        break;
      }
      // a wide step adds at most 32 nodes to the stack; near its end single
      // steps (a depth-first walk of a tree of depth <= 64) cannot overflow
      const int take = sp > kQueueStack - 128 ? 1 : min(sp, 32);
      sp -= take;
      const int node = lane < take ? stack[sp + lane] : 0;
      __syncwarp();
      int push[2], npush = 0;
      if (lane < take) {
        if (node < 0) {
          const uint32_t c = (uint32_t)(~node);
          if (c >= t.nleaves) {
            traversal_fault(t, kBadLeaf, c);
            bad = true;
          } else {
            const uint32_t b0 = c * t.leaf_size, b1 = min(b0 + t.leaf_size, t.nprims);
            for (uint32_t pi = b0; pi < b1; pi++) {
              double h, l;
              sq_dist_dd(bxy[pi], q, h, l);
              evals++;
              const uint32_t id = t.sorted_id[pi];
              if (have >= k && !key_less(h, l, id, kh[K - 1], kl[K - 1], ki[K - 1])) continue;
              bool placed = false;
#pragma unroll
              for (int c2 = K - 1; c2 > 0; c2--) {
                if (!placed) {
                  if (key_less(h, l, id, kh[c2 - 1], kl[c2 - 1], ki[c2 - 1])) {
                    kh[c2] = kh[c2 - 1];
                    kl[c2] = kl[c2 - 1];
                    ki[c2] = ki[c2 - 1];
                  } else {
                    kh[c2] = h;
                    kl[c2] = l;
                    ki[c2] = id;
                    placed = true;
                  }
                }
              }
              if (!placed) {
                kh[0] = h;
                kl[0] = l;
                ki[0] = id;
              }
              if (have < k) have++;
            }
          }
        } else if ((uint32_t)node + 1 >= t.nleaves) {
          traversal_fault(t, kBadNode, (unsigned)node);
          bad = true;
        } else {
          const float4 lb = t.node_box[2 * node], rb = t.node_box[2 * node + 1];
          const int2 ch = t.node_child[node];
          const float dl = __fsub_rd(__fmul_rd(box_dist(q32, lb), 0.99999905f), qs);
          const float dr = __fsub_rd(__fmul_rd(box_dist(q32, rb), 0.99999905f), qs);
          if (dl <= bound) push[npush++] = ch.x;
          if (dr <= bound) push[npush++] = ch.y;
        }
      }
      const unsigned one = __ballot_sync(all, npush >= 1), two = __ballot_sync(all, npush == 2);
      const unsigned lower = (1u << lane) - 1u;
      const int at = sp + __popc(one & lower) + __popc(two & lower);
      const int total = __popc(one) + __popc(two);
      if (sp + total > kQueueStack) {
        if (lane == 0) traversal_fault(t, kStackOverflow, (unsigned)qi);
        break;
      }
      if (npush >= 1) stack[at] = push[0];
      if (npush == 2) stack[at + 1] = push[1];
      sp += total;
      bad = __any_sync(all, bad);
      __syncwarp();
    }
    // merge: k rounds of the smallest head of the 32 lists
    uint32_t my_id = 0xFFFFFFFFu;
    double my_d = INFINITY;
    for (uint32_t c = 0; c < k; c++) {
      double h = kh[0], l = kl[0];
      uint32_t id = ki[0];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const double oh = __shfl_xor_sync(all, h, o), ol = __shfl_xor_sync(all, l, o);
        const uint32_t oi = __shfl_xor_sync(all, id, o);
        if (key_less(oh, ol, oi, h, l, id)) {
          h = oh;
          l = ol;
          id = oi;
        }
      }
      if (id != 0xFFFFFFFFu && ki[0] == id) {  // the owner's list moves up
#pragma unroll
        for (int c2 = 0; c2 + 1 < K; c2++) {
          kh[c2] = kh[c2 + 1];
          kl[c2] = kl[c2 + 1];
          ki[c2] = ki[c2 + 1];
        }
        kh[K - 1] = INFINITY;
        kl[K - 1] = 0;
        ki[K - 1] = 0xFFFFFFFFu;
      }
      if (lane == (int)c) {
        my_id = id;
        my_d = id != 0xFFFFFFFFu ? sqrt(__dadd_rn(h, l)) : INFINITY;
      }
    }
    if (lane < (int)k) {
      out_idx[qi * k + lane] = my_id;
      out_dist[qi * k + lane] = my_d;
    }
    __syncwarp();
  }
  for (int o = 16; o > 0; o >>= 1) evals += __shfl_xor_sync(all, evals, o);
  if (lane == 0 && evals) atomicAdd(exact_evals, (unsigned long long)evals);
}

// Tie rows of include_tie_breakers (rust/sedona-spatial-join/src/index/
// default_spatial_index.rs:378-470): after a probe's k results come the
// build points outside them whose distance is within DISTANCE_TOLERANCE
// (1e-9, rust/sedona-spatial-join/src/index/spatial_index.rs:32) of the k-th
// distance, found as the reference finds them, by a box search around the
// probe.  A probe with fewer than k results has no ties.  The counting pass
// writes each probe's output length (its valid results plus its ties); the
// scatter pass writes the results, then the ties in traversal order.
constexpr double kTieTolerance = 1e-9;

template <bool kScatter>
__global__ void __launch_bounds__(kKnnThreads)
    k_knn_ties(LbvhView t, const double2* __restrict__ bxy, const double2* __restrict__ probe,
               uint64_t n, uint32_t k, bool ties, const uint32_t* __restrict__ kidx,
               const double* __restrict__ kdist, uint32_t* __restrict__ counts,
               const uint64_t* __restrict__ offs, uint32_t* __restrict__ out_idx,
               double* __restrict__ out_dist, uint64_t cap) {
  __shared__ int stack[kKnnStack * kKnnThreads];
  const uint64_t max_steps = 2ull * t.nleaves + 2;
  for (uint64_t qi = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; qi < n;
       qi += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t* ki = kidx + qi * k;
    uint32_t nvalid = 0;
    while (nvalid < k && ki[nvalid] != 0xFFFFFFFFu) nvalid++;
    uint64_t pos = kScatter ? offs[qi] : 0;
    if (kScatter) {
      for (uint32_t c = 0; c < nvalid; c++, pos++)
        if (pos < cap) {
          out_idx[pos] = ki[c];
          out_dist[pos] = kdist[qi * k + c];
        }
    }
    uint32_t cnt = 0;
    const double2 q = probe[qi];
    if (ties && nvalid == k && t.nprims > 0 && !(isnan(q.x) || isnan(q.y))) {
      const double kth = kdist[qi * k + k - 1];
      const double r = __dadd_ru(kth, kTieTolerance);
      // every build point within r of q has its RN32 box in this box
      const float4 qb = make_float4(__double2float_rd(__dsub_rd(q.x, r)),
                                    __double2float_rd(__dsub_rd(q.y, r)),
                                    __double2float_ru(__dadd_ru(q.x, r)),
                                    __double2float_ru(__dadd_ru(q.y, r)));
      int sp = 0;
      int node = t.nleaves > 1 ? 0 : ~0;
      uint64_t steps = 0;
      while (true) {
        if (++steps > max_steps) {
          traversal_fault(t, kTooLong, (unsigned)qi);
          break;
        }
        if (node < 0) {
          const uint32_t c = (uint32_t)(~node);
          if (c >= t.nleaves) {
            traversal_fault(t, kBadLeaf, c);
            break;
          }
          const uint32_t b0 = c * t.leaf_size, b1 = min(b0 + t.leaf_size, t.nprims);
          for (uint32_t kk = b0; kk < b1; kk++) {
            if (!box_overlap(t.sorted_box[kk], qb)) continue;
            const uint32_t id = t.sorted_id[kk];
            bool mine = false;
            for (uint32_t c2 = 0; c2 < k; c2++) mine |= ki[c2] == id;
            if (mine) continue;
            const double2 b = bxy[kk];
            const double dx = __dsub_rn(b.x, q.x), dy = __dsub_rn(b.y, q.y);
            const double dist = __dsqrt_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)));
            if (!(__dsub_rn(dist, kth) <= kTieTolerance)) continue;
            if (kScatter) {
              if (pos < cap) {
                out_idx[pos] = id;
                out_dist[pos] = dist;
              }
              pos++;
            } else {
              cnt++;
            }
          }
        } else {
          if ((uint32_t)node + 1 >= t.nleaves) {
            traversal_fault(t, kBadNode, (unsigned)node);
            break;
          }
          const float4 lb = t.node_box[2 * node], rb = t.node_box[2 * node + 1];
          const int2 ch = t.node_child[node];
          const bool hl = box_overlap(lb, qb), hr = box_overlap(rb, qb);
          if (hl && hr) {
            if (sp >= kKnnStack) {  // deeper than any tree built here: record, stop
              traversal_fault(t, kStackOverflow, (unsigned)qi);
              break;
            }
            stack[sp * kKnnThreads + threadIdx.x] = ch.y;
            sp++;
            node = ch.x;
            continue;
          }
          if (hl || hr) {
            node = hl ? ch.x : ch.y;
            continue;
          }
        }
        if (sp == 0) break;
        sp--;
        node = stack[sp * kKnnThreads + threadIdx.x];
      }
    }
    if (!kScatter) counts[qi] = nvalid + cnt;
  }
}

__global__ void k_points_to_boxes(const double2* __restrict__ xy, uint64_t n,
                                  float4* __restrict__ boxes) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const double2 p = xy[i];
    const float x = __double2float_rn(p.x), y = __double2float_rn(p.y);
    boxes[i] = make_float4(x, y, x, y);
  }
}

// sorted FP64 points and their (hi, lo) FP32 splits
__global__ void k_gather_xy(const double2* __restrict__ xy, const uint32_t* __restrict__ ids,
                            uint32_t m, double2* __restrict__ out, float4* __restrict__ hl) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
    const double2 p = xy[ids[i]];
    out[i] = p;
    const float hx = __double2float_rn(p.x), hy = __double2float_rn(p.y);
    hl[i] = make_float4(hx, hy, __double2float_rn(__dsub_rn(p.x, (double)hx)),
                        __double2float_rn(__dsub_rn(p.y, (double)hy)));
  }
}

}  // namespace

KnnIndex::KnnIndex(uint32_t leaf_size, int form) : leaf_size_(leaf_size), form_(form) {
  SPJ_CUDA(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking));
}

KnnIndex::~KnnIndex() {
  if (stream_) {
    cudaStreamSynchronize(stream_);
    bvh_ = Lbvh();
    xy_sorted_.release();
    xy_split_.release();
    probe_.release();
    oidx_.release();
    odist_.release();
    counters_.release();
    redo_.release();
    tie_probe_.release();
    tie_kidx_.release();
    tie_kdist_.release();
    tie_counts_.release();
    tie_offs_.release();
    tie_tmp_.release();
    tie_out_idx_.release();
    tie_out_dist_.release();
    osc_ = ProbeScratch();
    cudaStreamSynchronize(stream_);
    cudaStreamDestroy(stream_);
  }
}

void KnnIndex::build(const double* xy_host, uint64_t n) {
  SPJ_CHECK(n < 0xFFFFFFFFull, "too many build points");
  SPJ_CHECK(n == 0 || xy_host != nullptr, "null build points");
  cudaStream_t s = stream_;
  n_ = n;
  DevBuf xy((n + 1) * 16, s), boxes((n + 1) * 16, s);
  if (n) SPJ_CUDA(cudaMemcpyAsync(xy.get(), xy_host, n * 16, cudaMemcpyHostToDevice, s));
  k_points_to_boxes<<<grid_for((int64_t)n, 256), 256, 0, s>>>(xy.as<double2>(), n,
                                                               boxes.as<float4>());
  build_lbvh(boxes.as<float4>(), (uint32_t)n, leaf_size_, bvh_, s);
  xy_sorted_.reserve(((size_t)bvh_.nprims + 1) * 16, s);
  xy_split_.reserve(((size_t)bvh_.nprims + 1) * 16, s);
  if (bvh_.nprims)
    k_gather_xy<<<grid_for(bvh_.nprims, 256), 256, 0, s>>>(
        xy.as<double2>(), bvh_.sorted_id.as<uint32_t>(), bvh_.nprims, xy_sorted_.as<double2>(),
        xy_split_.as<float4>());
  // |p - RN32(p)| <= 2^-24 (|x| + |y|) <= 2^-24 * 2 * max|coord|
  double mx = 0, l1 = 0;
  bool split_ok = true;
  for (uint64_t i = 0; i < n; i++) {
    const double x = xy_host[2 * i], y = xy_host[2 * i + 1];
    if (std::isnan(x) || std::isnan(y)) continue;  // left out of the tree
    const double ax = std::fabs(x), ay = std::fabs(y);
    if (!(ax <= kSplitMaxCoord && ay <= kSplitMaxCoord)) split_ok = false;
    if (std::isfinite(ax) && ax > mx) mx = ax;
    if (std::isfinite(ay) && ay > mx) mx = ay;
    if (std::isfinite(ax + ay) && ax + ay > l1) l1 = ax + ay;
  }
  slack_ = (float)(mx * 2.0 * std::ldexp(1.0, -23));
  split_ok_ = split_ok;
  // rounded up so that it bounds max(|x| + |y|)
  bmag_ = (float)l1;
  if ((double)bmag_ < l1) bmag_ = std::nextafter(bmag_, INFINITY);
  SPJ_CUDA(cudaStreamSynchronize(s));
}

uint64_t KnnIndex::query_ties(const double* probe_xy, uint64_t n, uint32_t k, bool device_ptrs,
                              uint64_t* offsets, uint32_t* out_idx, double* out_dist,
                              uint64_t capacity, bool ties) {
  SPJ_CHECK(offsets != nullptr, "null offsets");
  cudaStream_t s = stream_;
  const double2* dp;
  if (device_ptrs) {
    dp = reinterpret_cast<const double2*>(probe_xy);
  } else {
    tie_probe_.reserve((n + 1) * 16, s);
    if (n) SPJ_CUDA(cudaMemcpyAsync(tie_probe_.get(), probe_xy, n * 16, cudaMemcpyHostToDevice, s));
    dp = tie_probe_.as<double2>();
  }
  tie_kidx_.reserve((n * k + 1) * 4, s);
  tie_kdist_.reserve((n * k + 1) * 8, s);
  query(reinterpret_cast<const double*>(dp), n, k, tie_kidx_.as<uint32_t>(),
        tie_kdist_.as<double>(), true);  // syncs
  tie_counts_.reserve((n + 1) * 4, s);
  tie_offs_.reserve((n + 1) * 8, s);
  const LbvhView t = bvh_.view();
  const int g = grid_for((int64_t)n, kKnnThreads, kNumSMs * 16);
  if (n)
    k_knn_ties<false><<<g, kKnnThreads, 0, s>>>(t, xy_sorted_.as<double2>(), dp, n, k, ties,
                                                 tie_kidx_.as<uint32_t>(), tie_kdist_.as<double>(),
                                                 tie_counts_.as<uint32_t>(), nullptr, nullptr,
                                                 nullptr, 0);
  scan_u32_u64(tie_counts_.as<uint32_t>(), tie_offs_.as<uint64_t>(), (int64_t)n, tie_tmp_, s);
  SPJ_CUDA(cudaMemcpyAsync(offsets, tie_offs_.get(), (n + 1) * 8, cudaMemcpyDeviceToHost, s));
  SPJ_CUDA(cudaStreamSynchronize(s));
  check_traversal(t, s);
  const uint64_t total = offsets[n];
  if (total > capacity || n == 0) return total;
  SPJ_CHECK(out_idx && out_dist, "null outputs");
  tie_out_idx_.reserve((total + 1) * 4, s);
  tie_out_dist_.reserve((total + 1) * 8, s);
  k_knn_ties<true><<<g, kKnnThreads, 0, s>>>(t, xy_sorted_.as<double2>(), dp, n, k, ties,
                                              tie_kidx_.as<uint32_t>(), tie_kdist_.as<double>(),
                                              nullptr, tie_offs_.as<uint64_t>(),
                                              tie_out_idx_.as<uint32_t>(),
                                              tie_out_dist_.as<double>(), total);
  SPJ_CUDA(cudaGetLastError());
  if (total) {
    SPJ_CUDA(cudaMemcpyAsync(out_idx, tie_out_idx_.get(), total * 4, cudaMemcpyDeviceToHost, s));
    SPJ_CUDA(cudaMemcpyAsync(out_dist, tie_out_dist_.get(), total * 8, cudaMemcpyDeviceToHost, s));
  }
  SPJ_CUDA(cudaStreamSynchronize(s));
  check_traversal(t, s);
  return total;
}

void KnnIndex::query(const double* probe_xy, uint64_t n, uint32_t k, uint32_t* out_idx,
                     double* out_dist, bool device_ptrs) {
  SPJ_CHECK(k >= 1 && k <= 32, "k must be in [1, 32]");
  SPJ_CHECK(n < 0xFFFFFFFFull, "too many probe points");
  cudaStream_t s = stream_;
  const double2* dp;
  uint32_t* di;
  double* dd;
  if (device_ptrs) {
    dp = reinterpret_cast<const double2*>(probe_xy);
    di = out_idx;
    dd = out_dist;
  } else {
    probe_.reserve((n + 1) * 16, s);
    oidx_.reserve((n * k + 1) * 4, s);
    odist_.reserve((n * k + 1) * 8, s);
    if (n) SPJ_CUDA(cudaMemcpyAsync(probe_.get(), probe_xy, n * 16, cudaMemcpyHostToDevice, s));
    dp = probe_.as<double2>();
    di = oidx_.as<uint32_t>();
    dd = odist_.as<double>();
  }
  counters_.reserve(24, s);
  SPJ_CUDA(cudaMemsetAsync(counters_.get(), 0, 24, s));
  if (n) {
    const LbvhView t = bvh_.view();
    const uint32_t* order = point_order(t, dp, (uint32_t)n, osc_, s);
    const int g = grid_for((int64_t)n, kKnnThreads, kNumSMs * 16);
    auto* ev = counters_.as<unsigned long long>();
    uint32_t* nredo = reinterpret_cast<uint32_t*>(ev + 1);
    if (form_ == 1 && k <= 16 && split_ok_) {
      // queues: near ties, probes past the split range, probes of warps whose
      // 32 searches lie apart
      const bool packet = order != nullptr && n >= bvh_.nprims;
      redo_.reserve((n + 1) * (packet ? 16 : 12), s);
      uint32_t* rows = redo_.as<uint32_t>();
      const KnnQueue queue{rows, reinterpret_cast<float*>(rows + (n + 1)), nredo};
      const KnnQueue big{rows + 2 * (n + 1), nullptr, nredo + 1};
      const KnnQueue wide{packet ? rows + 3 * (n + 1) : nullptr, nullptr, nredo + 2};
      const int gr = grid_for((int64_t)n, kKnnThreads, kNumSMs * 4);
#define SPJ_KNN_SPLIT(KK)                                                                        \
  if (packet)                                                                                    \
    k_knn_packet<KK><<<g, kKnnThreads, 0, s>>>(t, xy_split_.as<float4>(),                        \
                                               xy_sorted_.as<double2>(), dp, n, order, k,        \
                                               slack_, bmag_, di, dd, queue, big, wide,          \
                                               kPacketSteps, ev);                                \
  k_knn_split<KK><<<g, kKnnThreads, 0, s>>>(                                                     \
      t, xy_split_.as<float4>(), xy_sorted_.as<double2>(), dp, n, packet ? wide.rows : order,    \
      packet ? wide.count : nullptr, k, slack_, bmag_, di, dd, queue, big, ev);                  \
  k_knn_queued<KK><<<gr, kKnnThreads, 0, s>>>(t, xy_sorted_.as<double2>(), dp, n, queue, k,      \
                                              slack_, di, dd, ev);                               \
  k_knn<KK, false><<<gr, kKnnThreads, 0, s>>>(t, xy_sorted_.as<double2>(), dp, n, big.rows,      \
                                              big.count, k, slack_, di, dd, ev);
      if (k == 1) {
        SPJ_KNN_SPLIT(1)
      } else if (k <= 4) {
        SPJ_KNN_SPLIT(4)
      } else if (k <= 8) {
        SPJ_KNN_SPLIT(8)
      } else {
        SPJ_KNN_SPLIT(16)
      }
#undef SPJ_KNN_SPLIT
    } else {
#define SPJ_KNN_LAUNCH(KK)                                                                       \
  if (form_ == 1)                                                                                \
    k_knn<KK, true><<<g, kKnnThreads, 0, s>>>(t, xy_sorted_.as<double2>(), dp, n, order, nullptr, \
                                              k, slack_, di, dd, ev);                            \
  else                                                                                           \
    k_knn<KK, false><<<g, kKnnThreads, 0, s>>>(t, xy_sorted_.as<double2>(), dp, n, order,        \
                                               nullptr, k, slack_, di, dd, ev);
      if (k <= 8) {
        SPJ_KNN_LAUNCH(8)
      } else if (k <= 16) {
        SPJ_KNN_LAUNCH(16)
      } else {
        SPJ_KNN_LAUNCH(32)
      }
#undef SPJ_KNN_LAUNCH
    }
    SPJ_CUDA(cudaGetLastError());
  }
  if (!device_ptrs && n) {
    SPJ_CUDA(cudaMemcpyAsync(out_idx, di, n * k * 4, cudaMemcpyDeviceToHost, s));
    SPJ_CUDA(cudaMemcpyAsync(out_dist, dd, n * k * 8, cudaMemcpyDeviceToHost, s));
  }
  unsigned long long cnt[2] = {0, 0};
  SPJ_CUDA(cudaMemcpyAsync(cnt, counters_.get(), 16, cudaMemcpyDeviceToHost, s));
  SPJ_CUDA(cudaStreamSynchronize(s));
  check_traversal(bvh_.view(), s);
  exact_evals_ += cnt[0];
  redone_ += (cnt[1] & 0xFFFFFFFFull) + (cnt[1] >> 32);
  queries_ += n;
}

}  // namespace spj
