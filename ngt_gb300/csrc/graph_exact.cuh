// Exact-order graph search: one query per CTA, FP32 (or the object's native
// type), reproducing NGT's sequential best-first search step for step.
//
// Reference: NeighborhoodGraph::searchReadOnlyGraph (lib/NGT/Graph.cpp:716-835)
// and NeighborhoodGraph::search (lib/NGT/Graph.cpp:840-1024), seeded by
// GraphAndTreeIndex::getSeedsFromTree (lib/NGT/Index.h:2173-2220) through
// DVPTree::search in SearchLeaf mode (lib/NGT/Tree.cpp:403-559), with
// setupDistances/setupSeeds (lib/NGT/Graph.cpp:420-586).
//
// Why the results are the reference's, not just close to them:
//   * The neighbours of the expanded node are filtered against the visited set
//     in edge order and their distances computed in parallel.  The result-set
//     updates are the only order-dependent step: what the reference's sequence of
//     push / push_pop leaves is merged at once (merge_results); where the order
//     decides (epsilon < 0, negative distances, a tie at the last result) one warp
//     replays them one by one in edge order.
//   * The candidate queue only needs the set of entries <= explorationRadius:
//     the radius never grows, the loop stops at the first popped entry above it,
//     so pushing a chunk's survivors after the chunk (against the radius reached
//     at its end) leaves the pop sequence unchanged.
//   * The queue is a sorted array in shared memory, merged with each chunk's
//     sorted survivors; (distance, id) keys make the order total, like
//     ObjectDistance::operator< (lib/NGT/Common.h:2347-2360).
//   * The queue has two tiers: the best `ccap` entries sorted in shared memory
//     and an unsorted overflow tier in global memory whose entries are all
//     larger than every shared-memory entry.  When the shared list drains, the
//     overflow's live entries (<= explorationRadius) are filtered and the smallest
//     of them, up to the edge of a radix bin that fills at least half the list,
//     sorted and moved back (exact_refill).  Pops therefore follow the reference's
//     order exactly.
// The only limit that can make a query inexact is the overflow tier's capacity
// (reported in QueryStats::status).  The visited set never loses entries: it
// is a bitmap in shared memory where that fits, else a hash table there that moves
// to a per-CTA bitmap in global memory when it is half full.
#pragma once
#include <cfloat>
#include <type_traits>
#include "distance.cuh"
#include "device_index.h"

namespace ngtg {

constexpr int kExactThreads = 128;
constexpr int kExactWarps = kExactThreads / 32;
constexpr int kExactChunk = kExactThreads;   // neighbours processed per round

// Neighbours processed per round by a CTA of T threads, at most one per thread.
template <int T> constexpr int exact_chunk() { return T < 256 ? T : 256; }
// Rows each group of threads keeps in flight while computing distances.
// (One where a row has three sums: two rows' twenty-four would spill.)
template <class A, int T> constexpr int exact_rows() { return T == 128 && A::kUseF12 ? 1 : 2; }

struct ExactShared {
  float radius;
  uint32_t nres;
  uint32_t keep[3];               // neighbours of the round within the exploration radius (rounds in turn)
  uint32_t live_old;
  uint32_t seed_leaf;
  uint32_t seed_status;
  uint32_t nmoved;                // refill: keys moved to shared memory
  uint32_t ovf_n;                 // refill: keys left in the overflow tier
  uint32_t sel_bin, sel_acc;
  uint32_t query;
  unsigned long long key_min, key_max;
  unsigned long long evict_min;
  unsigned long long edge[2];     // merge_results: the keys at places size - 1 and size
  __align__(16) uint32_t warp_cnt[8];
  uint32_t hist[256];
};

struct ExactConfig {
  uint32_t kcap;     // result capacity (>= max size in the batch)
  uint32_t ccap;     // candidate-list capacity
  uint32_t hcap;     // visited hash capacity (power of two), or words of the shared-memory bitmap
  uint32_t mode;     // GraphMode
  uint32_t group;    // lanes per distance (power of two <= 32)
  uint32_t bitmap_words;  // words per CTA in the spill bitmap
  uint32_t ocap;          // overflow-tier capacity per CTA (keys)
  uint32_t table_bytes;   // quantized graph: qg_table_bytes
  uint32_t smem_bitmap;   // 1: the visited set is a bitmap of every id in shared memory (hcap words)
  uint32_t* work;         // zeroed counter from which the CTAs take the queries; null: CTA i
                          // takes queries i, i + grid, ...
};

// The next query of this CTA (nq or more: none); `at` is the query just searched (or
// UINT32_MAX).  Executed by the whole CTA; sh: a shared word.
__device__ __forceinline__ uint32_t exact_next_query(uint32_t at, uint32_t* work, uint32_t* sh) {
  if (!work) return at == 0xffffffffu ? blockIdx.x : at + gridDim.x;
  if (threadIdx.x == 0) *sh = atomicAdd(work, 1u);
  __syncthreads();
  return *sh;
}

__device__ __forceinline__ uint32_t hash_slot(uint32_t id, uint32_t mask) {
  return (id * 0x9E3779B1u) & mask;
}

// Returns true when `id` was not in the visited set (and inserts it).
__device__ __forceinline__ bool visit_insert(uint32_t* table, uint32_t mask, uint32_t* bitmap, bool spilled,
                                             uint32_t id) {
  if (spilled) {
    uint32_t bit = 1u << (id & 31u);
    uint32_t old = atomicOr(&bitmap[id >> 5], bit);
    return (old & bit) == 0u;
  }
  uint32_t h = hash_slot(id, mask);
  // The table is kept at most half full (plus one chunk), so probing ends.
  for (uint32_t probe = 0; probe <= mask; probe++) {
    uint32_t old = atomicCAS(&table[h], 0u, id);
    if (old == 0u) return true;
    if (old == id) return false;
    h = (h + 1u) & mask;
  }
  return false;
}

// Insert key x into the sorted array res[0..n) with the reference's semantics.
// Returns the new count; updates radius when the reference would.
// Executed by one full warp.
__device__ __forceinline__ void result_insert(unsigned long long* res, uint32_t& n, float& radius,
                                              uint32_t size, uint32_t mode, unsigned long long x, int lane) {
  // Read-only search: push_pop replaces the current maximum when full
  // (ResultSet::push_pop, lib/NGT/Common.h:2421-2428).  Updatable search:
  // push, then pop the maximum if the set grew beyond `size`
  // (lib/NGT/Graph.cpp:990-1004).
  uint32_t live = n;
  bool full = n >= size;
  if (mode == (uint32_t)GraphMode::ReadOnly && full) live = n - 1;   // drop the max first
  uint32_t cnt = 0;
  for (uint32_t i = lane; i < live; i += 32) cnt += res[i] < x ? 1u : 0u;
  uint32_t p = __reduce_add_sync(0xffffffffu, cnt);
  // shift res[p..live) right by one, from the top down
  for (int hi = (int)live; hi > (int)p; hi -= 32) {
    int lo = max((int)p, hi - 32);
    int idx = lo + lane;
    unsigned long long v = 0;
    bool act = idx < hi;
    if (act) v = res[idx];
    __syncwarp();
    if (act) res[idx + 1] = v;
    __syncwarp();
  }
  if (lane == 0) res[p] = x;
  __syncwarp();
  if (mode == (uint32_t)GraphMode::ReadOnly) {
    if (full) {
      radius = key_dist(res[n - 1]);
    } else {
      n = n + 1;
    }
  } else {
    n = n + 1;
    if (n > size) n = size;          // pop the maximum (it sits at index size)
    if (n >= size) radius = key_dist(res[n - 1]);
  }
}

// Rank sort of up to kExactChunk keys (unique) by the whole CTA.
__device__ __forceinline__ void rank_sort(const unsigned long long* in, unsigned long long* out, uint32_t m) {
  for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) {
    unsigned long long k = in[i];
    uint32_t r = 0;
    for (uint32_t j = 0; j < m; j++) r += in[j] < k ? 1u : 0u;
    out[r] = k;
  }
}

// In-place ascending bitonic sort of a[0..n) in shared memory by the whole CTA;
// entries [n, p) are padded with ~0 where p is the next power of two (<= cap).
__device__ __forceinline__ void bitonic_sort(unsigned long long* a, uint32_t n, uint32_t cap) {
  uint32_t p = 1;
  while (p < n) p <<= 1;
  for (uint32_t i = n + threadIdx.x; i < p && i < cap; i += blockDim.x) a[i] = ~0ull;
  __syncthreads();
  for (uint32_t k = 2; k <= p; k <<= 1) {
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      for (uint32_t i = threadIdx.x; i < p; i += blockDim.x) {
        uint32_t l = i ^ j;
        if (l > i) {
          unsigned long long x = a[i], y = a[l];
          bool up = (i & k) == 0;
          if ((x > y) == up) { a[i] = y; a[l] = x; }
        }
      }
      __syncthreads();
    }
  }
}

__device__ __forceinline__ uint32_t lower_bound_keys(const unsigned long long* a, uint32_t n, unsigned long long x) {
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    uint32_t mid = (lo + hi) >> 1;
    if (a[mid] < x) lo = mid + 1; else hi = mid;
  }
  return lo;
}

__device__ __forceinline__ uint32_t upper_bound_dist(const unsigned long long* a, uint32_t n, float r) {
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    uint32_t mid = (lo + hi) >> 1;
    if (key_dist(a[mid]) <= r) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// Asks for the first KB of a row (rc 16-byte chunks) to be brought into L2.
__device__ __forceinline__ void prefetch_row(const uint4* row, uint32_t rc) {
#pragma unroll
  for (uint32_t c = 0; c < 64; c += 8)
    if (c < rc) asm volatile("prefetch.global.L2 [%0];" ::"l"(row + c));
}

// A round's updates of the result set res (n = s.nres keys, ascending) as one merge: the
// neighbours within `radius` (a prefix of the sorted survivors sv[0..m)) join in edge
// order nd / nid, exploration coefficient >= 1.  Executed by the whole CTA; false (nothing
// changed) when the order of the updates could matter: the replay decides.
//
// What the sequence of updates leaves, without going through it: once the set is full and
// `radius` is its largest distance, every update drops the maximum and takes a neighbour
// no farther, so the distances kept are always the `size` smallest seen, and so are the
// keys unless the distances at places size - 1 and size of the union are equal (then it
// is the order that decides, read-only search; the updatable one keeps the smaller key).
// The read-only search fills the set first, with the first size - n neighbours, and the
// next one then replaces the maximum of that moment whatever it is, because the radius
// still is the initial one: that maximum alone is missing from the union.
// One by one, an update costs warp 0 about 400 cycles, and a search that approaches its
// query takes most neighbours of its first expansions: half the time of short searches.
template <int T>
__device__ __noinline__ bool merge_results(unsigned long long* res, uint32_t size, uint32_t mode, float radius,
                                           const unsigned long long* sv, uint32_t m, const float* nd,
                                           const uint32_t* nid, uint32_t nnew, ExactShared& s) {
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t n = s.nres;
  // below zero (the scalar-quantized inner product) the exploration radius is the tighter one
  if (key_dist(sv[0]) < 0.f || (n && key_dist(res[0]) < 0.f)) {
    __syncthreads();                         // every warp has decided before the replay rewrites res and s.nres
    return false;
  }
  const uint32_t p = upper_bound_dist(sv, m, radius);
  const bool ro = mode == (uint32_t)GraphMode::ReadOnly;
  const uint32_t fill = n < size ? size - n : 0u;
  const bool stale = ro && n >= size && key_dist(res[n - 1]) != radius;
  const bool removal = ro && ((fill && p > fill) || stale);
  unsigned long long rem = ~0ull;
  if (tid == 0) {
    s.edge[0] = s.edge[1] = ~0ull;
    s.key_max = n ? res[n - 1] : 0ull;
  }
  if (removal) {
    const bool in = tid < nnew && nd[tid] <= radius;
    const uint32_t mask = __ballot_sync(0xffffffffu, in);
    if (lane == 0 && warp < 8) s.warp_cnt[warp] = __popc(mask);     // nnew <= 256: eight warps at most
    __syncthreads();
    if (in && fill) {
      uint32_t o = __popc(mask & ((1u << lane) - 1u));
      for (uint32_t w = 0; w < warp; w++) o += s.warp_cnt[w];
      if (o < fill) atomicMax(&s.key_max, pack_key(nd[tid], nid[tid]));
    }
    __syncthreads();
    rem = s.key_max;
  } else {
    __syncthreads();
  }
  const uint32_t total = n + p - (removal ? 1u : 0u);
  // places of this thread's survivor, and the keys at the cut
  unsigned long long mine = ~0ull;
  uint32_t at = 0xffffffffu;
  if (tid < p) {
    mine = sv[tid];
    if (!(removal && mine == rem)) {
      at = tid + lower_bound_keys(res, n, mine) - (removal && mine > rem ? 1u : 0u);
      if (at == size - 1) s.edge[0] = mine;
      if (at == size) s.edge[1] = mine;
    }
  }
  for (uint32_t i = tid; i < n; i += T) {
    const unsigned long long r = res[i];
    if (removal && r == rem) continue;
    const uint32_t to = i + lower_bound_keys(sv, p, r) - (removal && r > rem ? 1u : 0u);
    if (to == size - 1) s.edge[0] = r;
    if (to == size) s.edge[1] = r;
  }
  __syncthreads();
  if (ro && total > size && key_dist(s.edge[0]) == key_dist(s.edge[1])) {
    __syncthreads();                         // s.edge is read before a later call resets it
    return false;
  }
  // the old keys move up, from the top; then the survivors take their places
  for (uint32_t top = n; top > 0;) {
    const uint32_t b = top > (uint32_t)T ? top - T : 0u, i = b + tid;
    unsigned long long r = ~0ull;
    uint32_t to = 0xffffffffu;
    if (i < top) {
      r = res[i];
      if (!(removal && r == rem)) to = i + lower_bound_keys(sv, p, r) - (removal && r > rem ? 1u : 0u);
    }
    __syncthreads();
    if (to < size) res[to] = r;
    __syncthreads();
    top = b;
  }
  if (at < size) res[at] = mine;
  if (tid == 0) {
    s.nres = min(total, size);
    const bool moved = ro ? n >= size || p > fill : total >= size;
    s.radius = moved ? key_dist(s.edge[0]) : radius;
  }
  __syncthreads();
  return true;
}

// Moves the smallest live keys of the overflow tier (ovf[0..n), scratch tmp) into the
// empty shared list cl, sorted: entries above the exploration radius are dropped, and
// when more than ccap live, a threshold is taken at the edge of a radix bin, so that at
// least half of the list is filled and every key left behind is larger.  (Which keys
// wait in which tier does not change the order of the pops.)  Returns the keys moved;
// n and ovf_min are updated.  Executed by the whole CTA of T threads.
template <int T>
__device__ __noinline__ uint32_t exact_refill(unsigned long long* cl, uint32_t ccap, unsigned long long* ovf,
                                              unsigned long long* tmp, uint32_t& n, unsigned long long& ovf_min,
                                              float expR, ExactShared& s) {
  const uint32_t tid = threadIdx.x, lane = tid & 31;
  const uint32_t below = (1u << lane) - 1u;
  if (tid == 0) {
    s.nmoved = 0;
    s.key_min = ~0ull;
    s.key_max = 0ull;
  }
  __syncthreads();
  unsigned long long mn = ~0ull, mx = 0ull;
  for (uint32_t b = 0; b < n; b += T) {
    const uint32_t i = b + tid;
    const unsigned long long k = i < n ? ovf[i] : ~0ull;
    const bool live = i < n && key_dist(k) <= expR;
    const uint32_t mask = __ballot_sync(0xffffffffu, live);
    uint32_t at = 0;
    if (lane == 0 && mask) at = atomicAdd(&s.nmoved, (uint32_t)__popc(mask));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (live) {
      tmp[at + __popc(mask & below)] = k;
      mn = k < mn ? k : mn;
      mx = k > mx ? k : mx;
    }
  }
  for (int off = 16; off > 0; off >>= 1) {
    const unsigned long long a = __shfl_xor_sync(0xffffffffu, mn, off), c = __shfl_xor_sync(0xffffffffu, mx, off);
    mn = a < mn ? a : mn;
    mx = c > mx ? c : mx;
  }
  if (lane == 0 && mn != ~0ull) {
    atomicMin(&s.key_min, mn);
    atomicMax(&s.key_max, mx);
  }
  __syncthreads();
  const uint32_t r = s.nmoved;
  if (r <= ccap) {
    for (uint32_t i = tid; i < r; i += T) cl[i] = tmp[i];
    __syncthreads();
    bitonic_sort(cl, r, ccap);
    n = 0;
    ovf_min = ~0ull;
    return r;
  }
  // radix bins of 8 bits from the highest byte in which the keys differ
  const unsigned long long diff = s.key_min ^ s.key_max;
  int shift = (63 - __clzll((long long)diff)) / 8 * 8;
  unsigned long long prefix = s.key_min >> shift >> 8 << 8 << shift;      // the common bits above the digit
  uint32_t acc = 0;                    // keys below the prefix
  unsigned long long thr;
  while (true) {
    for (uint32_t i = tid; i < 256; i += T) s.hist[i] = 0;
    __syncthreads();
    for (uint32_t i = tid; i < r; i += T) {
      const unsigned long long x = tmp[i];
      if ((x >> shift >> 8) == (prefix >> shift >> 8)) atomicAdd(&s.hist[(uint32_t)(x >> shift) & 255u], 1u);
    }
    __syncthreads();
    if (tid < 32) {
      // the bins that fit: the largest b with acc + (keys in bins below b) <= ccap
      uint32_t c[8], sum = 0;
#pragma unroll
      for (int j = 0; j < 8; j++) {
        c[j] = s.hist[lane * 8 + j];
        sum += c[j];
      }
      uint32_t incl = sum;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= (uint32_t)off) incl += y;
      }
      uint32_t run = acc + incl - sum, fit = 0, got = run;
      if (run <= ccap)
#pragma unroll
        for (int j = 0; j < 8; j++) {
          run += c[j];
          if (run <= ccap) {
            fit = j + 1;
            got = run;
          }
        }
      // bins fit in order: the last lane whose first bin starts within the capacity
      const uint32_t okm = __ballot_sync(0xffffffffu, acc + incl - sum <= ccap);
      if ((int)lane == 31 - __clz((int)okm)) {
        s.sel_bin = lane * 8 + fit;
        s.sel_acc = got;
      }
    }
    __syncthreads();
    const uint32_t bin = s.sel_bin;
    acc = s.sel_acc;
    __syncthreads();
    thr = prefix + ((unsigned long long)bin << shift) - 1ull;
    if (acc >= ccap / 2 || shift == 0 || bin > 255) break;
    prefix += (unsigned long long)bin << shift;          // the bin that does not fit, split further
    shift -= 8;
  }
  if (tid == 0) {
    s.nmoved = 0;
    s.ovf_n = 0;
    s.key_min = ~0ull;
  }
  __syncthreads();
  mn = ~0ull;
  for (uint32_t b = 0; b < r; b += T) {
    const uint32_t i = b + tid;
    const unsigned long long k = i < r ? tmp[i] : ~0ull;
    const bool take = i < r && k <= thr, leave = i < r && k > thr;
    const uint32_t tm = __ballot_sync(0xffffffffu, take), lm = __ballot_sync(0xffffffffu, leave);
    uint32_t at = 0, al = 0;
    if (lane == 0) {
      if (tm) at = atomicAdd(&s.nmoved, (uint32_t)__popc(tm));
      if (lm) al = atomicAdd(&s.ovf_n, (uint32_t)__popc(lm));
    }
    at = __shfl_sync(0xffffffffu, at, 0);
    al = __shfl_sync(0xffffffffu, al, 0);
    if (take) cl[at + __popc(tm & below)] = k;
    if (leave) {
      ovf[al + __popc(lm & below)] = k;
      mn = k < mn ? k : mn;
    }
  }
  for (int off = 16; off > 0; off >>= 1) {
    const unsigned long long a = __shfl_xor_sync(0xffffffffu, mn, off);
    mn = a < mn ? a : mn;
  }
  if (lane == 0 && mn != ~0ull) atomicMin(&s.key_min, mn);
  __syncthreads();
  n = s.ovf_n;
  ovf_min = s.key_min;
  const uint32_t moved = s.nmoved;
  bitonic_sort(cl, moved, ccap);
  __syncthreads();
  return moved;
}

// Bound by latency and instruction issue: each expansion is a chain of dependent accesses
// (the node's offsets, its edges, their visited bits, the new rows) and the chunk's
// bookkeeping between CTA barriers.  What keeps the chain short:
//   * the list's head, which is the next node unless a survivor is nearer (four times in
//     five), has its offsets and edges loaded beside the current node's rows; another next
//     node's offsets load while the list is merged;
//   * a chunk without survivors (two in three: nearly all neighbours are past the
//     exploration radius) leaves the list as it is and takes two barriers; with survivors
//     four (twelve before);
//   * distances by packed groups of threads (packed_sums), two rows each in flight, and no
//     square root for rows past the exploration radius;
//   * result updates merged at once (merge_results);
//   * T: launches that leave SMs idle give each query 512 threads (128 float rows in
//     flight instead of 32) and, where it fits, a visited bitmap in shared memory.
// Measured on 1M x 128 float objects (fixed seeds, L2): single queries, k = 20, epsilon 0.1
// (about 2,000 expansions): 25.1 ms before, 6.4 ms with 512 threads; 2,000 queries, k = 10,
// epsilon 0.08: 17.3 -> 10.7 ms; 100 of them: 2.8 ms with 512 threads, 5.0 ms with 128;
// 300 of them: 6.1 and 5.2 ms, so 512 threads serve launches of at most one CTA per SM.
// Six 128-thread CTAs per SM (80 registers): seven (72, spills) are as fast for L2 and
// 5-8 % slower for cosine and short searches; four 56.5 ms, nine 46.7 ms for 10,000
// queries against 44.1 ms; then the work counter and the shorter shared list, 33.9 ms.
// Not kept: fetching a survivor's neighbours' rows into L2 when it joins the list (512
// threads; 10 % slower), the result set in a warp's registers (slower than shared memory).
template <ObjType OT, Metric M, int T>
__global__ void __launch_bounds__(T, T == 128 ? 6 : 1)
graph_search_exact_kernel(DevGraph g, const uint4* __restrict__ queries, uint32_t nq,
                          const QueryParams* __restrict__ params, const uint32_t* __restrict__ seed_list,
                          ObjDist* __restrict__ out, uint32_t* __restrict__ out_count,
                          QueryStats* __restrict__ stats, uint32_t* __restrict__ bitmaps,
                          unsigned long long* __restrict__ overflow, ExactConfig cfg) {
  constexpr uint32_t CH = (uint32_t)exact_chunk<T>();
  constexpr uint32_t CW = CH / 32;                        // warps that hold a chunk's neighbours
  constexpr int U = exact_rows<Acc<OT, M>, T>();
  extern __shared__ __align__(16) unsigned char smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t rc = g.row_chunks;
  // ---- shared-memory carve-up -------------------------------------------
  uint4* qv = reinterpret_cast<uint4*>(smem);
  unsigned long long* res = reinterpret_cast<unsigned long long*>(qv + rc);
  unsigned long long* cand0 = res + (cfg.kcap + 1) / 2 * 2;
  unsigned long long* cand1 = cand0 + cfg.ccap;
  unsigned long long* bkeys = cand1 + cfg.ccap;          // chunk survivors (unsorted)
  unsigned long long* bsorted = bkeys + CH;              // chunk survivors (sorted)
  uint32_t* table = reinterpret_cast<uint32_t*>(bsorted + CH);
  uint32_t* seg = table + (cfg.hcap + 3) / 4 * 4;        // new ids, 32 slots per warp of the chunk
  uint32_t* nid = seg + CH;                              // new ids in edge order
  float* nd = reinterpret_cast<float*>(nid + CH);
  ExactShared& s = *reinterpret_cast<ExactShared*>(nd + CH);
  uint32_t* bitmap = bitmaps + (size_t)blockIdx.x * cfg.bitmap_words;
  unsigned long long* ovf = overflow + (size_t)blockIdx.x * 2 * cfg.ocap;     // overflow tier
  unsigned long long* ovf_tmp = ovf + cfg.ocap;                                 // refill scratch
  const uint32_t hmask = cfg.hcap - 1;
  const int G = (int)cfg.group;
  const int gl = lane & (G - 1);                   // lane inside the distance group
  const uint32_t ngroups = T / G;
  const int pw = packed_width(G);                  // threads per row in the loop
  const uint32_t npacked = T / pw;

  for (uint32_t q = exact_next_query(0xffffffffu, cfg.work, &s.query); q < nq;
       q = exact_next_query(q, cfg.work, &s.query)) {
    const QueryParams P = params[q];
    // ---- per-query initialisation ----------------------------------------
    for (uint32_t i = tid; i < rc; i += T) qv[i] = queries[(size_t)q * rc + i];
    for (uint32_t i = tid; i < (cfg.hcap + 3) / 4; i += T)
      reinterpret_cast<uint4*>(table)[i] = make_uint4(0u, 0u, 0u, 0u);
    if (tid == 0) {
      s.seed_status = 0;
      s.keep[0] = s.keep[1] = 0;
    }
    __syncthreads();
    if (P.size == 0) {          // GraphIndex::search returns nothing for size 0
      if (tid == 0) { out_count[q] = 0; stats[q] = QueryStats{0, 0, 0, 0, 0}; }
      __syncthreads();
      continue;
    }
    // ---- seeds --------------------------------------------------------------
    const uint32_t* seeds = nullptr;
    uint32_t nseeds = 0;
    if (P.seed_cnt == 0xffffffffu) {
      // DVP-tree descent with radius 0 (one region per level) -- warp 0.
      if (warp == 0) {
        uint32_t node = g.root;
        int depth = 0;
        while (!(node & 0x80000000u) && depth < 64) {
          const DevInternal& in = g.internals[node];
          float d = group_distance<TreeSpace<OT, M>::ot, TreeSpace<OT, M>::m>(qv, g.pivots + (size_t)in.pivot * rc, (int)rc, lane, 32);
          uint32_t bsize = in.nchildren - 1, mid;
          for (mid = 0; mid < bsize; mid++)
            if (d < in.borders[mid]) break;
          node = in.children[mid];
          depth++;
        }
        if (lane == 0) {
          if (node & 0x80000000u) s.seed_leaf = node & 0x7fffffffu;
          else { s.seed_leaf = 0xffffffffu; s.seed_status = kStatusTreeError; }
        }
      }
      __syncthreads();
      if (s.seed_leaf != 0xffffffffu && s.seed_leaf < g.nleaves) {
        const uint32_t* off = g.leaf_seed_off + P.seed_off;    // this query's seed-size table
        uint32_t a = off[s.seed_leaf], b = off[s.seed_leaf + 1];
        seeds = g.leaf_seed_ids + a;
        nseeds = b - a;
      }
    } else {
      seeds = seed_list + P.seed_off;
      nseeds = P.seed_cnt;
    }
    nseeds = min(nseeds, (uint32_t)kExactChunk);
    uint32_t status = s.seed_status;
    if (nseeds == 0) {
      if (tid == 0) {
        out_count[q] = 0;
        stats[q] = QueryStats{0, 0, 0, 0, status | kStatusEmptySeeds};
      }
      __syncthreads();
      continue;
    }
    // setupDistances: exact distances of the seeds
    // (warp-uniform trip counts: every lane of a warp reaches the shuffles)
    for (uint32_t b = (uint32_t)(warp * (32 / G)); b < nseeds; b += ngroups) {
      uint32_t i = b + (uint32_t)(lane / G);
      bool valid = i < nseeds;
      uint32_t id = valid ? seeds[i] : 0u;
      bool inrange = id < g.nrows;
      float d = group_distance<OT, M>(qv, g.objects + (size_t)(inrange ? id : 0u) * rc, (int)rc, gl, G);
      if (valid && gl == 0) bkeys[i] = pack_key(inrange ? d : FLT_MAX, id);
    }
    __syncthreads();
    rank_sort(bkeys, bsorted, nseeds);
    __syncthreads();
    // setupSeeds: results take the leading seeds within the radius; all seeds are
    // marked visited and become candidates.
    if (tid == 0) {
      uint32_t n = 0;
      float radius = P.radius;
      for (uint32_t i = 0; i < nseeds; i++) {
        float d = key_dist(bsorted[i]);
        if (n < P.size && d <= radius) res[n++] = bsorted[i];
        else break;
      }
      if (n >= P.size) radius = key_dist(res[n - 1]);
      s.nres = n;
      s.radius = radius;
    }
    for (uint32_t i = tid; i < nseeds; i += T) {
      cand0[i] = bsorted[i];
      const uint32_t id = key_id(bsorted[i]);
      if (cfg.smem_bitmap) {
        if (id < g.nrows) atomicOr(&table[id >> 5], 1u << (id & 31u));
      } else {
        visit_insert(table, hmask, bitmap, false, id);
      }
    }
    __syncthreads();

    // ---- best-first loop -----------------------------------------------------
    // Alike in every thread: the shared list is cl[head..tail) (cl: cand1 when cur), the
    // overflow tier holds ovf_n keys, the smallest ovf_min.
    uint32_t head = 0, tail = nseeds, cur = 0, ovf_n = 0;
    unsigned long long ovf_min = ~0ull;
    uint32_t nvisited = nseeds, dc = nseeds, expansions = 0, edges = 0;
    bool spilled = false, have = false;
    float radius = s.radius;
    uint32_t e0 = 0, nsz = 0, eid = 0;            // the node to expand: edges, this thread's neighbour
    uint32_t guard = 0, turn = 0;
    while (true) {
      if (!have) {
        if (head >= tail && ovf_n > 0) {
          head = 0;
          tail = exact_refill<T>(cur ? cand1 : cand0, cfg.ccap, ovf, ovf_tmp, ovf_n, ovf_min, P.coef * radius, s);
        }
        if (head >= tail) break;
        const unsigned long long t = (cur ? cand1 : cand0)[head];
        if (key_dist(t) > P.coef * radius) break;
        head++;
        e0 = g.offsets[key_id(t)];
        nsz = min(g.offsets[key_id(t) + 1] - e0, P.edge_size);
        if ((uint32_t)tid < min(nsz, CH)) eid = g.edges[e0 + tid];
      }
      have = false;
      // the list's head is the next node unless this one has a nearer survivor: its edges
      // load beside this node's rows
      const unsigned long long guess = head < tail ? (cur ? cand1 : cand0)[head] : ~0ull;
      uint32_t g0 = 0, g1 = 0, gid = 0;
      if (head < tail) {
        g0 = __ldg(g.offsets + key_id(guess));
        g1 = __ldg(g.offsets + key_id(guess) + 1);
      }
      if (guard++ > g.nrows + 8) {     // cannot happen: each id is expanded at most once
        status |= kStatusIterationLimit;
        break;
      }
      expansions++;
      edges += nsz;
      bool finished = false;
      const uint32_t n_edges = nsz;                // nsz and e0 move on to the next node in the last chunk
      for (uint32_t c0 = 0; c0 < n_edges; c0 += CH) {
        const uint32_t clen = min(CH, n_edges - c0);
        // spill the visited set to the bitmap before it gets more than half full
        if (!cfg.smem_bitmap && !spilled && nvisited + clen > (cfg.hcap >> 1)) {
          for (uint32_t i = tid; i < cfg.hcap; i += T) {
            uint32_t id = table[i];
            if (id) atomicOr(&bitmap[id >> 5], 1u << (id & 31u));
          }
          __threadfence_block();
          __syncthreads();
          spilled = true;
          status |= kStatusVisitedSpill;
        }
        // visited filter in edge order; each warp packs its new ids
        if ((uint32_t)warp < CW) {
          bool isnew = false;
          if ((uint32_t)tid < clen) {
            if (cfg.smem_bitmap) {
              const uint32_t bit = 1u << (eid & 31u);
              isnew = (atomicOr(&table[eid >> 5], bit) & bit) == 0u;
            } else {
              isnew = visit_insert(table, hmask, bitmap, spilled, eid);
            }
          }
          const unsigned ballot = __ballot_sync(0xffffffffu, isnew);
          if (isnew) seg[warp * 32 + __popc(ballot & ((1u << lane) - 1u))] = eid;
          // the rows of later rounds are under way to L2 beside the first round's (10,000
          // queries: 35.9 -> 33.5 ms; no gain with 512 threads, whose rounds take them all)
          if (T == 128 && isnew) prefetch_row(g.objects + (size_t)eid * rc, rc);
          if (lane == 0) s.warp_cnt[warp] = __popc(ballot);
        }
        __syncthreads();
        uint32_t pre[CW + 1];                     // new ids before each warp's
        pre[0] = 0;
#pragma unroll
        for (uint32_t w = 0; w < CW; w++) pre[w + 1] = pre[w] + s.warp_cnt[w];
        const uint32_t nnew = pre[CW];
        const bool last = c0 + CH >= n_edges;
        if (last) {
          if (head < tail && (uint32_t)tid < min(min(g1 - g0, P.edge_size), CH)) gid = __ldg(g.edges + g0 + tid);
        } else if (tid < (int)CH && c0 + CH + tid < n_edges) {
          eid = __ldg(g.edges + e0 + c0 + CH + tid);
        }
        const float expR0 = P.coef * radius;
        // distances, U rows per group of threads in flight while that many are left
        bool pass = false;
        const float far = Acc<OT, M>::far_limit(expR0);
        auto rows = [&](auto rows_at_once, uint32_t b) {
          constexpr int R = decltype(rows_at_once)::value;
          uint32_t id[R];
          Acc<OT, M> sum[R];
#pragma unroll
          for (int u = 0; u < R; u++) {
            const uint32_t i = b + u * npacked + (uint32_t)(lane / pw);
            uint32_t at = i;
#pragma unroll
            for (uint32_t w = 1; w < CW; w++) at = i >= pre[w] ? w * 32 + i - pre[w] : at;
            id[u] = i < nnew ? seg[at] : 0u;
          }
          packed_sums<OT, M, R>(qv, g.objects, id, (int)rc, lane & (pw - 1), G, sum);
#pragma unroll
          for (int u = 0; u < R; u++) {
            const uint32_t i = b + u * npacked + (uint32_t)(lane / pw);
            if (i < nnew && (lane & (pw - 1)) == 0) {
              float d = FLT_MAX;                   // past the exploration radius: no more is asked of it
              if (!sum[u].is_far(far)) {
                d = sum[u].finish();
                pass = pass || (d <= radius && d <= expR0);
                if (d <= expR0) bkeys[atomicAdd(&s.keep[turn], 1u)] = pack_key(d, id[u]);
              }
              nd[i] = d;
              nid[i] = id[u];
            }
          }
        };
        for (uint32_t b = (uint32_t)(warp * (32 / pw)); b < nnew;) {
          if (U > 1 && b + npacked < nnew) {
            rows(std::integral_constant<int, U>(), b);
            b += U * npacked;
          } else {
            rows(std::integral_constant<int, 1>(), b);
            b += npacked;
          }
        }
        // the result-set updates, when there are some: merged at once, or (with epsilon < 0, or
        // a tie at the last result) replayed one by one by warp 0
        const bool replay = __syncthreads_or(pass ? 1 : 0) != 0;
        uint32_t m = s.keep[turn];                // survivors: within the exploration radius
        turn ^= 1u;
        if (tid == 0) s.keep[turn] = 0;           // the next round's (last read two rounds ago)
        if (replay) {
          rank_sort_split<T>(bkeys, bsorted, m);
          __syncthreads();
          if (!(P.coef >= 1.0f) || !merge_results<T>(res, P.size, cfg.mode, radius, bsorted, m, nd, nid, nnew, s)) {
            if (warp == 0) {
              uint32_t n = s.nres;
              float rad = radius;
              for (uint32_t b = 0; b < nnew; b += 32) {
                uint32_t i = b + lane;
                // a neighbour joins when within the exploration radius and the radius
                // of that moment (both only shrink; with epsilon < 0 the first is
                // the tighter one)
                float d = i < nnew ? nd[i] : FLT_MAX;
                float lim = fminf(rad, P.coef * rad);
                unsigned m = __ballot_sync(0xffffffffu, i < nnew && d <= lim);
                while (m) {
                  int src = __ffs(m) - 1;
                  float dj = __shfl_sync(0xffffffffu, d, src);
                  uint32_t idj = nid[b + src];
                  if (dj <= rad && dj <= P.coef * rad)
                    result_insert(res, n, rad, P.size, cfg.mode, pack_key(dj, idj), lane);
                  m &= (src == 31) ? 0u : ~((2u << src) - 1u);
                  lim = fminf(rad, P.coef * rad);
                  m &= __ballot_sync(0xffffffffu, i < nnew && d <= lim);
                }
              }
              if (lane == 0) {
                s.radius = rad;
                s.nres = n;
              }
            }
            __syncthreads();
          }
          radius = s.radius;
        }
        dc += nnew;
        nvisited += nnew;
        const float expR = P.coef * radius;
        unsigned long long* cl = cur ? cand1 : cand0;
        if (m == 0) {
          // no candidate came: the list stays, and its head is the guess unless an earlier
          // round of this node brought a nearer one (which is popped at the top then)
          if (last && head < tail && cl[head] == guess) {
            have = !(key_dist(guess) > expR);
            finished = !have;
            if (have) {
              head++;
              e0 = g0;
              nsz = min(g1 - g0, P.edge_size);
              eid = gid;
            }
          }
          continue;
        }
        // chunk survivors become candidates
        if (tid == 0) s.evict_min = ~0ull;
        unsigned long long* cn = cur ? cand0 : cand1;
        const unsigned long long* old = cl + head;
        if (!replay) rank_sort_split<T>(bkeys, bsorted, m);
        // entries above a smaller exploration radius can never be expanded again
        if (replay && tid == T - 1) s.live_old = upper_bound_dist(old, tail - head, expR);
        __syncthreads();
        uint32_t nold = tail - head;
        if (replay) {
          nold = s.live_old;
          m = upper_bound_dist(bsorted, m, expR);
        }
        // survivors not below the overflow tier's minimum join the tier directly
        const uint32_t mk = ovf_n && m && bsorted[m - 1] >= ovf_min ? lower_bound_keys(bsorted, m, ovf_min) : m;
        // the next node: unless it is the guess, its offsets load while the list is merged
        uint32_t o0 = g0, o1 = g1;
        bool known = true;
        if (last) {
          unsigned long long t = nold ? old[0] : ~0ull;
          if (mk && bsorted[0] < t) t = bsorted[0];
          if (nold + mk > 0) {
            have = !(key_dist(t) > expR);
            finished = !have;
          }
          if (have && t != guess) {
            known = false;
            o0 = __ldg(g.offsets + key_id(t));
            o1 = __ldg(g.offsets + key_id(t) + 1);
          }
        }
        const uint32_t obase = ovf_n;
        const uint32_t nevict = (nold + mk > cfg.ccap) ? nold + mk - cfg.ccap : 0u;
        for (uint32_t i = tid; i < m - mk; i += T) {
          uint32_t o = obase + i;
          if (o < cfg.ocap) ovf[o] = bsorted[mk + i];
        }
        for (uint32_t i = tid; i < nold; i += T) {
          unsigned long long k = old[i];
          uint32_t pos = i + lower_bound_keys(bsorted, mk, k);
          if (pos < cfg.ccap) cn[pos] = k;
          else {
            uint32_t o = obase + (m - mk) + (pos - cfg.ccap);
            if (o < cfg.ocap) ovf[o] = k;
            if (pos == cfg.ccap) s.evict_min = k;
          }
        }
        for (uint32_t i = tid; i < mk; i += T) {
          unsigned long long k = bsorted[i];
          uint32_t pos = i + lower_bound_keys(old, nold, k);
          if (pos < cfg.ccap) cn[pos] = k;
          else {
            uint32_t o = obase + (m - mk) + (pos - cfg.ccap);
            if (o < cfg.ocap) ovf[o] = k;
            if (pos == cfg.ccap) s.evict_min = k;
          }
        }
        if (have) {
          e0 = o0;
          nsz = min(o1 - o0, P.edge_size);
          if (known) eid = gid;
          else if ((uint32_t)tid < min(nsz, CH)) eid = __ldg(g.edges + e0 + tid);
        }
        __syncthreads();
        const uint32_t added = (m - mk) + nevict;
        if (added) {
          unsigned long long mn = s.evict_min;
          if (mk < m && bsorted[mk] < mn) mn = bsorted[mk];
          if (mn < ovf_min) ovf_min = mn;
          ovf_n += added;
          if (ovf_n > cfg.ocap) { ovf_n = cfg.ocap; status |= kStatusCandidateOverflow; }
        }
        head = have ? 1u : 0u;
        tail = nold + mk - nevict;
        cur ^= 1u;
      }
      if (finished) break;
    }
    // ---- results ---------------------------------------------------------------
    __syncthreads();
    {
      uint32_t n = s.nres;
      if (n > P.size_out) n = P.size_out;       // RESULT_DEFINED_RANGE: cut back to sizeBackup
      for (uint32_t i = tid; i < n; i += T) {
        unsigned long long k = res[i];
        out[P.out_off + i] = ObjDist{key_id(k), key_dist(k)};
      }
      if (tid == 0) {
        out_count[q] = n;
        stats[q] = QueryStats{dc, expansions, nvisited, edges, status};
      }
    }
    if (spilled) {                           // leave the bitmap clean for the next query
      for (uint32_t i = tid; i < cfg.bitmap_words; i += T) bitmap[i] = 0u;
      __threadfence();
    }
    __syncthreads();
  }
}

inline size_t exact_smem_bytes(uint32_t row_chunks, const ExactConfig& c, uint32_t threads = kExactThreads) {
  const size_t chunk = threads < 256 ? threads : 256;
  return (size_t)row_chunks * 16 + ((size_t)c.kcap + 1) / 2 * 16 + (size_t)c.ccap * 16 + chunk * 16 +
         ((size_t)c.hcap + 3) / 4 * 16 + chunk * 12 + sizeof(ExactShared) + 16;
}

}  // namespace ngtg
