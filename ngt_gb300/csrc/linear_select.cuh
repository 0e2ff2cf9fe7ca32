// Top-k selection stage of the exhaustive search (see linear_search.cuh for
// the reference semantics).  Included by exactly one translation unit.
//
// The k smallest 64-bit keys (order_bits(distance) << 32 | id) of a query's
// distances are found by a radix select whose passes run over the whole grid:
// three passes over the distance bits (11 + 11 + 10), then, only while more ties
// at the k-th distance remain than are needed, passes of 11 bits over the ids.
// In each pass every block counts its rows' digits in shared memory, adds its
// non-zero bins to the query's global histogram, and the block that finishes
// last picks the digit (LinearSelect) and clears the histogram for the next pass.
// Once the keys below a prefix are exactly the k wanted, later passes return at
// once.  linear_collect_kernel gathers the keys up to the prefix and its last
// block sorts them.
//
// Why over the grid: the distances of one query are a few MB that L2 holds, and a
// single block reads them at one SM's rate: at 1M rows, k = 100, one 512-thread
// block took 3300 us for its six passes, beside 485 us for the distances; these
// take about 40 us.  The whole call over 1M x 768: 4310 us before, 635 us now (its
// floor, reading the rows at the measured copy bandwidth: 454 us).
#pragma once
#include "linear_search.cuh"

namespace ngtg {

constexpr int kSelThreads = 512;
constexpr uint32_t kSelDigitBits = 11, kSelBins = 1u << kSelDigitBits;
constexpr uint32_t kSelRowsPerBlock = 4096;         // rows of a block of the selection grid, at least

// Selection state of one query (zeroed before the first pass, with hist).
struct LinearSelect {
  unsigned long long prefix;   // digits found so far, at the top of the key
  uint32_t need;               // keys still to take among those with the prefix
  uint32_t kk;                 // results: min(k, valid distances)
  uint32_t all_below;          // 1: every key with the prefix is wanted (no further pass)
  uint32_t ticket;             // blocks done with the current pass
  uint32_t count;              // keys collected
  uint32_t pad;
};

constexpr uint32_t kInfBits = 0xff800000u;   // order_bits(+inf): excluded rows
// Key bits of a distance; NaN (of either sign) orders past +inf, so it is never a result.
__device__ __forceinline__ uint32_t dist_bits(float d) { return d != d ? 0xffffffffu : order_bits(d); }

// One pass: the digit of `bits` bits at `shift` of the 64-bit key (shift >= 32: a
// distance digit).  first: the pass that also counts the valid distances.
__global__ void __launch_bounds__(kSelThreads)
linear_radix_kernel(const float* __restrict__ dist, uint32_t nrows, uint32_t k, uint32_t shift, uint32_t bits,
                    uint32_t first, uint32_t* __restrict__ hist_all, LinearSelect* __restrict__ sel_all) {
  __shared__ uint32_t hist[kSelBins];
  __shared__ uint32_t sh_last, sh_warp[kSelThreads / 32];
  const uint32_t qi = blockIdx.y, tid = threadIdx.x;
  LinearSelect& st = sel_all[qi];
  uint32_t* gh = hist_all + (size_t)qi * kSelBins;
  const float* D = dist + (size_t)qi * nrows;
  if (!first && st.all_below) return;        // written by an earlier launch: uniform over the grid
  const unsigned long long prefix = first ? 0ull : st.prefix;
  const unsigned long long above = shift + bits >= 64 ? 0ull : ~0ull << (shift + bits);   // bits of earlier digits
  const uint32_t dmask = (1u << bits) - 1u;
  for (uint32_t i = tid; i < kSelBins; i += kSelThreads) hist[i] = 0;
  __syncthreads();
  const uint32_t per = (nrows + gridDim.x - 1) / gridDim.x;
  const uint32_t r0 = blockIdx.x * per, r1 = min(nrows, r0 + per);
  for (uint32_t b = r0; b < r1; b += kSelThreads * 4) {
    uint32_t key[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const uint32_t r = b + u * kSelThreads + tid;
      key[u] = r < r1 ? dist_bits(__ldg(D + r)) : 0xffffffffu;
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const unsigned long long x = ((unsigned long long)key[u] << 32) | (b + u * kSelThreads + tid);
      const bool on = key[u] < kInfBits && (x & above) == prefix;
      const uint32_t digit = (uint32_t)(x >> shift) & dmask;
      // distances share few leading digits: the two commonest of a warp are counted once each
      uint32_t left = __ballot_sync(0xffffffffu, on);
#pragma unroll
      for (int t = 0; t < 2; t++) {
        if (left == 0) break;                // warp-uniform
        const int lead = __ffs(left) - 1;
        const uint32_t d = __shfl_sync(0xffffffffu, digit, lead);
        const uint32_t same = __ballot_sync(0xffffffffu, digit == d) & left;
        if ((int)(tid & 31) == lead) atomicAdd(&hist[d], (uint32_t)__popc(same));
        left &= ~same;
      }
      if ((left >> (tid & 31)) & 1u) atomicAdd(&hist[digit], 1u);
    }
  }
  __syncthreads();
  for (uint32_t i = tid; i <= dmask; i += kSelThreads)
    if (hist[i]) atomicAdd(gh + i, hist[i]);
  __threadfence();
  __syncthreads();
  if (tid == 0) sh_last = atomicAdd(&st.ticket, 1u) == gridDim.x - 1 ? 1u : 0u;
  __syncthreads();
  if (!sh_last) return;
  __threadfence();
  // the last block: every thread holds four consecutive bins
  static_assert(kSelBins == 4 * kSelThreads, "four bins per thread");
  uint32_t c[4], sum = 0;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const uint32_t i = tid * 4 + j;
    c[j] = i <= dmask ? __ldcg(gh + i) : 0u;
    sum += c[j];
    if (i <= dmask) gh[i] = 0;
  }
  const uint32_t lane = tid & 31, warp = tid >> 5;
  uint32_t incl = sum;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= (uint32_t)off) incl += y;
  }
  if (lane == 31) sh_warp[warp] = incl;
  __syncthreads();
  uint32_t before = 0, total = 0;
  for (uint32_t w = 0; w < kSelThreads / 32; w++) {
    if (w < warp) before += sh_warp[w];
    total += sh_warp[w];
  }
  const uint32_t excl = before + incl - sum;
  if (tid == 0) st.ticket = 0;
  if (first) {
    if (tid == 0) {
      st.kk = min(k, total);
      st.count = 0;
    }
    if (total <= k) {                        // every valid distance is a result
      if (tid == 0) {
        st.prefix = ~0ull;
        st.all_below = 1;
      }
      return;
    }
  }
  const uint32_t need = first ? k : st.need;
  __syncthreads();                           // st.need is read before one thread rewrites it
  if (excl < need && excl + sum >= need) {
    uint32_t acc = excl, j = 0;
    for (; j < 3; j++) {
      if (acc + c[j] >= need) break;
      acc += c[j];
    }
    // the keys wanted are those up to the prefix with every lower bit set
    const bool all = c[j] == need - acc;
    const unsigned long long p = prefix | ((unsigned long long)(tid * 4 + j) << shift);
    st.prefix = all ? p | ((1ull << shift) - 1ull) : p;
    st.need = need - acc;
    st.all_below = all || shift == 0 ? 1u : 0u;
  }
}

// The kk keys up to the prefix, and (the last block) their order by (distance, id).
// keys: kpow per query, a power of two >= k.
__global__ void __launch_bounds__(kSelThreads)
linear_collect_kernel(const float* __restrict__ dist, uint32_t nrows, uint32_t q0, uint32_t k, uint32_t kpow,
                      LinearSelect* __restrict__ sel_all, unsigned long long* __restrict__ keys_all,
                      ObjDist* __restrict__ out, uint32_t* __restrict__ out_count) {
  extern __shared__ __align__(16) unsigned char smem[];
  unsigned long long* keys = reinterpret_cast<unsigned long long*>(smem);   // kpow
  __shared__ uint32_t sh_last;
  const uint32_t qi = blockIdx.y, tid = threadIdx.x;
  LinearSelect& st = sel_all[qi];
  unsigned long long* gk = keys_all + (size_t)qi * kpow;
  const float* D = dist + (size_t)qi * nrows;
  const unsigned long long prefix = st.prefix;
  const uint32_t kk = st.kk;
  const uint32_t per = (nrows + gridDim.x - 1) / gridDim.x;
  const uint32_t r0 = blockIdx.x * per, r1 = min(nrows, r0 + per);
  for (uint32_t b = r0; b < r1; b += kSelThreads * 4) {
    uint32_t key[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const uint32_t r = b + u * kSelThreads + tid;
      key[u] = r < r1 ? dist_bits(__ldg(D + r)) : 0xffffffffu;
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const unsigned long long x = ((unsigned long long)key[u] << 32) | (b + u * kSelThreads + tid);
      if (key[u] < kInfBits && x <= prefix) {
        const uint32_t slot = atomicAdd(&st.count, 1u);
        if (slot < kk) gk[slot] = x;
      }
    }
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) sh_last = atomicAdd(&st.ticket, 1u) == gridDim.x - 1 ? 1u : 0u;
  __syncthreads();
  if (!sh_last) return;
  __threadfence();
  uint32_t p = 1;
  while (p < kk) p <<= 1;                    // <= kpow
  for (uint32_t i = tid; i < p; i += kSelThreads) keys[i] = i < kk ? __ldcg(gk + i) : ~0ull;
  __syncthreads();
  for (uint32_t k2 = 2; k2 <= p; k2 <<= 1) {
    for (uint32_t j = k2 >> 1; j > 0; j >>= 1) {
      for (uint32_t i = tid; i < p; i += kSelThreads) {
        const uint32_t l = i ^ j;
        if (l > i) {
          const unsigned long long x = keys[i], y = keys[l];
          if ((x > y) == ((i & k2) == 0)) {
            keys[i] = y;
            keys[l] = x;
          }
        }
      }
      __syncthreads();
    }
  }
  for (uint32_t i = tid; i < kk; i += kSelThreads) {
    const unsigned long long x = keys[i];
    out[(size_t)(q0 + qi) * k + i] = ObjDist{(uint32_t)x, order_float((uint32_t)(x >> 32))};
  }
  if (tid == 0) {
    out_count[q0 + qi] = kk;
    st.ticket = 0;
  }
}

}  // namespace ngtg
