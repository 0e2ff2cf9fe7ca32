// Batched graph search with one query per CTA ("wide"): the same relaxed
// best-first search as graph_fast.cuh (sorted candidate list with expanded
// bits, P parents per iteration within (1+epsilon) x r_k, spill tier, exact
// re-rank of the best candidates), with every phase of an iteration spread
// over the CTA so that one query moves many rows at once:
//   * the P parents' edge slots are read, filtered against the query's
//     visited bitmap and compacted by all threads of the CTA (64 to 512);
//   * the new neighbours' search rows (bf16 or 8-bit copies of float objects, or
//     the objects themselves) are loaded straight into registers, several rows per
//     lane group in flight, and scored; a row within the limit goes to the new
//     keys (or the spill tier) at once;
//   * every survivor's place in the list is its rank among the new keys (counted
//     when there are few, else after a sort) plus its rank in the list; keys land
//     in a second list buffer.
// A step takes four CTA barriers: parents chosen, new ids gathered, rows scored,
// list merged.
// One warp (warp 0) owns the control decisions (parent selection, the refill
// from the spill tier), exactly as the warp-per-query kernel makes them.
// Per-query latency is set by a few memory round trips per iteration instead of
// one per 16 rows, which is what a lightly loaded server needs.
#pragma once
#include <cuda_bf16.h>
#include <cfloat>
#include <type_traits>
#include "distance.cuh"
#include "device_index.h"
#include "graph_fast.cuh"

namespace ngtg {

constexpr int kWideMaxThreads = 512;

struct WideConfig {
  uint32_t list_cap;       // L: power of two
  uint32_t nbr_cap;        // neighbour slots per iteration (power of two >= L)
  uint32_t parents;        // P (<= 32)
  uint32_t sgroup;         // lanes per search distance (power of two <= 32)
  uint32_t ngroup;         // lanes per full-precision distance
  uint32_t search_chunks;  // 16-byte chunks per search row
  uint32_t rerank_x16;
  uint32_t bitmap_words;   // per CTA, multiple of 4
  uint32_t smem_bitmap;    // 1: the visited bitmap lies in shared memory
  uint32_t max_iters;
  uint32_t spill_cap;
  uint32_t l2_policy;      // 0: default caching; 1: visited bitmap kept in L2 (evict_last);
                           // 2: as 1, and search rows streamed through L2 (evict_first)
  // 8-bit search rows of float objects: code = rint((x - sq_offset) / s), the query
  // mapped the same way in 1/256 steps; distance = sqrt(sum) * sq_out (s / 256)
  uint32_t sq8, dim;
  uint32_t sq_dot;         // 1: integer dot products give the same distances for whole queries
  float sq_offset, sq_in, sq_out;   // sq_in = 256 / s
};

struct WideShared {
  uint32_t q, n, np, total, cnt, kept, spill_n, done, refill, first_new;
  uint32_t status, dc, expansions, edges;
  uint32_t qnorm, fraction;      // 8-bit rows: the query codes' squared sum; 1: not all whole
  unsigned long long spill_min;
  float limit;
  uint32_t parents[32], pexcl[32], pbase[32];
};

inline size_t wide_smem_bytes(uint32_t row_chunks, const WideConfig& c) {
  size_t b = (size_t)row_chunks * 16 + (size_t)c.search_chunks * (c.sq8 ? 64 + 16 : 16);
  b += (size_t)c.list_cap * 16;                                   // list, double-buffered
  b += (size_t)c.nbr_cap * 4;                                     // new ids
  b += (size_t)kWideMaxThreads * 8;                               // sorted new keys / histogram
  b += (size_t)c.nbr_cap * 8;                                     // new keys
  b += (sizeof(WideShared) + 15) / 16 * 16 + 16;
  if (c.smem_bitmap) b += (size_t)c.bitmap_words * 4;
  return b;
}

// A 16-byte chunk of a search row, read once: no place in L1, and L2 by `policy`.
__device__ __forceinline__ uint4 load_row_chunk(const uint4* p, uint64_t policy) {
  uint4 v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
      : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
      : "l"(p), "l"(policy));
  return v;
}
// atomicOr on a visited-bitmap word, with an L2 eviction-priority hint when `hint`
__device__ __forceinline__ uint32_t visit_or(uint32_t* word, uint32_t bit, bool hint, uint64_t policy) {
  if (!hint) return atomicOr(word, bit);
  uint32_t old;
  asm volatile("atom.global.or.L2::cache_hint.b32 %0, [%1], %2, %3;\n"
               : "=r"(old) : "l"(word), "r"(bit), "l"(policy) : "memory");
  return old;
}
// The same without a branch: where `on` is false nothing is touched and the bit reads as set.
// A step's atomics then all go out before the first result is waited for.
__device__ __forceinline__ uint32_t visit_or_if(bool on, uint32_t* word, uint32_t bit, uint64_t policy) {
  uint32_t old;
  asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %4, 0;\nmov.u32 %0, %2;\n"
               "@p atom.global.or.L2::cache_hint.b32 %0, [%1], %2, %3;\n}\n"
               : "=&r"(old) : "l"(word), "r"(bit), "l"(policy), "r"((uint32_t)on) : "memory");
  return old;
}
__device__ __forceinline__ void store_zero16(uint4* p, bool hint, uint64_t policy) {
  if (!hint) { *p = make_uint4(0, 0, 0, 0); return; }
  asm volatile("st.global.L2::cache_hint.v4.u32 [%0], {%1, %1, %1, %1}, %2;\n" ::"l"(p), "r"(0u), "l"(policy)
               : "memory");
}
__device__ __forceinline__ uint64_t l2_policy_evict_last() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;\n" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t l2_policy_evict_normal() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;\n" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t l2_policy_evict_first() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;\n" : "=l"(p));
  return p;
}

// CTA-wide ascending bitonic sort of a[0..n) (shared memory), padded with ~0 to
// the next power of two (<= cap).
__device__ __forceinline__ void cta_bitonic_sort(unsigned long long* a, uint32_t n, uint32_t cap) {
  if (n <= 1) return;
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

// (row - query)^2 of one 16-byte row chunk, two float lanes at a time, against the
// query chunk prepared once per query: bf16 / fp32 rows through PackedL2, 8-bit
// rows of float objects (Sq8) by placing each code in the mantissa of 2^23
// (2^23 + 256 c, one byte permute) and adding the negated 2^23 + rint(256 q'),
// so that the difference 256 (c - q') is exact.
template <ObjType ST, ObjType OT, Metric M>
struct WideDot {
  typedef PackedL2<ST, M> PL;
  static constexpr bool kSq8 = ST == ObjType::Uint8 && OT == ObjType::Float && M == Metric::L2;
  static constexpr bool kOn = kSq8 || PL::kOn;
  static constexpr int NQ = kSq8 ? 8 : (PL::P / 2 > 0 ? PL::P / 2 : 1);
  // query chunk c: qs holds the search-type query (4 uint4 of floats per chunk for Sq8)
  __device__ __forceinline__ static void prepare(const uint4* qs, uint32_t c, float2 (&nq)[NQ]) {
    if constexpr (kSq8) {
      const float2* f = reinterpret_cast<const float2*>(qs + 4 * (size_t)c);
#pragma unroll
      for (int i = 0; i < 8; i++) nq[i] = f[i];
    } else if constexpr (PL::kOn) {
      PL::prepare(qs[c], nq);
    }
  }
  __device__ __forceinline__ static void zero(float2 (&nq)[NQ]) {
#pragma unroll
    for (int i = 0; i < NQ; i++) nq[i] = make_float2(0.f, 0.f);
  }
  __device__ __forceinline__ static float2 add(float2 acc, const float2 (&nq)[NQ], const uint4& x) {
    if constexpr (kSq8) {
      const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const float a = __uint_as_float(__byte_perm(w[i], 0x4B000000u, 0x7504u));
        const float b = __uint_as_float(__byte_perm(w[i], 0x4B000000u, 0x7514u));
        const float c = __uint_as_float(__byte_perm(w[i], 0x4B000000u, 0x7524u));
        const float d = __uint_as_float(__byte_perm(w[i], 0x4B000000u, 0x7534u));
        const float2 d0 = __fadd2_rn(make_float2(a, b), nq[2 * i]);
        const float2 d1 = __fadd2_rn(make_float2(c, d), nq[2 * i + 1]);
        acc = __ffma2_rn(d0, d0, acc);
        acc = __ffma2_rn(d1, d1, acc);
      }
      return acc;
    } else if constexpr (PL::kOn) {
      return PL::add(acc, nq, x);
    } else {
      return acc;
    }
  }
};

// The KR sums over SG lanes of partial sums v (a group's lanes lie side by side; KR and SG
// powers of two), the rows spread over the lanes: each exchange with the lane `off` away
// halves the rows a lane still adds up, then the rest of the lanes are added to all.  A lane
// ends with the sums of rows first .. in v[0 ..] (max(KR / SG, 1) of them); the lanes without
// one of their own get first = 2^31 - 1.  The pairs added are a butterfly's.
template <uint32_t KR, class Add>
__device__ __forceinline__ uint32_t group_sums(uint32_t (&v)[KR], int SG, int lane, Add add) {
  uint32_t first = 0;
  int off = SG >> 1;
#pragma unroll
  for (uint32_t h = KR / 2; h > 0; h >>= 1) {
    if (off > 0) {
      const bool up = (lane & off) != 0;
#pragma unroll
      for (uint32_t i = 0; i < h; i++) {
        const uint32_t send = up ? v[i] : v[i + h], keep = up ? v[i + h] : v[i];
        v[i] = add(keep, __shfl_xor_sync(0xffffffffu, send, off));
      }
      if (up) first += h;
      off >>= 1;
    }
  }
  if (off > 0) {
    if (lane & (2 * off - 1)) first = 0x7fffffffu;
    for (; off > 0; off >>= 1) v[0] = add(v[0], __shfl_xor_sync(0xffffffffu, v[0], off));
  }
  return first;
}

// T: threads per CTA (64, 128, 256 or 512), one query per CTA.
// Bound by the dependent round trips of a step (parents' offsets, edges, visited bits,
// rows) and by instruction issue: 0.97M warp instructions per query of 22,400 rows before
// the integer dot products, 0.55 issued per cycle and scheduler.  Measured on 1M x 128,
// 8-bit rows, k = 10, epsilon 0.08, 10,000 queries, 128 threads: 15.35 ms with a shared-memory
// row stage (two barriers per 64 rows); rows loaded into registers 15.1 ms; dot products
// 14.2 ms; one body for every number of rows, sums spread over the lanes 12.55 ms (stalls per
// issue on instruction fetches 2.8 -> 0.4); visited-bit updates without a branch each 11.5 ms;
// row loads likewise, a batch ahead 9.2 ms.  152 queries: 1.22 ms with 256 threads, 1.03 ms with
// 512 and the visited bitmap in shared memory.  200k x 100 cosine, 1,500 queries from host
// buffers: 1.80 -> 1.0 ms (packed lanes, three CTAs per SM instead of two).  Not kept:
// prefetching a step's rows into L2 when they are gathered (5 % slower), 1,024 threads (8 %
// slower than 512), seven and eight CTAs an SM (10 and 24 % slower: their visited bitmaps of
// 125 KB no longer fit L2; eight on 200k x 64, bitmaps of 25 KB, 10 %).
template <ObjType ST, ObjType OT, Metric M, int T>
__global__ void __launch_bounds__(T, T == 64 ? 10 : T == 128 ? 6 : T == 256 ? 3 : 1)
graph_search_wide_kernel(DevGraph g, const uint4* __restrict__ srows, const uint4* __restrict__ queries,
                         uint32_t nq, const QueryParams* __restrict__ params, const uint32_t* __restrict__ seed_list,
                         ObjDist* __restrict__ out, uint32_t* __restrict__ out_count, QueryStats* __restrict__ stats,
                         uint32_t* __restrict__ bitmaps, uint32_t* __restrict__ work,
                         unsigned long long* __restrict__ spills, WideConfig cfg) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t rc = g.row_chunks, sc = cfg.search_chunks;
  const uint32_t L = cfg.list_cap, NB = cfg.nbr_cap;
  uint4* qn = reinterpret_cast<uint4*>(smem);
  typedef WideDot<ST, OT, M> Dot;
  uint4* qs = qn + rc;                                                           // sc (x 4 for Sq8) chunks
  unsigned long long* lists = reinterpret_cast<unsigned long long*>(qs + (Dot::kSq8 ? 4 * sc : sc));   // 2 x L
  unsigned long long* nkey = lists + 2 * (size_t)L;                              // NB new keys
  unsigned long long* nsorted = nkey + NB;                                       // up to T of them, sorted
  uint32_t* nid = reinterpret_cast<uint32_t*>(nsorted + kWideMaxThreads);        // NB new ids
  uint8_t* qcode = reinterpret_cast<uint8_t*>(nid + NB);                         // Sq8: 16 sc query codes
  WideShared& s = *reinterpret_cast<WideShared*>(qcode + (Dot::kSq8 ? 16 * sc : 0));
  uint32_t* sbitmap = reinterpret_cast<uint32_t*>(reinterpret_cast<unsigned char*>(&s) + (sizeof(WideShared) + 15) / 16 * 16);
  uint32_t* bitmap = bitmaps + (size_t)blockIdx.x * cfg.bitmap_words;
  unsigned long long* spill = spills + (size_t)blockIdx.x * 2 * cfg.spill_cap;
  unsigned long long* spill_tmp = spill + cfg.spill_cap;
  const int SG = (int)cfg.sgroup, NG = (int)cfg.ngroup;
  const int sgl = lane & (SG - 1);
  const bool keep_visited = cfg.l2_policy >= 1, stream_rows = cfg.l2_policy >= 2;
  const uint64_t pol_keep = keep_visited ? l2_policy_evict_last() : l2_policy_evict_normal();
  const uint64_t pol_stream = stream_rows ? l2_policy_evict_first() : l2_policy_evict_normal();

  // A scored row within the limit: below the list's worst entry it joins the new keys,
  // else the spill tier.  Rows past the limit are not kept (their sums need no root).
  struct Limits {
    float limit;                 // largest distance kept
    float far;                   // sums past it are past the limit beyond doubt
    unsigned long long worst;    // keys from here on go to the spill tier
    bool all;                    // seeds: every distance is kept
  };
  auto place = [&](float d, uint32_t id, const Limits& w) {
    if (!(d <= w.limit) && !w.all) return;
    const unsigned long long key = pack_key(d, id);
    if (key < w.worst || w.all) {
      nkey[atomicAdd(&s.kept, 1u)] = key;
    } else {
      const uint32_t o = atomicAdd(&s.spill_n, 1u);
      if (o < cfg.spill_cap) spill[o] = key;
      atomicMin(&s.spill_min, key);
    }
  };
  // scores nid[0..cnt): every lane group loads the chunks of several rows before it adds any
  // up.  Lanes, chunks and the order of summation are the same for every number of rows.
  // One body for every number of rows and one call of it in the kernel: with bodies for 8, 4,
  // 2 and 1 rows, once for the seeds and once for the steps, a sixth of the warps' time went
  // on instruction fetches, and a step's last rows took up to three round trips.
  auto score = [&](uint32_t cnt, const Limits& w) {
    const uint32_t gpb = (uint32_t)T / SG;
    const uint32_t gi = (uint32_t)(tid / SG);
    constexpr int kQC = Dot::kSq8 ? 1 : 2;
    if (Dot::kOn && sc <= (uint32_t)(kQC * SG)) {
      // the query chunks this lane reads (c = sgl + j * SG), negated and unpacked once; the
      // host sets sgroup so that a lane reads at most two chunks (one for 8-bit rows)
      float2 nqc[kQC][Dot::NQ];
      auto prepare = [&]() {
#pragma unroll
        for (int j = 0; j < kQC; j++) {
          const uint32_t c = (uint32_t)sgl + (uint32_t)(j * SG);
          if (c < sc) Dot::prepare(qs, c, nqc[j]);
          else Dot::zero(nqc[j]);
        }
      };
      if (!Dot::kSq8) prepare();                 // 8-bit rows: with each batch, the registers are needed
      const bool dots = Dot::kSq8 && s.fraction == 0;
      const uint4 qc = dots && (uint32_t)sgl < sc ? reinterpret_cast<const uint4*>(qcode)[sgl] : make_uint4(0, 0, 0, 0);
      // KR rows a lane group and batch (8-bit rows: 4 take 14.0 ms on the sizes above, 8 take
      // 11.5, 16 with four or five CTAs an SM as long as 8)
      constexpr uint32_t KR = Dot::kSq8 ? 8 : 4;
      const uint32_t step = KR * gpb;
      uint4 x[KR][kQC];
      // Without a branch: past cnt the last row, past a row's end its last chunk, neither of
      // which counts.  The loads of a batch with a branch each cost 11.5 instead of 9.9 ms.
      auto load = [&](uint32_t u, uint32_t b) {
        const uint32_t id = nid[min(b + u * gpb + gi, cnt - 1)];
#pragma unroll
        for (int j = 0; j < kQC; j++)
          x[u][j] = load_row_chunk(srows + (size_t)id * sc + min((uint32_t)sgl + (uint32_t)(j * SG), sc - 1),
                                   pol_stream);
      };
      if (cnt > 0) {
#pragma unroll
        for (uint32_t u = 0; u < KR; u++) load(u, 0);
      }
      for (uint32_t b = 0; b < cnt; b += step) {               // uniform over the CTA
        const bool more = b + step < cnt;
        const uint32_t nu = min(KR, (cnt - b + gpb - 1) / gpb);
        uint32_t sum[KR];                                      // a lane's part of each row's sum, as bits
        uint32_t first;                                        // the first of the rows whose sum it holds then
        // the next batch's rows are loaded as this one's are taken (9.9 -> 9.2 ms)
        auto take = [&](auto part) {
          if (more) {
#pragma unroll
            for (uint32_t u = 0; u < KR; u++) {
              sum[u] = part(x[u]);
              load(u, b + step);
            }
          } else {
#pragma unroll
            for (uint32_t u = 0; u < KR; u++) sum[u] = part(x[u]);
          }
        };
        if (Dot::kSq8 && dots) {
          // sum (c - q)^2 = sum c c - 2 sum c q + sum q q over whole codes, exact in 32 bits;
          // times 2^16 it is the sum of the squared 1/256 steps that the float form adds up
          // (exact there too, below 2^24 steps of one)
          take([&](const uint4 (&y)[kQC]) {
            uint32_t cc = 0, cq = 0;
            cc = __dp4a(y[0].x, y[0].x, cc); cq = __dp4a(y[0].x, qc.x, cq);
            cc = __dp4a(y[0].y, y[0].y, cc); cq = __dp4a(y[0].y, qc.y, cq);
            cc = __dp4a(y[0].z, y[0].z, cc); cq = __dp4a(y[0].z, qc.z, cq);
            cc = __dp4a(y[0].w, y[0].w, cc); cq = __dp4a(y[0].w, qc.w, cq);
            return (uint32_t)sgl < sc ? cc - 2u * cq : 0u;
          });
          first = group_sums<KR>(sum, SG, lane, [](uint32_t p, uint32_t r) { return p + r; });
        } else {
          if (Dot::kSq8) prepare();
          take([&](const uint4 (&y)[kQC]) {
            float2 acc[kQC];
#pragma unroll
            for (int j = 0; j < kQC; j++) {
              acc[j] = make_float2(0.f, 0.f);
              if ((uint32_t)sgl + (uint32_t)(j * SG) < sc) acc[j] = Dot::add(acc[j], nqc[j], y[j]);
            }
            float t = acc[0].x + acc[0].y;
#pragma unroll
            for (int j = 1; j < kQC; j++) t += acc[j].x + acc[j].y;
            return __float_as_uint(t);
          });
          first = group_sums<KR>(sum, SG, lane, [](uint32_t p, uint32_t r) {
            return __float_as_uint(__uint_as_float(p) + __uint_as_float(r));
          });
        }
        const uint32_t held = max(KR / (uint32_t)SG, 1u);
        for (uint32_t r = 0; r < held && first + r < nu; r++) {
          uint32_t bits = sum[0];
#pragma unroll
          for (uint32_t k = 1; k < KR; k++) bits = r == k ? sum[k] : bits;
          const float v = dots ? (float)((int)bits + (int)s.qnorm) * 65536.f : __uint_as_float(bits);
          const uint32_t i = b + (first + r) * gpb + gi;
          if (i < cnt && !(v > w.far)) place(Dot::kSq8 ? sqrtf(v) * cfg.sq_out : sqrtf(v), nid[i], w);
        }
      }
    } else if constexpr (Dot::kOn) {
      // long rows: chunk after chunk, two rows at once
      for (uint32_t b = 0; b < cnt; b += 2 * gpb) {
        float2 acc[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        uint32_t id[2];
#pragma unroll
        for (int u = 0; u < 2; u++) {
          const uint32_t i = b + (uint32_t)u * gpb + gi;
          id[u] = i < cnt ? nid[i] : 0u;
        }
#pragma unroll 2
        for (uint32_t c = (uint32_t)sgl; c < sc; c += (uint32_t)SG) {
          float2 nq[Dot::NQ];
          uint4 x[2];
#pragma unroll
          for (int u = 0; u < 2; u++) x[u] = load_row_chunk(srows + (size_t)id[u] * sc + c, pol_stream);
          Dot::prepare(qs, c, nq);
#pragma unroll
          for (int u = 0; u < 2; u++) acc[u] = Dot::add(acc[u], nq, x[u]);
        }
#pragma unroll
        for (int u = 0; u < 2; u++) {
          float v = acc[u].x + acc[u].y;
#pragma unroll
          for (int off = 16; off > 0; off >>= 1)
            if (off < SG) v += __shfl_xor_sync(0xffffffffu, v, off);
          const uint32_t i = b + (uint32_t)u * gpb + gi;
          if (i < cnt && sgl == 0 && !(v > w.far)) place(Dot::kSq8 ? sqrtf(v) * cfg.sq_out : sqrtf(v), id[u], w);
        }
      }
    } else {
      // the objects' own comparator, the lanes of a group packed four to a thread
      const int pw = packed_width(SG);
      const uint32_t ppb = (uint32_t)T / (uint32_t)pw;
      for (uint32_t b = 0; b < cnt; b += ppb) {
        const uint32_t i = b + (uint32_t)(tid / pw);
        const uint32_t id[1] = {i < cnt ? nid[i] : 0u};
        Acc<ST, M> sum[1];
        packed_sums<ST, M, 1>(qs, srows, id, (int)sc, lane & (pw - 1), SG, sum);
        if (i < cnt && (lane & (pw - 1)) == 0) place(sum[0].finish(), id[0], w);
      }
    }
  };

  // true when `id` was not visited yet (and marks it)
  auto visit = [&](uint32_t id) {
    const uint32_t bit = 1u << (id & 31u);
    if (cfg.smem_bitmap) return (atomicOr(&sbitmap[id >> 5], bit) & bit) == 0u;
    return (visit_or(&bitmap[id >> 5], bit, keep_visited, pol_keep) & bit) == 0u;
  };
  while (true) {
    if (tid == 0) {
      s.q = atomicAdd(work, 1u);
      s.qnorm = 0;
      s.fraction = 0;
    }
    __syncthreads();
    const uint32_t q = s.q;
    if (q >= nq) break;
    const QueryParams P = params[q];
    for (uint32_t i = tid; i < rc; i += blockDim.x) qn[i] = queries[(size_t)q * rc + i];
    if (cfg.smem_bitmap)
      for (uint32_t i = tid; i < cfg.bitmap_words / 4; i += blockDim.x)
        reinterpret_cast<uint4*>(sbitmap)[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    if constexpr (Dot::kSq8) {
      // 16 negated values per row chunk: -(2^23 + rint(256 (q - offset) / s)), 0 past dim
      const float* qf = reinterpret_cast<const float*>(qn);
      float* qv = reinterpret_cast<float*>(qs);
      bool whole = cfg.sq_dot != 0;
      uint32_t qq = 0;
      for (uint32_t i = tid; i < sc * 16; i += blockDim.x) {
        float v = 0.f;
        if (i < cfg.dim) v = fminf(fmaxf(rintf((qf[i] - cfg.sq_offset) * cfg.sq_in), -8388607.f), 8388607.f);
        qv[i] = -(8388608.f + v);
        // a query of whole codes 0..255 is scored by integer dot products
        const float c = v * (1.f / 256.f);
        const bool code = c >= 0.f && c <= 255.f && c == rintf(c);
        whole = whole && code;
        const uint32_t u = code ? (uint32_t)c : 0u;
        qcode[i] = (uint8_t)u;
        qq += u * u;
      }
      qq = __reduce_add_sync(0xffffffffu, qq);
      if (lane == 0 && qq) atomicAdd(&s.qnorm, qq);
      if (!whole) s.fraction = 1;
    } else if constexpr (ST != OT) {
      const float* qf = reinterpret_cast<const float*>(qn);
      uint32_t* qb = reinterpret_cast<uint32_t*>(qs);
      for (uint32_t i = tid; i < sc * 4; i += blockDim.x) {
        uint32_t lo = __bfloat16_as_ushort(__float2bfloat16_rn(qf[2 * i]));
        uint32_t hi = __bfloat16_as_ushort(__float2bfloat16_rn(qf[2 * i + 1]));
        qb[i] = lo | (hi << 16);
      }
    } else {
      for (uint32_t i = tid; i < sc; i += blockDim.x) qs[i] = qn[i];
    }
    if (tid == 0) {
      s.spill_n = 0; s.spill_min = ~0ull; s.refill = 0; s.first_new = 0xffffffffu; s.kept = 0;
      s.status = 0; s.dc = 0; s.expansions = 0; s.edges = 0;
    }
    __syncthreads();
    if (P.size == 0) {
      if (tid == 0) { out_count[q] = 0; stats[q] = QueryStats{0, 0, 0, 0, 0}; }
      __syncthreads();
      continue;
    }
    // ---- seeds (warp 0): tree leaf or explicit list, marked visited, compacted ----
    if (warp == 0) {
      const uint32_t* seeds = nullptr;
      uint32_t nseeds = 0, st = 0;
      if (P.seed_cnt == 0xffffffffu) {
        uint32_t node = g.root;
        int depth = 0;
        while (!(node & 0x80000000u) && depth < 64) {
          const DevInternal& in = g.internals[node];
          float d = group_distance<TreeSpace<OT, M>::ot, TreeSpace<OT, M>::m>(qn, g.pivots + (size_t)in.pivot * rc, (int)rc, lane, 32);
          uint32_t bsize = in.nchildren - 1, mid;
          for (mid = 0; mid < bsize; mid++)
            if (d < in.borders[mid]) break;
          node = in.children[mid];
          depth++;
        }
        if (node & 0x80000000u) {
          uint32_t leaf = node & 0x7fffffffu;
          if (leaf < g.nleaves) {
            const uint32_t* off = g.leaf_seed_off + P.seed_off;
            seeds = g.leaf_seed_ids + off[leaf];
            nseeds = off[leaf + 1] - off[leaf];
          }
        } else {
          st |= kStatusTreeError;
        }
      } else {
        seeds = seed_list + P.seed_off;
        nseeds = P.seed_cnt;
      }
      nseeds = min(nseeds, NB);
      if (nseeds == 0) st |= kStatusEmptySeeds;
      uint32_t m = 0;
      for (uint32_t b = 0; b < nseeds; b += 32) {
        uint32_t i = b + lane;
        bool fresh = false;
        uint32_t id = 0;
        if (i < nseeds) {
          id = seeds[i];
          if (id < g.nrows) fresh = visit(id);
        }
        unsigned bal = __ballot_sync(0xffffffffu, fresh);
        if (fresh) nid[m + __popc(bal & ((1u << lane) - 1u))] = id;
        m += __popc(bal);
      }
      if (lane == 0) { s.cnt = m; s.status |= st; s.dc = m; }
    }
    __syncthreads();
    // Alike in every thread: the list is lists[cur * L ..], n entries; warp 0 also keeps
    // the first entry that may be unexpanded.
    uint32_t n = 0, cur = 0, scan0 = 0;
    const float user_radius = P.radius;

    // ---- the seeds' step (it = 0), then best-first iterations ----------------------------
    for (uint32_t it = 0; it == 0 || it - 1 < cfg.max_iters; it++) {
      if (it > 0) {
      // control (warp 0): refill from the spill tier when flagged, then pick parents
      if (warp == 0) {
        unsigned long long* list = lists + (size_t)cur * L;
        uint32_t spill_n = s.spill_n;
        unsigned long long spill_min = s.spill_min;
        const bool refill = s.refill != 0;
        scan0 = min(scan0, s.first_new);
        __syncwarp();
        if (spill_n > cfg.spill_cap) {
          spill_n = cfg.spill_cap;
          if (lane == 0) s.status |= kStatusCandidateOverflow;
        }
        float rk = (n >= P.size) ? fminf(key_dist(list[P.size - 1]), user_radius) : user_radius;
        const float limit = P.coef * rk;
        if (refill) {
          n = min(n, P.size);
          const uint32_t room = L - n;
          uint32_t r = 0;
          for (uint32_t b = 0; b < spill_n; b += 32) {
            uint32_t i = b + lane;
            unsigned long long k = i < spill_n ? spill[i] : ~0ull;
            bool live = i < spill_n && key_dist(k) <= limit;
            unsigned bal = __ballot_sync(0xffffffffu, live);
            if (live) spill_tmp[r + __popc(bal & ((1u << lane) - 1u))] = k;
            r += __popc(bal);
          }
          __syncwarp();
          unsigned long long thr = ~0ull;
          if (r > room) {
            unsigned long long prefix = 0, mask = 0;
            uint32_t need = room;
            uint32_t* hist = reinterpret_cast<uint32_t*>(nsorted);
            for (int shift = 56; shift >= 0; shift -= 8) {
              for (uint32_t i = lane; i < 256; i += 32) hist[i] = 0;
              __syncwarp();
              for (uint32_t i = lane; i < r; i += 32) {
                unsigned long long k = spill_tmp[i];
                if ((k & mask) == prefix) atomicAdd(&hist[(uint32_t)(k >> shift) & 255u], 1u);
              }
              __syncwarp();
              uint32_t acc = 0, bsel = 255;
              for (uint32_t b = 0; b < 256; b++) {
                uint32_t h = hist[b];
                if (acc + h >= need) { bsel = b; break; }
                acc += h;
              }
              prefix |= (unsigned long long)bsel << shift;
              need -= acc;
              mask |= 255ull << shift;
              __syncwarp();
            }
            thr = prefix;
          }
          uint32_t moved = 0, stay = 0;
          unsigned long long smin = ~0ull;
          for (uint32_t b = 0; b < r; b += 32) {
            uint32_t i = b + lane;
            unsigned long long k = i < r ? spill_tmp[i] : ~0ull;
            bool take = i < r && k <= thr;
            bool keep = i < r && k > thr;
            unsigned bt = __ballot_sync(0xffffffffu, take), bk = __ballot_sync(0xffffffffu, keep);
            if (take) nkey[moved + __popc(bt & ((1u << lane) - 1u))] = k;
            if (keep) { spill[stay + __popc(bk & ((1u << lane) - 1u))] = k; smin = k < smin ? k : smin; }
            moved += __popc(bt);
            stay += __popc(bk);
          }
          for (int off = 16; off > 0; off >>= 1) {
            unsigned long long o = __shfl_xor_sync(0xffffffffu, smin, off);
            smin = o < smin ? o : smin;
          }
          __syncwarp();
          warp_bitonic_sort(nkey, moved, lane);
          for (uint32_t i = lane; i < moved; i += 32) list[n + i] = nkey[i];
          __syncwarp();
          scan0 = n;
          n += moved;
          spill_n = stay;
          spill_min = smin;
        }
        uint32_t np = 0;
        bool stop = false;
        for (uint32_t b = scan0 & ~31u; b < n && !stop && np < cfg.parents; b += 32) {
          uint32_t i = b + lane;
          unsigned long long k = i < n ? list[i] : ~0ull;
          // the unexpanded entries within the limit, in order, as many as there is room for
          const unsigned open = __ballot_sync(0xffffffffu, i < n && !key_expanded(k));
          const unsigned within = open & __ballot_sync(0xffffffffu, i < n && !(key_dist(k) > limit));
          const uint32_t rank = (uint32_t)__popc(within & ((1u << lane) - 1u));
          const bool take = ((within >> lane) & 1u) && np + rank < cfg.parents;
          if (take) {
            list[i] = k | kExpandedBit;
            s.parents[np + rank] = key_rawid(k);
          }
          const unsigned taken = __ballot_sync(0xffffffffu, take);
          if (taken) scan0 = b + 32u - (uint32_t)__clz((int)taken);
          np += (uint32_t)__popc(taken);
          stop = np < cfg.parents && open != within;       // the list is sorted: the rest is past the limit
        }
        __syncwarp();
        uint32_t done = 0, next_refill = 0;
        if (np == 0) {
          if (!stop && spill_n > 0 && key_dist(spill_min) <= limit) {
            scan0 = n;
            next_refill = 1;
          } else {
            done = 1;
          }
        } else {
          // edge slots of the parents
          const uint32_t per_parent = min(P.edge_size, NB / np);
          uint32_t pe0 = 0, pne = 0;
          if ((uint32_t)lane < np) {
            const uint32_t v = s.parents[lane];
            const uint32_t a = g.offsets[v];
            pe0 = a;
            pne = min(g.offsets[v + 1] - a, per_parent);
          }
          uint32_t incl = pne;
#pragma unroll
          for (int off = 1; off < 32; off <<= 1) {
            uint32_t t = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += t;
          }
          const uint32_t total = __shfl_sync(0xffffffffu, incl, np - 1);
          if ((uint32_t)lane < np) {
            s.pexcl[lane] = incl - pne;
            s.pbase[lane] = pe0;
          }
          if (lane == 0) { s.total = total; s.edges += total; s.expansions += np; }
        }
        if (lane == 0) {
          s.n = n; s.spill_n = spill_n; s.spill_min = spill_min;
          s.refill = next_refill; s.done = done; s.np = np; s.limit = limit;
          // counters of this step's gather, placement and merge
          s.cnt = 0; s.kept = 0; s.first_new = 0xffffffffu;
        }
      }
      __syncthreads();
      const uint32_t done = s.done, refill_next = s.refill, np = s.np, total = s.total;
      n = s.n;
      if (done) break;
      if (refill_next) {
        __syncthreads();            // everyone has read the decision before warp 0 writes the next one
        continue;
      }
      // ---- gather: unvisited neighbours of the parents ----------------------------------
      // Every thread takes up to kGatherSlots edge slots (t = base + j*T + tid): all
      // edge loads, then all visited-bit atomics, then one CTA scan of the per-thread
      // counts places the new ids (their order does not matter to this search).
      constexpr int kGatherSlots = T >= 512 ? 2 : 8;
      for (uint32_t base0 = 0; base0 < total; base0 += kGatherSlots * (uint32_t)T) {
        uint32_t ids[kGatherSlots];
        uint32_t fm = 0, p2 = 0;
#pragma unroll
        for (int j = 0; j < kGatherSlots; j++) {
          const uint32_t t = base0 + (uint32_t)j * (uint32_t)T + (uint32_t)tid;
          ids[j] = 0;
          if (t < total) {
            while (p2 + 1 < np && t >= s.pexcl[p2 + 1]) p2++;       // slots increase with j
            ids[j] = __ldg(g.edges + s.pbase[p2] + (t - s.pexcl[p2]));
          }
        }
        if (cfg.smem_bitmap) {
#pragma unroll
          for (int j = 0; j < kGatherSlots; j++) {
            const uint32_t t = base0 + (uint32_t)j * (uint32_t)T + (uint32_t)tid;
            if (t < total && visit(ids[j])) fm |= 1u << j;
          }
        } else {
          uint32_t old[kGatherSlots];
#pragma unroll
          for (int j = 0; j < kGatherSlots; j++) {
            const uint32_t t = base0 + (uint32_t)j * (uint32_t)T + (uint32_t)tid;
            old[j] = visit_or_if(t < total, &bitmap[ids[j] >> 5], 1u << (ids[j] & 31u), pol_keep);
          }
#pragma unroll
          for (int j = 0; j < kGatherSlots; j++)
            if (!((old[j] >> (ids[j] & 31u)) & 1u)) fm |= 1u << j;
        }
        // places in nid: a warp scan of the per-thread counts and one counter
        // increment per warp (the order of the new ids does not matter to this search)
        const uint32_t c = (uint32_t)__popc(fm);
        uint32_t incl = c;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          uint32_t v = __shfl_up_sync(0xffffffffu, incl, off);
          if (lane >= off) incl += v;
        }
        uint32_t wbase = 0;
        if (lane == 31 && incl) wbase = atomicAdd(&s.cnt, incl);
        wbase = __shfl_sync(0xffffffffu, wbase, 31);
        uint32_t pos = wbase + incl - c;
#pragma unroll
        for (int j = 0; j < kGatherSlots; j++)
          if (fm & (1u << j)) nid[pos++] = ids[j];
      }
      __syncthreads();
      if (tid == 0) s.dc += s.cnt;
      }
      const uint32_t cnt = s.cnt;
      // ---- distances and placement: below the list's worst -> new keys; else spill ----------
      const unsigned long long* list = lists + (size_t)cur * L;
      {
        const float rk = (n >= P.size) ? fminf(key_dist(list[P.size - 1]), user_radius) : user_radius;
        Limits w;
        w.limit = P.coef * rk;
        const float root = Dot::kSq8 ? w.limit / cfg.sq_out : w.limit;
        w.far = it == 0 ? INFINITY : root * root * 1.0001f;
        w.worst = (n >= L) ? (list[L - 1] & ~(unsigned long long)kExpandedBit) : ~0ull;
        w.all = it == 0;                                       // every seed is kept
        score(cnt, w);
      }
      __syncthreads();
      if (it == 0) {
        cta_bitonic_sort(nkey, cnt, NB);
        n = min(cnt, L);
        for (uint32_t i = tid; i < n; i += blockDim.x) lists[i] = nkey[i];
        __syncthreads();
        continue;
      }
      const uint32_t kept = s.kept;
      if (kept == 0) {
        __syncthreads();            // everyone has read the counter before warp 0 clears it
        continue;
      }
      // ---- merge into the other list buffer (entries compare without the expanded bit) ---
      // Every key's place is its rank among the new keys plus its rank among the list's.
      // Few new keys are counted against (no barrier); more are sorted first, up to T by
      // rank, and searched.
      const bool by_count = kept <= 12;
      const unsigned long long* nk = nkey;
      if (!by_count) {
        if (kept <= (uint32_t)T) {
          rank_sort_split<T>(nkey, nsorted, kept);
          nk = nsorted;
          __syncthreads();
        } else {
          cta_bitonic_sort(nkey, kept, NB);
        }
      }
      auto rank_new = [&](unsigned long long x) -> uint32_t {
        if (!by_count) return warp_lower_bound(nk, kept, x);
        uint32_t r = 0;
        for (uint32_t t = 0; t < kept; t++) r += nk[t] < x ? 1u : 0u;
        return r;
      };
      unsigned long long* dst = lists + (size_t)(cur ^ 1u) * L;
      for (uint32_t i = tid; i < n; i += blockDim.x) {
        const unsigned long long k = list[i];
        const uint32_t pos = i + rank_new(k & ~(unsigned long long)kExpandedBit);
        if (pos < L) dst[pos] = k;
        else if (!key_expanded(k)) {
          const uint32_t o = atomicAdd(&s.spill_n, 1u);
          if (o < cfg.spill_cap) spill[o] = k;
          atomicMin(&s.spill_min, k);
        }
      }
      for (uint32_t j = tid; j < kept; j += blockDim.x) {
        const unsigned long long k = nk[j];
        uint32_t lo = 0, hi = n;
        while (lo < hi) {
          uint32_t mid = (lo + hi) >> 1;
          if ((list[mid] & ~(unsigned long long)kExpandedBit) < k) lo = mid + 1; else hi = mid;
        }
        const uint32_t pos = (by_count ? rank_new(k) : j) + lo;
        if (pos < L) {
          dst[pos] = k;
          atomicMin(&s.first_new, pos);
        } else {
          const uint32_t o = atomicAdd(&s.spill_n, 1u);
          if (o < cfg.spill_cap) spill[o] = k;
          atomicMin(&s.spill_min, k);
        }
      }
      __syncthreads();
      cur ^= 1u;
      n = min(n + kept, L);
    }
    // ---- exact re-rank of the best entries with the full-precision rows --------------------
    {
      const unsigned long long* list = lists + (size_t)cur * L;
      const uint32_t R = min(n, max(P.size, (uint32_t)((P.size * cfg.rerank_x16 + 15) / 16)));
      const int pw = packed_width(NG);
      const uint32_t gpb = (uint32_t)T / (uint32_t)pw;
      for (uint32_t b = 0; b < R; b += gpb) {
        const uint32_t i = b + (uint32_t)(tid / pw);
        const uint32_t id[1] = {i < R ? key_rawid(list[i]) : 0u};
        Acc<OT, M> sum[1];
        packed_sums<OT, M, 1>(qn, g.objects, id, (int)rc, lane & (pw - 1), NG, sum);
        if (i < R && (lane & (pw - 1)) == 0) nkey[i] = pack_key(sum[0].finish(), id[0]);
      }
      __syncthreads();
      cta_bitonic_sort(nkey, R, NB);
      if (warp == 0) {
        uint32_t nout = 0;
        for (uint32_t b = 0; b < R && nout < P.size_out; b += 32) {
          uint32_t i = b + lane;
          bool ok = i < R && key_dist(nkey[i]) <= user_radius;
          unsigned bal = __ballot_sync(0xffffffffu, ok);
          uint32_t pos = nout + __popc(bal & ((1u << lane) - 1u));
          if (ok && pos < P.size_out) out[P.out_off + pos] = ObjDist{key_id(nkey[i]), key_dist(nkey[i])};
          nout = min(P.size_out, nout + __popc(bal));
        }
        if (lane == 0) {
          out_count[q] = nout;
          stats[q] = QueryStats{s.dc, s.expansions, s.dc, s.edges, s.status};
        }
      }
    }
    if (!cfg.smem_bitmap) {
      uint4* bm4 = reinterpret_cast<uint4*>(bitmap);
      for (uint32_t i = tid; i < cfg.bitmap_words / 4; i += blockDim.x) store_zero16(bm4 + i, keep_visited, pol_keep);
    }
    __syncthreads();
  }
}

}  // namespace ngtg
