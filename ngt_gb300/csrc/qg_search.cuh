// Quantized-graph search (NGTQG): one query per CTA, reproducing
// NGTQG::Index::searchQuantizedGraph (lib/NGT/NGTQ/QuantizedGraph.h:283-447)
// step for step, so that results equal the reference's.
//
// Per query:
//   1. the query is rotated (Rotation::mul, lib/NGT/NGTQ/Quantizer.h:117-160)
//      and its uint8 distance table built (createFloatL2DistanceLookup,
//      lib/NGT/NGTQ/Quantizer.h:1731-1810): squared L2 of each subvector to each
//      of the 16 local centroids, one global offset (the minimum) and scale
//      ((max - min) / 255), entries rounded to nearest even.  The rotation sums
//      in the order of the x86-64 OpenBLAS sgemv the reference links (one FMA
//      chain for dimensions <= 48, else blocks of 8 columns).
//   2. seeds come from the DVP tree (getSeedsFromTree, thinned to the requested
//      size) with exact L2 distances, as setupDistances(L2Float) / setupSeeds do.
//   3. best-first loop: each expanded node's neighbours are scored by the 4-bit
//      scan of its code stream (lib/NGT/NGTQ/Quantizer.h:2331-2440): every lane
//      keeps the 16-entry tables of ceil(m/32) subspaces in registers and looks
//      up four neighbours per byte_perm pair, the per-lane sums of 16 neighbours
//      are reduce-scattered over the warp; distance = sqrt(sum * scale + offset)
//      with the multiply-add fused.
//   4. a neighbour enters the visited set only when it is within the
//      exploration radius, then joins the results (updatable-search semantics:
//      push, pop the maximum when over size, radius = maximum) when within the
//      radius; the result size is size x result expansion.
//   5. with result expansion >= 1 the results are re-ranked by exact L2, cut at
//      the radius (kept when distance < radius) and truncated to the size.
// Order independence inside one expanded node follows the exact graph kernel:
// the radius never grows, so marking visited against the radius at the start
// of a chunk, replaying the result updates in edge order with the reference's
// conditions and pushing candidates against the radius at the end of the chunk
// gives the reference's pop sequence.
#pragma once
#include <cfloat>
#include "graph_exact.cuh"

namespace ngtg {

struct QGShared {
  ExactShared x;                  // the exact kernel's shared state (merge_results, exact_refill)
  uint32_t nkept;
  float lut_min, lut_scale, lut_offset;
  float wmin[kExactWarps], wmax[kExactWarps];
};

// Four table lookups per byte_perm triple: nibble i of w (neighbour i) selects
// entry i of the subspace's 16-byte table held in L[0..3].  Adds the entries of
// neighbours 0,2 / 1,3 of each half-word into a[0] / a[1] (low half-word) and
// a[2] / a[3] (high half-word) as two 16-bit lanes.
__device__ __forceinline__ void qg_lookup8(uint32_t w, const uint32_t (&L)[4], uint32_t* a) {
  const uint32_t sel = ((w >> 1) & 0x44444444u) | 0x32103210u;   // bit 3 of a code picks the upper 8 entries
  uint32_t v = __byte_perm(__byte_perm(L[0], L[1], w), __byte_perm(L[2], L[3], w), sel);
  a[0] += __byte_perm(v, 0u, 0x4240u);
  a[1] += __byte_perm(v, 0u, 0x4341u);
  const uint32_t wh = w >> 16, selh = sel >> 16;
  v = __byte_perm(__byte_perm(L[0], L[1], wh), __byte_perm(L[2], L[3], wh), selh);
  a[2] += __byte_perm(v, 0u, 0x4240u);
  a[3] += __byte_perm(v, 0u, 0x4341u);
}

// The code words of one 16-neighbour block this lane reads (subspaces lane + 32j).
template <int SPL>
__device__ __forceinline__ void qg_block_words(const uint8_t* __restrict__ blk, uint32_t ma, int lane,
                                               uint2 (&w)[SPL]) {
#pragma unroll
  for (int j = 0; j < SPL; j++) {
    const uint32_t s = (uint32_t)lane + 32u * (uint32_t)j;
    w[j] = s < ma ? *reinterpret_cast<const uint2*>(blk + 8u * s) : make_uint2(0u, 0u);
  }
}

// The neighbour (0..15) of a block whose distance qg_block_distance_words returns in
// `lane`, or -1.
__device__ __forceinline__ int qg_lane_object(uint32_t m, int lane) {
  if (m > 256) return (lane & 1) ? -1 : ((lane >> 1) & 15);
  const int g = ((lane >> 3) & 1) | (((lane >> 4) & 1) << 1), par = (lane >> 2) & 1, sub = lane & 3;
  return sub == 0 ? 4 * g + par : sub == 1 ? 4 * g + 2 + par : -1;
}

// Quantized distances of the 16 neighbours of one code block, by one warp, from the
// words qg_block_words loaded.  Returns, in lanes whose bits 1..0 select it, one
// neighbour's distance: *obj receives the neighbour (0..15) the lane holds, or -1.
template <int SPL>
__device__ __forceinline__ float qg_block_distance_words(const uint2 (&w)[SPL], const uint32_t (&L)[SPL][4],
                                                         uint32_t m, float scale, float offset, int lane, int* obj) {
  uint32_t acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
  for (int j = 0; j < SPL; j++) {
    qg_lookup8(w[j].x, L[j], acc);
    qg_lookup8(w[j].y, L[j], acc + 4);
  }
  uint32_t sum;
  int o;
  if (m <= 256) {
    // every 16-bit lane stays below 65536: reduce-scatter the packed pairs
    // (register r = 2*group + parity holds neighbours 4g+p and 4g+2+p)
    uint32_t r4[4], r2[2];
    {
      const bool b = (lane & 16) != 0;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        uint32_t send = b ? acc[i] : acc[i + 4], keep = b ? acc[i + 4] : acc[i];
        r4[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
      }
    }
    {
      const bool b = (lane & 8) != 0;
#pragma unroll
      for (int i = 0; i < 2; i++) {
        uint32_t send = b ? r4[i] : r4[i + 2], keep = b ? r4[i + 2] : r4[i];
        r2[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
      }
    }
    const bool b4 = (lane & 4) != 0;
    uint32_t r1 = (b4 ? r2[1] : r2[0]) + __shfl_xor_sync(0xffffffffu, b4 ? r2[0] : r2[1], 4);
    r1 += __shfl_xor_sync(0xffffffffu, r1, 2);
    r1 += __shfl_xor_sync(0xffffffffu, r1, 1);
    const int r = ((lane >> 2) & 1) | (((lane >> 3) & 1) << 1) | (((lane >> 4) & 1) << 2);
    const int g = r >> 1, par = r & 1;
    const int sub = lane & 3;
    o = sub == 0 ? 4 * g + par : sub == 1 ? 4 * g + 2 + par : -1;
    sum = sub == 0 ? (r1 & 0xFFFFu) : (r1 >> 16);
  } else {
    // wide sums: per-neighbour 32-bit values; even and odd subspaces (lane
    // parity) saturate separately at 65535 like the reference's 16-bit lanes
    uint32_t u[16];
#pragma unroll
    for (int g = 0; g < 4; g++) {
      u[4 * g + 0] = acc[2 * g] & 0xFFFFu;
      u[4 * g + 2] = acc[2 * g] >> 16;
      u[4 * g + 1] = acc[2 * g + 1] & 0xFFFFu;
      u[4 * g + 3] = acc[2 * g + 1] >> 16;
    }
    uint32_t r8[8], r4[4], r2[2];
    {
      const bool b = (lane & 16) != 0;
#pragma unroll
      for (int i = 0; i < 8; i++) {
        uint32_t send = b ? u[i] : u[i + 8], keep = b ? u[i + 8] : u[i];
        r8[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
      }
    }
    {
      const bool b = (lane & 8) != 0;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        uint32_t send = b ? r8[i] : r8[i + 4], keep = b ? r8[i + 4] : r8[i];
        r4[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
      }
    }
    {
      const bool b = (lane & 4) != 0;
#pragma unroll
      for (int i = 0; i < 2; i++) {
        uint32_t send = b ? r4[i] : r4[i + 2], keep = b ? r4[i + 2] : r4[i];
        r2[i] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
      }
    }
    const bool b2 = (lane & 2) != 0;
    uint32_t r1 = (b2 ? r2[1] : r2[0]) + __shfl_xor_sync(0xffffffffu, b2 ? r2[0] : r2[1], 2);
    r1 = min(r1, 65535u);
    sum = r1 + __shfl_xor_sync(0xffffffffu, r1, 1);
    o = (lane & 1) ? -1 : ((lane >> 1) & 15);
  }
  *obj = o;
  return __fsqrt_rn(__fmaf_rn(__uint2float_rn(sum), scale, offset));
}

// Quantized distances of the 16 neighbours of one code block, by one warp.
template <int SPL>
__device__ __forceinline__ float qg_block_distance(const uint8_t* __restrict__ blk, const uint32_t (&L)[SPL][4],
                                                   uint32_t m, uint32_t ma, float scale, float offset, int lane,
                                                   int* obj) {
  uint2 w[SPL];
  qg_block_words<SPL>(blk, ma, lane, w);
  return qg_block_distance_words<SPL>(w, L, m, scale, offset, lane, obj);
}

// Shared memory of the float table, later reused by the lists and the visited hash.
inline size_t qg_table_bytes(uint32_t m, const ExactConfig& c) {
  const size_t lists = (size_t)c.ccap * 16 + (size_t)kExactChunk * 16 + (size_t)c.hcap * 4;
  const size_t table = (size_t)m * 16 * 4;
  return ((lists > table ? lists : table) + 15) / 16 * 16;
}
inline size_t qg_smem_bytes(uint32_t row_chunks, uint32_t dim, uint32_t m, const ExactConfig& c) {
  size_t b = (size_t)row_chunks * 16;
  b += ((size_t)dim * 4 + 15) / 16 * 16;                 // rotated query
  b += ((size_t)m * 16 + 15) / 16 * 16;                  // uint8 table
  b += ((size_t)c.kcap + 1) / 2 * 16;                    // results
  b += qg_table_bytes(m, c);
  b += (size_t)kExactChunk * 8;                          // a round's distances and ids
  b += sizeof(QGShared) + 16;
  return b;
}

// Bound by latency and instruction issue like the exact graph kernel, whose round it
// shares: the guessed next node's ids and code lines load beside the current node's
// codes, each lane that holds a distance checks and records its neighbour at once (one
// barrier per round without survivors, twelve before), result updates are merged
// (merge_results), the shared list holds 256 keys and the float table lies under the
// lists, so that six CTAs fit an SM instead of three on indexes below 262,144 objects.
// A visited set holds only neighbours within the exploration radius (hundreds), so a small
// hash serves every index.  200k x 128, 128 subspaces, 2,000 queries from host buffers
// (k = 20, epsilon 0.03, expansion 3): 2.87 -> 1.46 ms.
template <int SPL>
__global__ void __launch_bounds__(kExactThreads, SPL <= 4 ? 6 : 2)
qg_search_kernel(DevGraph g, DevQG qg, const uint4* __restrict__ queries, uint32_t nq,
                 const QGParams* __restrict__ params, const uint32_t* __restrict__ seed_list,
                 ObjDist* __restrict__ out, uint32_t* __restrict__ out_count, QueryStats* __restrict__ stats,
                 uint32_t* __restrict__ bitmaps, unsigned long long* __restrict__ overflow, ExactConfig cfg) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t rc = g.row_chunks;
  const uint32_t D = qg.dim, M = qg.m, LD = qg.ld;
  // ---- shared-memory carve-up -------------------------------------------
  uint4* qv = reinterpret_cast<uint4*>(smem);
  float* rq = reinterpret_cast<float*>(qv + rc);
  uint8_t* lut = reinterpret_cast<uint8_t*>(rq + (D + 3) / 4 * 4);
  unsigned long long* res = reinterpret_cast<unsigned long long*>(lut + ((size_t)M * 16 + 15) / 16 * 16);
  unsigned long long* cand0 = res + (cfg.kcap + 1) / 2 * 2;
  unsigned long long* cand1 = cand0 + cfg.ccap;
  unsigned long long* bkeys = cand1 + cfg.ccap;
  unsigned long long* bsorted = bkeys + kExactChunk;
  uint32_t* table = reinterpret_cast<uint32_t*>(bsorted + kExactChunk);
  float* flut = reinterpret_cast<float*>(cand0);     // while the tables are built
  uint32_t* nid = reinterpret_cast<uint32_t*>(reinterpret_cast<unsigned char*>(cand0) + cfg.table_bytes);
  float* nd = reinterpret_cast<float*>(nid + kExactChunk);
  QGShared& qs = *reinterpret_cast<QGShared*>(nd + kExactChunk);
  ExactShared& s = qs.x;
  uint32_t* bitmap = bitmaps + (size_t)blockIdx.x * cfg.bitmap_words;
  unsigned long long* ovf = overflow + (size_t)blockIdx.x * 2 * cfg.ocap;
  unsigned long long* ovf_tmp = ovf + cfg.ocap;
  const uint32_t hmask = cfg.hcap - 1;
  const int G = (int)cfg.group;
  const int gl = lane & (G - 1);
  const int ngroups = kExactThreads / G;
  const float* qf = reinterpret_cast<const float*>(qv);
  const uint32_t qlen = rc * 4;                      // floats in the padded query row

  for (uint32_t q = exact_next_query(0xffffffffu, cfg.work, &s.query); q < nq;
       q = exact_next_query(q, cfg.work, &s.query)) {
    const QGParams P = params[q];
    for (uint32_t i = tid; i < rc; i += blockDim.x) qv[i] = queries[(size_t)q * rc + i];
    if (tid == 0) {
      s.seed_status = 0;
      s.keep[0] = s.keep[1] = s.keep[2] = 0;
    }
    __syncthreads();
    if (P.size == 0 || P.k == 0) {
      if (tid == 0) { out_count[q] = 0; stats[q] = QueryStats{0, 0, 0, 0, 0}; }
      __syncthreads();
      continue;
    }
    // ---- rotation and distance table ---------------------------------------
    for (uint32_t c = tid; c < D; c += blockDim.x) {
      float acc = 0.f;
      if (qg.rotation == nullptr) {
        acc = c < qlen ? qf[c] : 0.f;
      } else if (D <= 48) {
        for (uint32_t p = 0; p < D; p++)
          acc = __fmaf_rn(qg.rotation[(size_t)p * D + c], p < qlen ? qf[p] : 0.f, acc);
      } else {
        for (uint32_t p0 = 0; p0 < D; p0 += 8) {
          const uint32_t p1 = min(p0 + 8u, D);
          float t = __fmul_rn(qg.rotation[(size_t)p0 * D + c], p0 < qlen ? qf[p0] : 0.f);
          for (uint32_t p = p0 + 1; p < p1; p++)
            t = __fmaf_rn(qg.rotation[(size_t)p * D + c], p < qlen ? qf[p] : 0.f, t);
          acc = __fadd_rn(acc, t);
        }
      }
      rq[c] = acc;
    }
    __syncthreads();
    {
      float lmin = FLT_MAX, lmax = -FLT_MAX;
      for (uint32_t e = tid; e < M * 16; e += blockDim.x) {
        const uint32_t sv = e >> 4, c = e & 15u;
        float v = 0.f;
        for (uint32_t d = 0; d < LD; d++) {
          const float rsv = __fsub_rn(rq[sv * LD + d], qg.gcentroid[sv * LD + d]);
          const float sub = __fsub_rn(rsv, qg.lcentroids[((size_t)sv * 16 + c) * LD + d]);
          v = d == 0 ? __fmul_rn(sub, sub) : __fmaf_rn(sub, sub, v);
        }
        flut[e] = v;
        lmin = fminf(lmin, v);
        lmax = fmaxf(lmax, v);
      }
      for (int off = 16; off > 0; off >>= 1) {
        lmin = fminf(lmin, __shfl_xor_sync(0xffffffffu, lmin, off));
        lmax = fmaxf(lmax, __shfl_xor_sync(0xffffffffu, lmax, off));
      }
      if (lane == 0) { qs.wmin[warp] = lmin; qs.wmax[warp] = lmax; }
      __syncthreads();
      if (tid == 0) {
        float mn = qs.wmin[0], mx = qs.wmax[0];
        for (int w = 1; w < kExactWarps; w++) { mn = fminf(mn, qs.wmin[w]); mx = fmaxf(mx, qs.wmax[w]); }
        qs.lut_min = mn;
        qs.lut_scale = __double2float_rn(__ddiv_rn((double)__fsub_rn(mx, mn), 255.0));
        qs.lut_offset = __fmul_rn(mn, (float)M);
      }
      __syncthreads();
      const float mn = qs.lut_min, scale = qs.lut_scale;
      for (uint32_t e = tid; e < M * 16; e += blockDim.x)
        lut[e] = (uint8_t)(int)rintf(__fdiv_rn(__fsub_rn(flut[e], mn), scale));
      __syncthreads();
      for (uint32_t i = tid; i < cfg.hcap; i += blockDim.x) table[i] = 0u;   // the float table is done with
    }
    uint32_t L[SPL][4];
#pragma unroll
    for (int j = 0; j < SPL; j++) {
      const uint32_t sv = (uint32_t)lane + 32u * (uint32_t)j;
      const uint4 t = sv < M ? reinterpret_cast<const uint4*>(lut)[sv] : make_uint4(0, 0, 0, 0);
      L[j][0] = t.x; L[j][1] = t.y; L[j][2] = t.z; L[j][3] = t.w;
    }
    const float lscale = qs.lut_scale, loffset = qs.lut_offset;
    // ---- seeds --------------------------------------------------------------
    const uint32_t* seeds = nullptr;
    uint32_t nseeds = 0;
    if (P.seed_cnt == 0xffffffffu) {
      if (warp == 0) {
        uint32_t node = g.root;
        int depth = 0;
        while (!(node & 0x80000000u) && depth < 64) {
          const DevInternal& in = g.internals[node];
          float d = group_distance<ObjType::Float, Metric::L2>(qv, g.pivots + (size_t)in.pivot * rc, (int)rc, lane,
                                                               32);
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
        const uint32_t* off = g.leaf_seed_off + P.seed_off;
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
    for (uint32_t b = (uint32_t)(warp * (32 / G)); b < nseeds; b += ngroups) {
      uint32_t i = b + (uint32_t)(lane / G);
      bool valid = i < nseeds;
      uint32_t id = valid ? seeds[i] : 0u;
      bool inrange = id < g.nrows;
      float d = group_distance<ObjType::Float, Metric::L2>(qv, g.objects + (size_t)(inrange ? id : 0u) * rc,
                                                           (int)rc, gl, G);
      if (valid && gl == 0) bkeys[i] = pack_key(inrange ? d : FLT_MAX, id);
    }
    __syncthreads();
    rank_sort(bkeys, bsorted, nseeds);
    __syncthreads();
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
    for (uint32_t i = tid; i < nseeds; i += blockDim.x) {
      cand0[i] = bsorted[i];
      visit_insert(table, hmask, bitmap, false, key_id(bsorted[i]));
    }
    __syncthreads();

    // ---- best-first loop -----------------------------------------------------
    // Alike in every thread, as in the exact graph kernel.
    uint32_t head = 0, tail = nseeds, cur = 0, ovf_n = 0;
    unsigned long long ovf_min = ~0ull;
    uint32_t nvisited = nseeds, dc = nseeds, expansions = 0, edges = 0;
    bool spilled = false, have = false;
    float radius = s.radius;
    uint32_t e0 = 0, deg = 0, code0 = 0;          // the node to expand: its ids, its codes
    uint32_t guard = 0, turn = 0;
    auto node = [&](uint32_t id, uint32_t& first, uint32_t& count, uint32_t& code) {
      const bool has = id < qg.nnodes;            // nodes beyond the quantized graph have no edges
      first = has ? __ldg(qg.offsets + id) : 0u;
      count = has ? __ldg(qg.offsets + id + 1) - first : 0u;
      code = has ? __ldg(qg.code_off16 + id) : 0u;
    };
    while (true) {
      if (!have) {
        if (head >= tail && ovf_n > 0) {
          head = 0;
          tail = exact_refill<kExactThreads>(cur ? cand1 : cand0, cfg.ccap, ovf, ovf_tmp, ovf_n, ovf_min,
                                             __fmul_rn(P.coef, radius), s);
        }
        if (head >= tail) break;
        const unsigned long long t = (cur ? cand1 : cand0)[head];
        if (key_dist(t) > __fmul_rn(P.coef, radius)) break;
        head++;
        node(key_id(t), e0, deg, code0);
      }
      have = false;
      const unsigned long long guess = head < tail ? (cur ? cand1 : cand0)[head] : ~0ull;
      uint32_t ge0 = 0, gdeg = 0, gcode = 0;
      if (head < tail) node(key_id(guess), ge0, gdeg, gcode);
      if (guard++ > g.nrows + 8) {
        status |= kStatusIterationLimit;
        break;
      }
      expansions++;
      edges += deg;
      dc += deg;
      bool finished = false;
      const uint32_t n_edges = deg;
      const uint8_t* stream = qg.codes + (size_t)code0 * 16;
      for (uint32_t c0 = 0; c0 < n_edges; c0 += kExactChunk) {
        const uint32_t clen = min((uint32_t)kExactChunk, n_edges - c0);
        const bool last = c0 + kExactChunk >= n_edges;
        if (!spilled && nvisited + clen > (cfg.hcap >> 1)) {
          for (uint32_t i = tid; i < cfg.hcap; i += blockDim.x) {
            uint32_t id = table[i];
            if (id) atomicOr(&bitmap[id >> 5], 1u << (id & 31u));
          }
          __threadfence_block();
          __syncthreads();
          spilled = true;
          status |= kStatusVisitedSpill;
        }
        // quantized distances of the chunk, a 16-neighbour block per warp at a time; within
        // the exploration radius and not visited yet: new
        const float expR0 = __fmul_rn(P.coef, radius);
        const uint32_t nblk = (clen + 15) / 16;
        const int o = qg_lane_object(M, lane);
        bool pass = false;
        for (uint32_t bi = (uint32_t)warp; bi < nblk; bi += kExactWarps) {
          uint2 w[SPL];
          qg_block_words<SPL>(stream + (size_t)(c0 / 16 + bi) * 8 * qg.ma, qg.ma, lane, w);
          const uint32_t pos = bi * 16 + (uint32_t)o;
          const bool mine = o >= 0 && pos < clen;
          const uint32_t id = mine ? __ldg(qg.ids + e0 + c0 + pos) : 0u;
          if (last && bi == (uint32_t)warp) {
            // the guess's code lines (and ids) are asked for beside this node's
            const uint32_t bytes = (gdeg + 15) / 16 * 8 * qg.ma;
            if ((uint32_t)tid * 128u < bytes)
              asm volatile("prefetch.global.L2 [%0];" ::"l"(qg.codes + (size_t)gcode * 16 + (uint32_t)tid * 128u));
            if ((uint32_t)tid * 32u < gdeg) asm volatile("prefetch.global.L2 [%0];" ::"l"(qg.ids + ge0 + tid * 32));
          }
          int oo;
          const float d = qg_block_distance_words<SPL>(w, L, M, lscale, loffset, lane, &oo);
          if (mine) {
            const bool isnew = d <= expR0 && visit_insert(table, hmask, bitmap, spilled, id);
            if (isnew) {
              bkeys[atomicAdd(&s.keep[turn], 1u)] = pack_key(d, id);
              pass = pass || d <= radius;
            }
            if (!(P.coef >= 1.0f)) {               // the replay below goes through them in edge order
              nd[pos] = isnew ? d : INFINITY;
              nid[pos] = id;
            }
          }
        }
        const bool replay = __syncthreads_or(pass ? 1 : 0) != 0;
        uint32_t m = s.keep[turn];
        // one barrier a round: the counter cleared is the one last read a round ago, and first
        // used again after the next barrier
        if (tid == 0) s.keep[turn == 0 ? 2 : turn - 1] = 0;
        turn = turn == 2 ? 0 : turn + 1;
        nvisited += m;
        // result-set updates: a neighbour joins when within both the exploration radius and
        // the radius of that moment
        if (replay) {
          rank_sort_split<kExactThreads>(bkeys, bsorted, m);
          __syncthreads();
          if (!(P.coef >= 1.0f) || !merge_results<kExactThreads>(res, P.size, (uint32_t)GraphMode::Updatable, radius,
                                                                 bsorted, m, nullptr, nullptr, 0, s)) {
            if (warp == 0) {
              float rad = radius;
              uint32_t n = s.nres;
              for (uint32_t b = 0; b < clen; b += 32) {
                uint32_t i = b + lane;
                float d = i < clen ? nd[i] : INFINITY;
                float lim = fminf(rad, __fmul_rn(P.coef, rad));
                unsigned m = __ballot_sync(0xffffffffu, i < clen && d <= lim);
                while (m) {
                  int src = __ffs(m) - 1;
                  float dj = __shfl_sync(0xffffffffu, d, src);
                  uint32_t idj = nid[b + src];
                  if (dj <= rad && dj <= __fmul_rn(P.coef, rad))
                    result_insert(res, n, rad, P.size, (uint32_t)GraphMode::Updatable, pack_key(dj, idj), lane);
                  m &= (src == 31) ? 0u : ~((2u << src) - 1u);
                  lim = fminf(rad, __fmul_rn(P.coef, rad));
                  m &= __ballot_sync(0xffffffffu, i < clen && d <= lim);
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
        const float expR = __fmul_rn(P.coef, radius);
        unsigned long long* cl = cur ? cand1 : cand0;
        if (m == 0) {
          // no candidate came: the list stays, and its head is the guess unless an earlier
          // round of this node brought a nearer one (which is popped at the top then)
          if (last && head < tail && cl[head] == guess) {
            have = !(key_dist(guess) > expR);
            finished = !have;
            if (have) {
              head++;
              e0 = ge0;
              deg = gdeg;
              code0 = gcode;
            }
          }
          continue;
        }
        if (tid == 0) s.evict_min = ~0ull;
        unsigned long long* cn = cur ? cand0 : cand1;
        const unsigned long long* old = cl + head;
        if (!replay) rank_sort_split<kExactThreads>(bkeys, bsorted, m);
        if (replay && tid == kExactThreads - 1) s.live_old = upper_bound_dist(old, tail - head, expR);
        __syncthreads();
        uint32_t nold = tail - head;
        if (replay) {
          nold = s.live_old;
          m = upper_bound_dist(bsorted, m, expR);
        }
        const uint32_t mk = ovf_n && m && bsorted[m - 1] >= ovf_min ? lower_bound_keys(bsorted, m, ovf_min) : m;
        if (last) {
          unsigned long long t = nold ? old[0] : ~0ull;
          if (mk && bsorted[0] < t) t = bsorted[0];
          if (nold + mk > 0) {
            have = !(key_dist(t) > expR);
            finished = !have;
          }
          if (have) {
            if (t == guess) {
              e0 = ge0;
              deg = gdeg;
              code0 = gcode;
            } else {
              node(key_id(t), e0, deg, code0);     // under way while the list is merged
            }
          }
        }
        const uint32_t obase = ovf_n;
        const uint32_t nevict = (nold + mk > cfg.ccap) ? nold + mk - cfg.ccap : 0u;
        for (uint32_t i = tid; i < m - mk; i += blockDim.x) {
          uint32_t o = obase + i;
          if (o < cfg.ocap) ovf[o] = bsorted[mk + i];
        }
        for (uint32_t i = tid; i < nold; i += blockDim.x) {
          unsigned long long k = old[i];
          uint32_t pos = i + lower_bound_keys(bsorted, mk, k);
          if (pos < cfg.ccap) cn[pos] = k;
          else {
            uint32_t o = obase + (m - mk) + (pos - cfg.ccap);
            if (o < cfg.ocap) ovf[o] = k;
            if (pos == cfg.ccap) s.evict_min = k;
          }
        }
        for (uint32_t i = tid; i < mk; i += blockDim.x) {
          unsigned long long k = bsorted[i];
          uint32_t pos = i + lower_bound_keys(old, nold, k);
          if (pos < cfg.ccap) cn[pos] = k;
          else {
            uint32_t o = obase + (m - mk) + (pos - cfg.ccap);
            if (o < cfg.ocap) ovf[o] = k;
            if (pos == cfg.ccap) s.evict_min = k;
          }
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
    uint32_t n = s.nres;
    if (P.rerank) {
      // exact L2 of every result, sorted by (distance, id); kept while distance <
      // radius (upper_bound at (0, radius)); at most k
      const int pw = packed_width(G);
      for (uint32_t b = (uint32_t)(warp * (32 / pw)); b < n; b += 2 * (kExactThreads / pw)) {
        uint32_t id[2], at[2];
        Acc<ObjType::Float, Metric::L2> sum[2];
#pragma unroll
        for (int u = 0; u < 2; u++) {
          at[u] = b + u * (kExactThreads / pw) + (uint32_t)(lane / pw);
          id[u] = at[u] < n ? key_id(res[at[u]]) : 0u;
        }
        packed_sums<ObjType::Float, Metric::L2, 2>(qv, g.objects, id, (int)rc, lane & (pw - 1), G, sum);
#pragma unroll
        for (int u = 0; u < 2; u++)
          if (at[u] < n && (lane & (pw - 1)) == 0) cand0[at[u]] = pack_key(sum[u].finish(), id[u]);
      }
      __syncthreads();
      bitonic_sort(cand0, n, cfg.ccap);
      if (tid == 0) {
        uint32_t keep = n;
        if (P.radius < FLT_MAX) {
          keep = 0;
          while (keep < n && key_dist(cand0[keep]) < P.radius) keep++;
        }
        qs.nkept = min(keep, P.k);
      }
      __syncthreads();
      n = qs.nkept;
      for (uint32_t i = tid; i < n; i += blockDim.x) {
        unsigned long long k = cand0[i];
        out[P.out_off + i] = ObjDist{key_id(k), key_dist(k)};
      }
    } else {
      for (uint32_t i = tid; i < n; i += blockDim.x) {
        unsigned long long k = res[i];
        out[P.out_off + i] = ObjDist{key_id(k), key_dist(k)};
      }
    }
    if (tid == 0) {
      out_count[q] = n;
      stats[q] = QueryStats{dc, expansions, nvisited, edges, status};
    }
    if (spilled) {
      for (uint32_t i = tid; i < cfg.bitmap_words; i += blockDim.x) bitmap[i] = 0u;
      __threadfence();
    }
    __syncthreads();
  }
}

}  // namespace ngtg
