// Quantized-blob-graph search (QBG): one query per CTA, reproducing
// QBG::Index::searchInOneStep (lib/NGT/NGTQ/QuantizedBlobGraph.h:1332-1594) as
// the C API (qbg_search_index_, lib/NGT/NGTQ/Capi.cpp:549-574) drives it, so
// that results equal the reference's.
//
// The index has a global NGT index over the blob centroids (graph + DVP tree)
// and, per blob (= global node), the 4-bit codes of its objects quantized
// against the rotated codebook centroid of the blob's subspace id.
//   1. seeds: the global tree's leaf (thinned to the result size) with exact L2
//      distances; the nearest is the current blob, the others are "discarded"
//      (waiting) blobs; all are untraced graph nodes.
//   2. while the nearest untraced node is within blob_coef x d(current blob),
//      it is expanded: its unvisited neighbours get exact L2 distances, become
//      untraced, and either replace the current blob (strictly nearer; the first
//      such neighbour in edge order) or wait.
//   3. otherwise the current blob is judged (QuantizedBlobGraph.h:1033-1080):
//      its LUT is built for the blob's subspace id (the rotated query minus that
//      centroid, as in the QG table) and its objects scanned; when the scan's
//      minimum is below the radius every object within the radius joins the
//      result set (kept to its size, radius = its maximum when full).  The search
//      stops when the minimum exceeds radius x (1 + epsilon), after
//      number_of_explored_blobs judgements, or when no blob waits; else the
//      nearest waiting blob becomes current.
// Results carry the quantized distances, number_of_results x result_expansion
// of them when the expansion is >= 1 (the C API never sets refinement).
// Both queues are exact two-tier min-queues (tier_queue.cuh).
#pragma once
#include <cfloat>
#include "qg_search.cuh"
#include "tier_queue.cuh"

namespace ngtg {

struct QBGShared {
  float radius, expR;
  uint32_t nres, rcur;
  unsigned long long current;       // (distance, id) of the current blob
  uint32_t done;
  uint32_t exploration;
  uint32_t nblobs, expansions, dc, status;
  uint32_t seed_leaf;
  uint32_t nnew, nacc;
  uint32_t lut_sid;
  float lut_min, lut_scale, lut_offset;
  float bmin;
  float wmin[kExactWarps], wmax[kExactWarps];
  uint32_t warp_cnt[kExactWarps];
  QueueState uq, dq;
  uint32_t hist[256];
};

struct QBGConfig {
  uint32_t rcap;          // result capacity (>= the largest result size), power of two
  uint32_t qcap;          // shared entries per queue (power of two)
  uint32_t ocap;          // overflow keys per queue and buffer
  uint32_t bitmap_words;  // visited bitmap words per CTA (global nodes)
  uint32_t blob_cap;      // distance scratch per CTA (largest blob, rounded up to 16)
  uint32_t group;         // lanes per exact distance (power of two <= 32)
};

inline size_t qbg_smem_bytes(uint32_t row_chunks, uint32_t dim, uint32_t m, const QBGConfig& c) {
  size_t b = (size_t)row_chunks * 16;
  b += ((size_t)dim * 4 + 15) / 16 * 16;
  b += (size_t)m * 16 * 4;
  b += ((size_t)m * 16 + 15) / 16 * 16;
  b += (size_t)c.rcap * 16;                            // results, double-buffered
  b += (size_t)c.qcap * 32;                            // two queues x two buffers
  b += (size_t)kExactChunk * 8 * 3;                    // keys, sorted keys, queue batch
  b += (size_t)kExactChunk * 8;                        // nid + nd
  b += sizeof(QBGShared) + 16;
  return b;
}

// Builds the uint8 LUT of the rotated query against codebook centroid `gc`
// (same arithmetic as the QG table) into lut[] and the scale / offset in s.
__device__ __forceinline__ void qbg_build_lut(const float* rq, const float* __restrict__ gc,
                                              const float* __restrict__ lc, float* flut, uint8_t* lut, uint32_t M,
                                              uint32_t LD, QBGShared& s) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float lmin = FLT_MAX, lmax = -FLT_MAX;
  for (uint32_t e = tid; e < M * 16; e += blockDim.x) {
    const uint32_t sv = e >> 4, c = e & 15u;
    float v = 0.f;
    for (uint32_t d = 0; d < LD; d++) {
      const float rsv = __fsub_rn(rq[sv * LD + d], gc[sv * LD + d]);
      const float sub = __fsub_rn(rsv, lc[((size_t)sv * 16 + c) * LD + d]);
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
  if (lane == 0) { s.wmin[warp] = lmin; s.wmax[warp] = lmax; }
  __syncthreads();
  if (tid == 0) {
    float mn = s.wmin[0], mx = s.wmax[0];
    for (int w = 1; w < kExactWarps; w++) { mn = fminf(mn, s.wmin[w]); mx = fmaxf(mx, s.wmax[w]); }
    s.lut_min = mn;
    s.lut_scale = __double2float_rn(__ddiv_rn((double)__fsub_rn(mx, mn), 255.0));
    s.lut_offset = __fmul_rn(mn, (float)M);
  }
  __syncthreads();
  const float mn = s.lut_min, scale = s.lut_scale;
  for (uint32_t e = tid; e < M * 16; e += blockDim.x)
    lut[e] = (uint8_t)(int)rintf(__fdiv_rn(__fsub_rn(flut[e], mn), scale));
  __syncthreads();
}

// Merges m sorted keys into the sorted result set (double-buffered), keeping the
// `size` smallest.
__device__ __forceinline__ void qbg_merge_results(unsigned long long* const* resb, QBGShared& s,
                                                  const unsigned long long* keys, uint32_t m, uint32_t size) {
  const uint32_t tid = threadIdx.x;
  const unsigned long long* old = resb[s.rcur];
  unsigned long long* dst = resb[s.rcur ^ 1u];
  const uint32_t nold = s.nres;
  for (uint32_t i = tid; i < nold; i += blockDim.x) {
    uint32_t pos = i + lower_bound_keys(keys, m, old[i]);
    if (pos < size) dst[pos] = old[i];
  }
  for (uint32_t i = tid; i < m; i += blockDim.x) {
    uint32_t pos = i + lower_bound_keys(old, nold, keys[i]);
    if (pos < size) dst[pos] = keys[i];
  }
  __syncthreads();
  if (tid == 0) {
    s.nres = min(nold + m, size);
    s.rcur ^= 1u;
  }
  __syncthreads();
}

// Rotation::mul of the query (the OpenBLAS sgemv order: one FMA chain for D <= 48,
// else blocks of 8 columns), the query zero-padded to D.
__device__ __forceinline__ void qbg_rotate(const DevQG& qb, const float* qf, uint32_t qlen, float* rq) {
  const uint32_t D = qb.dim;
  for (uint32_t c = threadIdx.x; c < D; c += blockDim.x) {
    float acc = 0.f;
    if (qb.rotation == nullptr) {
      acc = c < qlen ? qf[c] : 0.f;
    } else if (D <= 48) {
      for (uint32_t p = 0; p < D; p++) acc = __fmaf_rn(qb.rotation[(size_t)p * D + c], p < qlen ? qf[p] : 0.f, acc);
    } else {
      for (uint32_t p0 = 0; p0 < D; p0 += 8) {
        const uint32_t p1 = min(p0 + 8u, D);
        float t = __fmul_rn(qb.rotation[(size_t)p0 * D + c], p0 < qlen ? qf[p0] : 0.f);
        for (uint32_t p = p0 + 1; p < p1; p++) t = __fmaf_rn(qb.rotation[(size_t)p * D + c], p < qlen ? qf[p] : 0.f, t);
        acc = __fadd_rn(acc, t);
      }
    }
    rq[c] = acc;
  }
}

// judge (lib/NGT/NGTQ/QuantizedBlobGraph.h:1033-1080) of one blob by the whole CTA:
// the blob's LUT (rebuilt only when its subspace id differs from the last one),
// the scan of its codes into bdist, its minimum into s.bmin; when that minimum is
// below the radius, every object within the radius joins the result set (kept to
// `size`), and the radius becomes the set's maximum once it is full.
template <int SPL>
__device__ __forceinline__ void qbg_judge_blob(const DevQG& qb, const uint32_t* __restrict__ blob_sid, uint32_t blob,
                                               const float* rq, float* flut, uint8_t* lut, QBGShared& s,
                                               float* bdist, unsigned long long* const* resb,
                                               unsigned long long* bkeys, unsigned long long* bsorted,
                                               uint32_t size) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t M = qb.m, LD = qb.ld, D = qb.dim;
  if (tid == 0) s.bmin = FLT_MAX;
  __syncthreads();
  if (blob >= qb.nnodes) return;
  const uint32_t a = qb.offsets[blob];
  const uint32_t n = qb.offsets[blob + 1] - a;
  const uint32_t sid = blob_sid[blob];
  if (sid != s.lut_sid) {
    qbg_build_lut(rq, qb.gcentroid + (size_t)sid * D, qb.lcentroids, flut, lut, M, LD, s);
    if (tid == 0) s.lut_sid = sid;
  }
  uint32_t L[SPL][4];
#pragma unroll
  for (int j = 0; j < SPL; j++) {
    const uint32_t sv = (uint32_t)lane + 32u * (uint32_t)j;
    const uint4 v = sv < M ? reinterpret_cast<const uint4*>(lut)[sv] : make_uint4(0, 0, 0, 0);
    L[j][0] = v.x; L[j][1] = v.y; L[j][2] = v.z; L[j][3] = v.w;
  }
  const float lscale = s.lut_scale, loffset = s.lut_offset;
  const uint8_t* stream = qb.codes + (size_t)qb.code_off16[blob] * 16;
  const uint32_t nblk = (n + 15) / 16;
  float wmin = FLT_MAX;
  for (uint32_t bi = (uint32_t)warp; bi < nblk; bi += kExactWarps) {
    int o;
    float d = qg_block_distance<SPL>(stream + (size_t)bi * 8 * qb.ma, L, M, qb.ma, lscale, loffset, lane, &o);
    if (o >= 0 && bi * 16 + (uint32_t)o < n) {
      bdist[bi * 16 + o] = d;
      wmin = fminf(wmin, d);
    }
  }
  for (int off = 16; off > 0; off >>= 1) wmin = fminf(wmin, __shfl_xor_sync(0xffffffffu, wmin, off));
  if (lane == 0) s.wmin[warp] = wmin;
  __threadfence_block();
  __syncthreads();
  if (tid == 0) {
    float mn = s.wmin[0];
    for (int w = 1; w < kExactWarps; w++) mn = fminf(mn, s.wmin[w]);
    s.bmin = mn;
    s.nblobs++;
    s.dc += n;
  }
  __syncthreads();
  const float radius0 = s.radius;
  if (s.bmin < radius0) {
    for (uint32_t c0 = 0; c0 < n; c0 += kExactChunk) {
      const uint32_t clen = min((uint32_t)kExactChunk, n - c0);
      bool acc = false;
      float d = 0.f;
      if ((uint32_t)tid < clen) {
        d = bdist[c0 + tid];
        acc = d <= radius0;
      }
      unsigned ballot = __ballot_sync(0xffffffffu, acc);
      if (lane == 0) s.warp_cnt[warp] = __popc(ballot);
      __syncthreads();
      uint32_t base = 0, m = 0;
      for (int w = 0; w < kExactWarps; w++) {
        if (w < warp) base += s.warp_cnt[w];
        m += s.warp_cnt[w];
      }
      if (acc) bkeys[base + __popc(ballot & ((1u << lane) - 1u))] = pack_key(d, qb.ids[a + c0 + tid]);
      __syncthreads();
      rank_sort(bkeys, bsorted, m);
      __syncthreads();
      qbg_merge_results(resb, s, bsorted, m, size);
    }
    if (tid == 0 && s.nres >= size) s.radius = key_dist(resb[s.rcur][s.nres - 1]);
    __syncthreads();
  }
}

template <int SPL>
__global__ void __launch_bounds__(kExactThreads)
qbg_search_kernel(DevGraph g, DevQG qb, const uint32_t* __restrict__ blob_sid, const uint4* __restrict__ queries,
                  uint32_t nq, const QBGParams* __restrict__ params, const uint32_t* __restrict__ seed_list,
                  ObjDist* __restrict__ out, uint32_t* __restrict__ out_count, QueryStats* __restrict__ stats,
                  uint32_t* __restrict__ bitmaps, unsigned long long* __restrict__ overflow,
                  float* __restrict__ blob_dist, QBGConfig cfg) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t rc = g.row_chunks;
  const uint32_t D = qb.dim, M = qb.m, LD = qb.ld;
  uint4* qv = reinterpret_cast<uint4*>(smem);
  float* rq = reinterpret_cast<float*>(qv + rc);
  float* flut = rq + (D + 3) / 4 * 4;
  uint8_t* lut = reinterpret_cast<uint8_t*>(flut + (size_t)M * 16);
  unsigned long long* res0 = reinterpret_cast<unsigned long long*>(lut + ((size_t)M * 16 + 15) / 16 * 16);
  unsigned long long* res1 = res0 + cfg.rcap;
  unsigned long long* uq0 = res1 + cfg.rcap;
  unsigned long long* uq1 = uq0 + cfg.qcap;
  unsigned long long* dq0 = uq1 + cfg.qcap;
  unsigned long long* dq1 = dq0 + cfg.qcap;
  unsigned long long* bkeys = dq1 + cfg.qcap;
  unsigned long long* bsorted = bkeys + kExactChunk;
  unsigned long long* batch = bsorted + kExactChunk;
  uint32_t* nid = reinterpret_cast<uint32_t*>(batch + kExactChunk);
  float* nd = reinterpret_cast<float*>(nid + kExactChunk);
  QBGShared& s = *reinterpret_cast<QBGShared*>(nd + kExactChunk);
  unsigned long long* resb[2] = {res0, res1};
  uint32_t* bitmap = bitmaps + (size_t)blockIdx.x * cfg.bitmap_words;
  unsigned long long* ovf = overflow + (size_t)blockIdx.x * 4 * cfg.ocap;
  float* bdist = blob_dist + (size_t)blockIdx.x * cfg.blob_cap;
  const TierQueue uq{{uq0, uq1}, cfg.qcap, {ovf, ovf + cfg.ocap}, cfg.ocap, &s.uq, s.hist};
  const TierQueue dq{{dq0, dq1}, cfg.qcap, {ovf + 2 * (size_t)cfg.ocap, ovf + 3 * (size_t)cfg.ocap}, cfg.ocap,
                     &s.dq, s.hist};
  const int G = (int)cfg.group;
  const int gl = lane & (G - 1);
  const int ngroups = kExactThreads / G;
  const float* qf = reinterpret_cast<const float*>(qv);
  const uint32_t qlen = rc * 4;

  for (uint32_t q = blockIdx.x; q < nq; q += gridDim.x) {
    const QBGParams P = params[q];
    for (uint32_t i = tid; i < rc; i += blockDim.x) qv[i] = queries[(size_t)q * rc + i];
    if (tid == 0) {
      s.radius = FLT_MAX;
      s.nres = 0; s.rcur = 0; s.done = 0; s.exploration = 1;
      s.nblobs = 0; s.expansions = 0; s.dc = 0; s.status = 0;
      s.lut_sid = 0xffffffffu;
    }
    tq_init(uq);
    tq_init(dq);
    if (P.size == 0) {
      if (tid == 0) { out_count[q] = 0; stats[q] = QueryStats{0, 0, 0, 0, 0}; }
      __syncthreads();
      continue;
    }
    // ---- rotation (Rotation::mul, the OpenBLAS sgemv order) ------------------
    qbg_rotate(qb, qf, qlen, rq);
    // ---- seeds: tree leaf of the global index, else the fixed random list ---
    const uint32_t* seeds = nullptr;
    uint32_t nseeds = 0;
    if (tid == 0) s.seed_leaf = 0xffffffffu;
    __syncthreads();
    if (warp == 0 && P.seed_cnt == 0xffffffffu) {
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
        else { s.seed_leaf = 0xffffffffu; s.status |= kStatusTreeError; }
      }
    }
    __syncthreads();
    if (P.seed_cnt == 0xffffffffu && s.seed_leaf != 0xffffffffu && s.seed_leaf < g.nleaves) {
      const uint32_t* off = g.leaf_seed_off + P.seed_off;
      uint32_t a = off[s.seed_leaf], b = off[s.seed_leaf + 1];
      seeds = g.leaf_seed_ids + a;
      nseeds = b - a;
    }
    if (nseeds == 0) {
      seeds = seed_list + P.fb_off;
      nseeds = P.fb_cnt;
    }
    nseeds = min(nseeds, (uint32_t)kExactChunk);
    if (nseeds == 0) {
      if (tid == 0) { out_count[q] = 0; stats[q] = QueryStats{0, 0, 0, 0, s.status | kStatusEmptySeeds}; }
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
    for (uint32_t i = tid; i < nseeds; i += blockDim.x) {
      uint32_t id = key_id(bsorted[i]);
      atomicOr(&bitmap[id >> 5], 1u << (id & 31u));
    }
    if (tid == 0) {
      s.current = bsorted[0];
      s.expR = __fmul_rn(P.bcoef, key_dist(bsorted[0]));
      s.dc = nseeds;
    }
    __syncthreads();
    tq_push_sorted(uq, bsorted, nseeds);
    tq_push_sorted(dq, bsorted + 1, nseeds - 1);

    // ---- main loop ------------------------------------------------------------
    uint32_t guard = 0;
    while (true) {
      if (++guard > 4u * g.nrows + 64u) {            // each node is traced / judged at most once
        if (tid == 0) s.status |= kStatusIterationLimit;
        break;
      }
      const unsigned long long t = tq_top(uq);
      if (t == ~0ull || key_dist(t) > s.expR) {
        // ---- judge the current blob ----
        const uint32_t blob = key_id(s.current);
        if (tid == 0) s.exploration++;
        qbg_judge_blob<SPL>(qb, blob_sid, blob, rq, flut, lut, s, bdist, resb, bkeys, bsorted, P.size);
        // ---- stop, or take the nearest waiting blob ----
        if (s.bmin > __fmul_rn(s.radius, P.coef) || s.exploration > P.explored) break;
        const unsigned long long nxt = tq_top(dq);
        if (nxt == ~0ull) break;
        tq_pop(dq);
        if (tid == 0) {
          s.current = nxt;
          s.expR = __fmul_rn(P.bcoef, key_dist(nxt));
        }
        __syncthreads();
        continue;
      }
      // ---- expand the nearest untraced node of the global graph ----
      tq_pop(uq);
      const uint32_t target = key_id(t);
      const uint32_t e0 = g.offsets[target];
      const uint32_t deg = g.offsets[target + 1] - e0;
      const uint32_t nsz = min(deg, P.edge_size);
      if (tid == 0) s.expansions++;
      for (uint32_t c0 = 0; c0 < nsz; c0 += kExactChunk) {
        const uint32_t clen = min((uint32_t)kExactChunk, nsz - c0);
        bool isnew = false;
        uint32_t id = 0;
        if ((uint32_t)tid < clen) {
          id = g.edges[e0 + c0 + tid];
          const uint32_t bit = 1u << (id & 31u);
          isnew = (atomicOr(&bitmap[id >> 5], bit) & bit) == 0u;
        }
        unsigned ballot = __ballot_sync(0xffffffffu, isnew);
        if (lane == 0) s.warp_cnt[warp] = __popc(ballot);
        __syncthreads();
        uint32_t base = 0, nnew = 0;
        for (int w = 0; w < kExactWarps; w++) {
          if (w < warp) base += s.warp_cnt[w];
          nnew += s.warp_cnt[w];
        }
        if (isnew) nid[base + __popc(ballot & ((1u << lane) - 1u))] = id;
        __syncthreads();
        for (uint32_t b = (uint32_t)(warp * (32 / G)); b < nnew; b += ngroups) {
          uint32_t i = b + (uint32_t)(lane / G);
          bool valid = i < nnew;
          uint32_t v = valid ? nid[i] : 0u;
          float d = group_distance<ObjType::Float, Metric::L2>(qv, g.objects + (size_t)v * rc, (int)rc, gl, G);
          if (valid && gl == 0) nd[i] = d;
        }
        __syncthreads();
        if (nnew == 0) continue;
        // the first neighbour (edge order) strictly nearer than the current blob
        // replaces it; everything else waits
        if (warp == 0) {
          float best = FLT_MAX;
          uint32_t bi = 0xffffffffu;
          for (uint32_t i = lane; i < nnew; i += 32) {
            if (nd[i] < best) { best = nd[i]; bi = i; }
          }
          for (int off = 16; off > 0; off >>= 1) {
            float ob = __shfl_xor_sync(0xffffffffu, best, off);
            uint32_t oi = __shfl_xor_sync(0xffffffffu, bi, off);
            if (ob < best || (ob == best && oi < bi)) { best = ob; bi = oi; }
          }
          if (lane == 0) s.nacc = (best < key_dist(s.current)) ? bi : 0xffffffffu;
        }
        __syncthreads();
        const uint32_t rep = s.nacc;
        for (uint32_t i = tid; i < nnew; i += blockDim.x) bkeys[i] = pack_key(nd[i], nid[i]);
        __syncthreads();
        rank_sort(bkeys, bsorted, nnew);
        __syncthreads();
        tq_push_sorted(uq, bsorted, nnew);
        // waiting blobs: the new nodes except the replacement, plus the old current
        uint32_t nw = 0;
        {
          const unsigned long long repk = rep != 0xffffffffu ? pack_key(nd[rep], nid[rep]) : ~0ull;
          const unsigned long long oldc = s.current;
          // bsorted without repk, with oldc inserted in order (when replaced)
          for (uint32_t i = tid; i < nnew; i += blockDim.x) {
            unsigned long long k = bsorted[i];
            if (k == repk) continue;
            uint32_t pos = i - (repk != ~0ull && repk < k ? 1u : 0u) + (rep != 0xffffffffu && oldc < k ? 1u : 0u);
            batch[pos] = k;
          }
          if (tid == 0 && rep != 0xffffffffu) {
            uint32_t pos = lower_bound_keys(bsorted, nnew, oldc);
            pos -= (repk < oldc) ? 1u : 0u;
            batch[pos] = oldc;
          }
          nw = nnew;                                // -1 replacement +1 old current, or all new
        }
        __syncthreads();
        tq_push_sorted(dq, batch, nw);
        if (tid == 0 && rep != 0xffffffffu) {
          s.current = pack_key(nd[rep], nid[rep]);
          s.expR = __fmul_rn(P.bcoef, nd[rep]);
        }
        if (tid == 0) s.dc += nnew;
        __syncthreads();
      }
      __syncthreads();
    }
    // ---- results: ascending (distance, id), quantized distances ----------------
    __syncthreads();
    const uint32_t n = s.nres;
    const unsigned long long* res = resb[s.rcur];
    for (uint32_t i = tid; i < n; i += blockDim.x) out[P.out_off + i] = ObjDist{key_id(res[i]), key_dist(res[i])};
    if (tid == 0) {
      uint32_t st = s.status | (s.uq.status || s.dq.status ? kStatusCandidateOverflow : 0u);
      out_count[q] = n;
      stats[q] = QueryStats{s.dc, s.expansions, s.nblobs, 0, st};
    }
    // leave the visited bitmap clean for the next query
    for (uint32_t i = tid; i < cfg.bitmap_words; i += blockDim.x) bitmap[i] = 0u;
    __threadfence();
    __syncthreads();
  }
}

// ---- the two-step search's blob phase ------------------------------------------------

constexpr uint32_t kScanBatch = 64;                 // blobs scored before their objects are merged
constexpr uint32_t kScanLocalBytes = 16 << 10;      // local codebooks up to this size are kept in shared memory

constexpr uint32_t kScanKeys = 256;                 // candidates of a batch's selection
constexpr uint32_t kScanBins = 2 * kScanKeys * 2;   // its histogram lies over both key buffers

struct QBGScanShared {
  uint32_t query, nb, merged;
  uint32_t dmin, dmax;                              // bits of the batch's extreme eligible distances
  uint32_t bin, below, drop;
  uint32_t wsum[kExactWarps];
  uint32_t blob[kScanBatch], count[kScanBatch], at[kScanBatch];
  float bmin[kScanBatch];
};

// Distances a CTA buffers per batch: at least one blob of any size.
inline uint32_t qbg_scan_dist_cap(uint32_t blob_cap) { return blob_cap > 12288u ? blob_cap : 12288u; }

// A batch's selection needs larger key buffers than a chunk's: where the result set is small
// enough for it, and the query row is not most of the shared memory.
__host__ __device__ __forceinline__ bool qbg_scan_select(uint32_t dim, uint32_t rcap) {
  return rcap <= 1024u && dim <= 4096u;
}

// The local codebooks and each warp's residual lie in shared memory when they are small and
// the result set leaves the room; else they are read from global memory.
__host__ __device__ __forceinline__ bool qbg_scan_local(uint32_t dim, uint32_t rcap) {
  return (size_t)dim * 64 <= kScanLocalBytes && rcap <= 1024u;
}

inline size_t qbg_scan_smem_bytes(uint32_t row_chunks, uint32_t dim, uint32_t m, uint32_t rcap) {
  size_t b = (size_t)row_chunks * 16;
  b += ((size_t)dim * 4 + 15) / 16 * 16;
  b += (size_t)m * 16 * kExactWarps;
  b += (size_t)rcap * 16;
  b += (size_t)(qbg_scan_select(dim, rcap) ? kScanKeys : (uint32_t)kExactChunk) * 16;
  if (qbg_scan_local(dim, rcap)) b += (size_t)dim * (64 + 4 * kExactWarps);
  b += sizeof(QBGScanShared) + 16;
  return b;
}

// The uint8 distance table of the rotated query against subspace-id centroid `gc`, by one
// warp into its shared bytes lut[M * 16].  The entries, their minimum, scale and rounding
// are qbg_build_lut's: each entry is computed twice (once for the extremes) instead of
// being stored, and an entry's rounded quotient comes from a product with 1 / scale unless
// that lies within 1/1024 of a half, where the division decides (the product is at most
// 255 and within 3 half-units of the last place of the quotient).  The loops stay rolled:
// unrolled, the kernel's code no longer fitted the instruction cache (the scan took 4.0 ms instead of 0.94).
// lc: the local centroids [(subspace * 16 + c) * LD + d]; rsv: the residual, if the caller
// has room for it (D floats, written here), else null.  LDC: LD if it is known, else 0.
template <int LDC>
__device__ __forceinline__ void qbg_warp_lut(uint32_t M, uint32_t LD, const float* rq, const float* __restrict__ gc,
                                             const float* lc, float* rsv, uint8_t* lut, float& scale, float& offset,
                                             int lane) {
  if (LDC) LD = LDC;
  __syncwarp();                                              // the table before has been read
  if (rsv) {
    for (uint32_t i = (uint32_t)lane; i < M * LD; i += 32) rsv[i] = __fsub_rn(rq[i], __ldg(gc + i));
    __syncwarp();
  }
  auto entry = [&](uint32_t e) {
    const uint32_t s0 = (e >> 4) * LD;
    if constexpr (LDC == 2) {                                // rsv is given, both 8-byte aligned
      const float2 r = *reinterpret_cast<const float2*>(rsv + s0);
      const float2 l = *reinterpret_cast<const float2*>(lc + (size_t)e * 2);
      const float s0v = __fsub_rn(r.x, l.x), s1v = __fsub_rn(r.y, l.y);
      return __fmaf_rn(s1v, s1v, __fmul_rn(s0v, s0v));
    } else {
      float v = 0.f;
      for (uint32_t d = 0; d < LD; d++) {
        const float r = rsv ? rsv[s0 + d] : __fsub_rn(rq[s0 + d], __ldg(gc + s0 + d));
        const float sub = __fsub_rn(r, lc[(size_t)e * LD + d]);
        v = d == 0 ? __fmul_rn(sub, sub) : __fmaf_rn(sub, sub, v);
      }
      return v;
    }
  };
  float mn = FLT_MAX, mx = -FLT_MAX;
#pragma unroll 2
  for (uint32_t e = (uint32_t)lane; e < M * 16; e += 32) {
    const float v = entry(e);
    mn = fminf(mn, v);
    mx = fmaxf(mx, v);
  }
  for (int off = 16; off > 0; off >>= 1) {
    mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, off));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  }
  scale = __double2float_rn(__ddiv_rn((double)__fsub_rn(mx, mn), 255.0));
  offset = __fmul_rn(mn, (float)M);
  const float inv = 1.f / scale;
#pragma unroll 2
  for (uint32_t e = (uint32_t)lane; e < M * 16; e += 32) {
    const float x = __fsub_rn(entry(e), mn);
    const float y = x * inv;
    float r = rintf(y);
    if (!(fabsf(y - r) < 0.499f)) r = rintf(__fdiv_rn(x, scale));   // near a half (or not finite)
    lut[e] = (uint8_t)(int)r;
  }
  __syncwarp();
}

// The blob phase of searchInTwoSteps (lib/NGT/NGTQ/QuantizedBlobGraph.h:1240-1306):
// one query per CTA; its probed blobs (blobs[q * bstride ..], bcount[q] of them,
// nearest first, from the global index's graph search) are judged in that order
// with a result set of P.size.  Results: the quantized distances, ascending.
//
// A blob's distances do not depend on the radius that the blobs before it left, only which
// of its objects join the results does.  So a batch of blobs is scored first, each blob by
// one warp with the table in its registers, in the order of their subspace ids (blobs of
// one id share the table).  An object beyond the radius of its turn is beyond the last
// result too, so the batch's part of the results is its P.size smallest keys, which one
// histogram of the distances finds; only where the set's last distance is tied and a blob's
// nearest object lies at that very distance does the order of the blobs decide, and then
// (or when a histogram bin holds too many) the batch is judged blob by blob, a blob whose
// minimum is not below the radius taking no barrier.  Bound by instruction issue (the codes'
// table look-ups).  3,000 queries of 64 probes over 1M x 128, 64 subspaces: blob by blob,
// the whole CTA building each blob's table and about ten barriers a blob, 1346 us; scored by
// batch 942 us; selected by batch 762 us (9 CTAs an SM instead of 7: 769 us).
template <int SPL>
__global__ void __launch_bounds__(kExactThreads)
qbg_scan_kernel(DevQG qb, const uint32_t* __restrict__ blob_sid, const uint4* __restrict__ queries,
                uint32_t row_chunks, uint32_t nq, const QBGParams* __restrict__ params,
                const ObjDist* __restrict__ blobs, const uint32_t* __restrict__ bcount, uint32_t bstride,
                ObjDist* __restrict__ out, uint32_t* __restrict__ out_count, QueryStats* __restrict__ stats,
                float* __restrict__ blob_dist, uint32_t dist_cap, uint32_t rcap, uint32_t* __restrict__ work) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t rc = row_chunks;
  const uint32_t D = qb.dim, M = qb.m, LD = qb.ld;
  uint4* qv = reinterpret_cast<uint4*>(smem);
  float* rq = reinterpret_cast<float*>(qv + rc);
  uint8_t* lut = reinterpret_cast<uint8_t*>(rq + (D + 3) / 4 * 4) + (size_t)warp * M * 16;
  unsigned long long* res = reinterpret_cast<unsigned long long*>(rq + (D + 3) / 4 * 4 + (size_t)M * 4 * kExactWarps);
  unsigned long long* bkeys = res + 2 * (size_t)rcap;
  const bool select = qbg_scan_select(D, rcap);
  const uint32_t nkeys = select ? kScanKeys : (uint32_t)kExactChunk;
  unsigned long long* bsorted = bkeys + nkeys;
  uint32_t* hist = reinterpret_cast<uint32_t*>(bkeys);
  // the batch's subspace ids, and its positions in their order: needed until the judging
  uint32_t* bsid = reinterpret_cast<uint32_t*>(bkeys);
  uint32_t* order = reinterpret_cast<uint32_t*>(bsorted);
  const bool local = qbg_scan_local(D, rcap);
  float* lt = reinterpret_cast<float*>(bsorted + nkeys);
  float* rsv = lt + (size_t)D * 16 + (size_t)warp * D;
  QBGScanShared& s = *reinterpret_cast<QBGScanShared*>(lt + (local ? (size_t)D * (16 + kExactWarps) : 0));
  float* bdist = blob_dist + (size_t)blockIdx.x * dist_cap;
  const float* qf = reinterpret_cast<const float*>(qv);
  if (local)
    for (uint32_t i = tid; i < M * 16 * LD; i += kExactThreads) lt[i] = qb.lcentroids[i];
  for (uint32_t q = exact_next_query(0xffffffffu, work, &s.query); q < nq; q = exact_next_query(q, work, &s.query)) {
    const QBGParams P = params[q];
    for (uint32_t i = tid; i < rc; i += kExactThreads) qv[i] = queries[(size_t)q * rc + i];
    __syncthreads();
    const uint32_t nb = P.size == 0 ? 0u : bcount[q];
    if (nb > 0) qbg_rotate(qb, qf, rc * 4, rq);
    uint32_t nres = 0, cur = 0, judged = 0, dc = 0;              // alike in every thread
    float radius = FLT_MAX;
    for (uint32_t b0 = 0; b0 < nb;) {
      __syncthreads();
      // the batch: as many blobs as the distance buffer holds (one at least)
      const uint32_t bn = min(kScanBatch, nb - b0);
      if ((uint32_t)tid < bn) {
        const uint32_t blob = blobs[(size_t)q * bstride + b0 + tid].id;
        const bool has = blob < qb.nnodes;
        const uint32_t a = has ? qb.offsets[blob] : 0u;
        s.blob[tid] = blob;
        s.count[tid] = has ? qb.offsets[blob + 1] - a : 0u;
        bsid[tid] = has ? blob_sid[blob] : 0xffffffffu;
        s.bmin[tid] = FLT_MAX;
      }
      __syncthreads();
      if (warp == 0) {
        uint32_t sum = 0, fit = 0;
        for (uint32_t b = 0; b < bn; b += 32) {
          const uint32_t i = b + (uint32_t)lane;
          const uint32_t len = i < bn ? (s.count[i] + 15) / 16 * 16 : 0u;
          uint32_t incl = len;
#pragma unroll
          for (int off = 1; off < 32; off <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += y;
          }
          if (i < bn) s.at[i] = sum + incl - len;
          fit += (uint32_t)__popc(__ballot_sync(0xffffffffu, i < bn && (sum + incl <= dist_cap || i == 0)));
          sum += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) {
          s.nb = fit;
          s.dmin = 0xffffffffu;
          s.dmax = 0u;
          s.merged = 0u;
          s.drop = 0xffffffffu;
        }
      } else if (warp == 1 || warp == 2) {
        // positions by (subspace id, probe order)
        const uint32_t i = (uint32_t)tid - 32u;
        if (i < bn) {
          const uint32_t mine = bsid[i];
          uint32_t r = 0;
          for (uint32_t j = 0; j < bn; j++) r += (bsid[j] < mine || (bsid[j] == mine && j < i)) ? 1u : 0u;
          order[r] = i;
        }
      }
      __syncthreads();
      const uint32_t bfit = s.nb;
      // scoring: each warp a run of the sorted blobs (those past bfit wait for the next batch)
      {
        const uint32_t per = (bn + kExactWarps - 1) / kExactWarps;
        uint32_t L[SPL][4];
        float lscale = 0.f, loffset = 0.f;
        uint32_t have_sid = 0xffffffffu;
        float dmin = FLT_MAX, dmax = 0.f;                        // of this warp's eligible distances
        const uint32_t end = min(bn, ((uint32_t)warp + 1) * per);
        for (uint32_t k = (uint32_t)warp * per; k < end; k++) {
          const uint32_t i = order[k];
          const uint32_t n = s.count[i];
          if (i >= bfit || n == 0) continue;                     // warp-uniform
          if (bsid[i] != have_sid) {
            have_sid = bsid[i];
            const float* gc = qb.gcentroid + (size_t)have_sid * D;
            if (local && LD == 2)
              qbg_warp_lut<2>(M, LD, rq, gc, lt, rsv, lut, lscale, loffset, lane);
            else
              qbg_warp_lut<0>(M, LD, rq, gc, local ? lt : qb.lcentroids, local ? rsv : nullptr, lut, lscale, loffset,
                              lane);
#pragma unroll
            for (int j = 0; j < SPL; j++) {
              const uint32_t sv = (uint32_t)lane + 32u * (uint32_t)j;
              const uint4 v = sv < M ? reinterpret_cast<const uint4*>(lut)[sv] : make_uint4(0, 0, 0, 0);
              L[j][0] = v.x; L[j][1] = v.y; L[j][2] = v.z; L[j][3] = v.w;
            }
          }
          const uint8_t* stream = qb.codes + (size_t)qb.code_off16[s.blob[i]] * 16;
          float* dst = bdist + s.at[i];
          const uint32_t nblk = (n + 15) / 16;
          constexpr int BPI = SPL <= 4 ? 2 : 1;                  // code blocks loaded before they are scored
          float wmin = FLT_MAX;
          for (uint32_t bi = 0; bi < nblk; bi += BPI) {
            uint2 w[BPI][SPL];
#pragma unroll
            for (int u = 0; u < BPI; u++)
              qg_block_words<SPL>(stream + (size_t)min(bi + u, nblk - 1) * 8 * qb.ma, qb.ma, lane, w[u]);
#pragma unroll
            for (int u = 0; u < BPI; u++) {
              int o;
              const float d = qg_block_distance_words<SPL>(w[u], L, M, lscale, loffset, lane, &o);
              const uint32_t pos = (bi + u) * 16 + (uint32_t)o;
              if (o >= 0 && bi + u < nblk) {
                const bool in = pos < n;
                dst[pos] = in ? d : INFINITY;                    // a block's padding is never eligible
                if (in) {
                  wmin = fminf(wmin, d);
                  if (d <= radius) dmax = fmaxf(dmax, d);
                }
              }
            }
          }
          for (int off = 16; off > 0; off >>= 1) wmin = fminf(wmin, __shfl_xor_sync(0xffffffffu, wmin, off));
          if (lane == 0) s.bmin[i] = wmin;
          dmin = fminf(dmin, wmin);
        }
        if (select) {
          for (int off = 16; off > 0; off >>= 1) dmax = fmaxf(dmax, __shfl_xor_sync(0xffffffffu, dmax, off));
          if (lane == 0) {
            atomicMin(&s.dmin, __float_as_uint(dmin));
            atomicMax(&s.dmax, __float_as_uint(dmax));
          }
        }
      }
      __threadfence_block();
      __syncthreads();
      // selecting: the batch at once
      bool selected = false;
      if (select && P.size <= kScanKeys - 32) {
        const uint32_t total = s.at[bfit - 1] + (s.count[bfit - 1] + 15) / 16 * 16;
        const uint32_t mnb = s.dmin, span = s.dmax >= mnb ? s.dmax - mnb : 0u;
        uint32_t shift = 0;
        while ((span >> shift) >= kScanBins) shift++;
        for (uint32_t j = tid; j < kScanBins / 4; j += kExactThreads)
          reinterpret_cast<uint4*>(hist)[j] = make_uint4(0u, 0u, 0u, 0u);
        __syncthreads();
        const float4* b4 = reinterpret_cast<const float4*>(bdist);
#pragma unroll 2
        for (uint32_t j = tid; j < total / 4; j += kExactThreads) {
          const float4 v = b4[j];
          if (v.x <= radius) atomicAdd(&hist[(__float_as_uint(v.x) - mnb) >> shift], 1u);
          if (v.y <= radius) atomicAdd(&hist[(__float_as_uint(v.y) - mnb) >> shift], 1u);
          if (v.z <= radius) atomicAdd(&hist[(__float_as_uint(v.z) - mnb) >> shift], 1u);
          if (v.w <= radius) atomicAdd(&hist[(__float_as_uint(v.w) - mnb) >> shift], 1u);
        }
        __syncthreads();
        // the bin of the P.size-th distance (the last bin, if there are fewer)
        constexpr uint32_t kPer = kScanBins / kExactThreads;
        uint32_t mine = 0;
#pragma unroll
        for (uint32_t j = 0; j < kPer; j++) mine += hist[tid * kPer + j];
        uint32_t incl = mine;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const uint32_t y = __shfl_up_sync(0xffffffffu, incl, off);
          if (lane >= off) incl += y;
        }
        if (lane == 31) s.wsum[warp] = incl;
        __syncthreads();
        uint32_t all = 0;
#pragma unroll
        for (int w = 0; w < kExactWarps; w++) {
          if (w < warp) incl += s.wsum[w];
          all += s.wsum[w];
        }
        if (all < P.size) {
          if (tid == 0) { s.bin = kScanBins; s.below = all; }
        } else if (incl >= P.size && incl - mine < P.size) {
          uint32_t c = incl - mine;
          for (uint32_t j = 0; j < kPer; j++) {
            c += hist[tid * kPer + j];
            if (c >= P.size) { s.bin = tid * kPer + j; s.below = c; break; }
          }
        }
        __syncthreads();
        const uint32_t bin = s.bin, m = s.below;
        if (m <= kScanKeys) {                                    // else too many in one bin: blob by blob
          for (uint32_t j = tid; j < total / 4; j += kExactThreads) {
            const float4 v = b4[j];
            const float vs[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int u = 0; u < 4; u++) {
              if (!(vs[u] <= radius) || ((__float_as_uint(vs[u]) - mnb) >> shift) > bin) continue;
              const uint32_t p = j * 4 + (uint32_t)u;
              uint32_t lo = 0, hi = bfit;                        // the last blob that begins at or before p
              while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) / 2;
                if (s.at[mid] <= p) lo = mid; else hi = mid;
              }
              bkeys[atomicAdd(&s.merged, 1u)] = pack_key(vs[u], __ldg(qb.ids + qb.offsets[s.blob[lo]] + p - s.at[lo]));
            }
          }
          __syncthreads();
          for (uint32_t i = tid; i < m; i += kExactThreads) {
            const unsigned long long k = bkeys[i];
            uint32_t r = 0;
            for (uint32_t j = 0; j < m; j++) {
              const unsigned long long o = bkeys[j];
              r += (o < k || (o == k && j < i)) ? 1u : 0u;
            }
            bsorted[r] = k;
          }
          __syncthreads();
          const unsigned long long* old = res + (size_t)cur * rcap;
          unsigned long long* dst = res + (size_t)(cur ^ 1u) * rcap;
          auto place = [&](unsigned long long k, uint32_t pos) {
            if (pos < P.size) dst[pos] = k;
            else if (pos == P.size) s.drop = __float_as_uint(key_dist(k));
          };
          for (uint32_t j = tid; j < nres; j += kExactThreads) place(old[j], j + lower_bound_keys(bsorted, m, old[j]));
          for (uint32_t j = tid; j < m; j += kExactThreads)
            place(bsorted[j], j + lower_bound_keys(old, nres, bsorted[j]));
          __syncthreads();
          const uint32_t nnew = min(nres + m, P.size);
          const float last = nnew >= P.size ? key_dist(dst[P.size - 1]) : FLT_MAX;
          // a tie across the set's end, with a blob that begins at it: its turn decides
          selected = __float_as_uint(last) != s.drop ||
                     !__syncthreads_or((uint32_t)tid < bfit && s.bmin[tid] == last);
          if (selected) {
            nres = nnew;
            cur ^= 1u;
            radius = last;
            for (uint32_t i = 0; i < bfit; i++) {
              if (s.blob[i] >= qb.nnodes) continue;
              judged++;
              dc += s.count[i];
            }
          }
          __syncthreads();
        }
      }
      // judging, in probe order
      for (uint32_t i = 0; i < bfit && !selected; i++) {
        if (s.blob[i] >= qb.nnodes) continue;
        judged++;
        const uint32_t n = s.count[i];
        dc += n;
        const float radius0 = radius;
        if (!(s.bmin[i] < radius0)) continue;
        const uint32_t a = qb.offsets[s.blob[i]];
        const float* src = bdist + s.at[i];
        for (uint32_t c0 = 0; c0 < n; c0 += kExactChunk) {
          if (tid == 0) s.merged = 0;
          __syncthreads();
          const uint32_t e = c0 + (uint32_t)tid;
          const float d = e < n ? src[e] : FLT_MAX;
          const bool acc = e < n && d <= radius0;
          const uint32_t mask = __ballot_sync(0xffffffffu, acc);
          uint32_t at = 0;
          if (lane == 0 && mask) at = atomicAdd(&s.merged, (uint32_t)__popc(mask));
          at = __shfl_sync(0xffffffffu, at, 0);
          if (acc) bkeys[at + __popc(mask & ((1u << lane) - 1u))] = pack_key(d, __ldg(qb.ids + a + e));
          __syncthreads();
          const uint32_t m = s.merged;
          if (m == 0) continue;
          rank_sort_split<kExactThreads>(bkeys, bsorted, m);
          __syncthreads();
          // the smallest P.size of both, into the other buffer
          const unsigned long long* old = res + (size_t)cur * rcap;
          unsigned long long* dst = res + (size_t)(cur ^ 1u) * rcap;
          for (uint32_t j = tid; j < nres; j += kExactThreads) {
            const uint32_t pos = j + lower_bound_keys(bsorted, m, old[j]);
            if (pos < P.size) dst[pos] = old[j];
          }
          if ((uint32_t)tid < m) {
            const uint32_t pos = (uint32_t)tid + lower_bound_keys(old, nres, bsorted[tid]);
            if (pos < P.size) dst[pos] = bsorted[tid];
          }
          nres = min(nres + m, P.size);
          cur ^= 1u;
        }
        __syncthreads();
        if (nres >= P.size) radius = key_dist(res[(size_t)cur * rcap + nres - 1]);
      }
      b0 += bfit;
    }
    __syncthreads();
    const unsigned long long* r = res + (size_t)cur * rcap;
    for (uint32_t i = tid; i < nres; i += kExactThreads) out[P.out_off + i] = ObjDist{key_id(r[i]), key_dist(r[i])};
    if (tid == 0) {
      out_count[q] = nres;
      stats[q] = QueryStats{dc, 0, judged, 0, 0};
    }
    __syncthreads();
  }
}

// refineDistances (lib/NGT/NGTQ/QuantizedBlobGraph.h:1136-1185): per query (one CTA)
// the cand_count[q] candidates at cand[q * cstride ..] get their exact L2 distances
// over the object list (rows of `orc` 16-byte chunks, row 0 unused; the float query
// cast element-wise to the row type, as setObject does), are sorted by (distance,
// id) and the first min(exact[q], n) written to out[q * kmax ..].
// M: the comparator (L2 for QBG; the index's distance for a graph index's refinement
// objects, lib/NGT/Index.h:1146-1236).
template <ObjType OT, Metric M = Metric::L2>
__global__ void __launch_bounds__(256)
qbg_refine_kernel(const ObjDist* __restrict__ cand, const uint32_t* __restrict__ cand_count, uint32_t cstride,
                  const float* __restrict__ qrows, uint32_t qdim, const uint4* __restrict__ olist, uint32_t orc,
                  uint32_t odim, uint32_t nrows, const uint32_t* __restrict__ exact, uint32_t nq, uint32_t P,
                  ObjDist* __restrict__ out, uint32_t kmax, uint32_t* __restrict__ out_count) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint4* qv = reinterpret_cast<uint4*>(smem);                                        // orc chunks
  unsigned long long* keys = reinterpret_cast<unsigned long long*>(qv + orc);          // P
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t G = 1;
  while (G < orc && G < 32) G <<= 1;
  const uint32_t gl = lane & (G - 1), gpw = 32 / G, ngroups = blockDim.x / G;
  for (uint32_t q = blockIdx.x; q < nq; q += gridDim.x) {
    const uint32_t n = min(cand_count[q], P);
    if constexpr (OT == ObjType::Uint8) {
      uint8_t* qb = reinterpret_cast<uint8_t*>(qv);
      for (uint32_t i = threadIdx.x; i < orc * 16; i += blockDim.x)
        qb[i] = i < odim && i < qdim ? (uint8_t)__float2int_rz(qrows[(size_t)q * qdim + i]) : (uint8_t)0;
    } else {
      float* qb = reinterpret_cast<float*>(qv);
      for (uint32_t i = threadIdx.x; i < orc * 4; i += blockDim.x)
        qb[i] = i < odim && i < qdim ? qrows[(size_t)q * qdim + i] : 0.f;
    }
    for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) keys[i] = ~0ull;
    __syncthreads();
    for (uint32_t b = warp * gpw; b < n; b += ngroups) {
      const uint32_t i = b + lane / G;
      const bool valid = i < n;
      const uint32_t id = valid ? cand[(size_t)q * cstride + i].id : 0u;
      const bool inrange = id > 0 && id < nrows;
      const float d = group_distance<OT, M>(qv, olist + (size_t)(inrange ? id : 0u) * orc, (int)orc, (int)gl,
                                            (int)G);
      if (valid && gl == 0) keys[i] = pack_key(inrange ? d : FLT_MAX, id);
    }
    __syncthreads();
    for (uint32_t k2 = 2; k2 <= P; k2 <<= 1) {
      for (uint32_t j = k2 >> 1; j > 0; j >>= 1) {
        for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) {
          const uint32_t l = i ^ j;
          if (l > i) {
            const unsigned long long x = keys[i], y = keys[l];
            const bool up = (i & k2) == 0;
            if ((x > y) == up) {
              keys[i] = y;
              keys[l] = x;
            }
          }
        }
        __syncthreads();
      }
    }
    const uint32_t m = min(exact[q], n);
    for (uint32_t i = threadIdx.x; i < m; i += blockDim.x)
      out[(size_t)q * kmax + i] = ObjDist{key_id(keys[i]), key_dist(keys[i])};
    if (threadIdx.x == 0) out_count[q] = m;
    __syncthreads();
  }
}

}  // namespace ngtg
