// Exhaustive (linear) k-NN search with the reference's exact ordering.
//
// Reference: ObjectSpaceRepository::linearSearch (lib/NGT/ObjectSpaceRepository.h:860-922):
// every object id 1..N is compared, objects with d <= radius (or all, when the
// radius is negative) enter a bounded max-heap of `size`; ties keep the
// smaller id because the heap orders by (distance, id) and ids arrive in
// increasing order.  The result is therefore exactly the `size` smallest
// (distance, id) keys, which is what the kernels below compute:
//   1. linear_distance_kernel: distances for a block of queries x all rows
//      (group-cooperative 16-byte loads, same comparators as the graph search);
//   2. linear_radix_kernel, one launch per 11-bit digit: per query, a radix
//      select of the k-th smallest (distance, id) key over all blocks of a grid
//      (linear_select.cuh);
//   3. linear_collect_kernel: the keys up to it, sorted.
#pragma once
#include <cfloat>
#include "distance.cuh"
#include "device_index.h"

namespace ngtg {

constexpr int kLinThreads = 256;
constexpr int kLinRowsPerBlock = 512;
// Rows a lane group computes at once.  Bound by HBM: a group that loads one row and
// reduces it before the next keeps too few bytes in flight when a row is a single
// 16-byte chunk per lane (dim <= 128 float).  Every row's lanes and summation order
// are those of group_distance, so the distances do not depend on it.
constexpr int kLinRows = 4;

template <ObjType OT, Metric M>
__global__ void __launch_bounds__(kLinThreads)
linear_distance_kernel(DevGraph g, const uint4* __restrict__ queries, uint32_t q0, uint32_t nqb,
                       const uint8_t* __restrict__ present, float* __restrict__ dist, uint32_t group) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint4* qv = reinterpret_cast<uint4*>(smem);
  const uint32_t rc = g.row_chunks;
  const uint32_t qi = blockIdx.y;
  const uint32_t q = q0 + qi;
  for (uint32_t i = threadIdx.x; i < rc; i += blockDim.x) qv[i] = queries[(size_t)q * rc + i];
  __syncthreads();
  const int G = (int)group;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gl = lane & (G - 1);
  const uint32_t gpw = 32 / G, ngroups = kLinThreads / G;
  const uint32_t r0 = blockIdx.x * kLinRowsPerBlock;
  const uint32_t r1 = min(g.nrows, r0 + kLinRowsPerBlock);
  // a warp's groups take kLinRows x gpw consecutive rows at a time
  for (uint32_t b = r0 + warp * gpw * kLinRows; b < r1; b += ngroups * kLinRows) {
    uint32_t row[kLinRows];
    Acc<OT, M> acc[kLinRows];
#pragma unroll
    for (int u = 0; u < kLinRows; u++) {
      const uint32_t r = b + u * gpw + (uint32_t)(lane / G);
      row[u] = r < r1 ? r : 0u;
    }
    for (uint32_t c = gl; c < rc; c += G) {
      uint4 xv[kLinRows];
#pragma unroll
      for (int u = 0; u < kLinRows; u++) xv[u] = __ldg(g.objects + (size_t)row[u] * rc + c);
      const uint4 qc = qv[c];
#pragma unroll
      for (int u = 0; u < kLinRows; u++) acc[u].add(qc, xv[u], (int)c);
    }
#pragma unroll
    for (int u = 0; u < kLinRows; u++) {
      acc[u].reduce(G);
      const float d = acc[u].finish();
      const uint32_t r = b + u * gpw + (uint32_t)(lane / G);
      if (gl == 0 && r < r1) {
        const bool ok = r != 0 && present[r];
        dist[(size_t)qi * g.nrows + r] = ok ? d : __int_as_float(0x7f800000);  // +inf = excluded
      }
    }
  }
}

}  // namespace ngtg
