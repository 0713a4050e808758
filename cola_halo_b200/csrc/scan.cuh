// Exclusive prefix sum of unsigned counts on the device, shared by the
// counting sorts (friends-of-friends cell binning, particle cell order).
#pragma once
#include <cuda_runtime.h>

#include "internal.h"

namespace cgscan {
namespace {

constexpr int SCAN_B = 4096;   // elements per scan block
constexpr int SCAN_T = 256;    // its threads: 16 elements each, in 4 vectors
constexpr int SCAN_V = SCAN_B / (4 * SCAN_T);
constexpr int SUMS_T = 1024;   // threads of the scan over the block totals

// Vector v of a thread: warps take 512 consecutive elements each, a warp's
// lanes 4 of every 128.  Elements past n count as 0.
__device__ __forceinline__ long long scan_at(long long block, int v) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  return block * SCAN_B + warp * (SCAN_V * 128) + v * 128 + lane * 4;
}
__device__ __forceinline__ uint4 scan_load(const unsigned* __restrict__ in, long long i,
                                           long long n) {
  if (i + 4 <= n) return *reinterpret_cast<const uint4*>(in + i);
  return make_uint4(i < n ? in[i] : 0u, i + 1 < n ? in[i + 1] : 0u, i + 2 < n ? in[i + 2] : 0u,
                    0u);
}
// Inclusive scan over a warp's lanes.
__device__ __forceinline__ unsigned warp_scan(unsigned v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

// Totals of the blocks.
__global__ void __launch_bounds__(SCAN_T) k_scan_totals(const unsigned* __restrict__ in,
                                                        long long n,
                                                        unsigned* __restrict__ bsum) {
  __shared__ unsigned s[SCAN_T / 32];
  unsigned t = 0;
#pragma unroll
  for (int v = 0; v < SCAN_V; v++) {
    const uint4 q = scan_load(in, scan_at(blockIdx.x, v), n);
    t += q.x + q.y + q.z + q.w;
  }
  t = __reduce_add_sync(0xffffffffu, t);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = t;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned a = 0;
    for (int w = 0; w < SCAN_T / 32; w++) a += s[w];
    bsum[blockIdx.x] = a;
  }
}

// Exclusive scan of the block totals by one CTA, chunk by chunk with a carry.
__global__ void __launch_bounds__(SUMS_T) k_scan_sums(unsigned* __restrict__ bsum, long long nb,
                                                      unsigned* __restrict__ total) {
  __shared__ unsigned s[SUMS_T / 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned carry = 0;
  for (long long base = 0; base < nb; base += SUMS_T) {
    const long long i = base + threadIdx.x;
    const unsigned v = i < nb ? bsum[i] : 0u;
    const unsigned inc = warp_scan(v);
    if (lane == 31) s[warp] = inc;
    __syncthreads();
    if (warp == 0) s[lane] = warp_scan(s[lane]);
    __syncthreads();
    if (i < nb) bsum[i] = carry + (warp ? s[warp - 1] : 0u) + inc - v;
    carry += s[SUMS_T / 32 - 1];
    __syncthreads();
  }
  if (threadIdx.x == 0 && total) *total = carry;
}

// Exclusive scan of a block from its start bsum (out may be in: a block's
// elements are read before they are written).
__global__ void __launch_bounds__(SCAN_T) k_scan_apply(const unsigned* in, unsigned* out,
                                                       long long n,
                                                       const unsigned* __restrict__ bsum) {
  __shared__ unsigned s[SCAN_T / 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint4 q[SCAN_V];
  unsigned before[SCAN_V], run = 0;
#pragma unroll
  for (int v = 0; v < SCAN_V; v++) q[v] = scan_load(in, scan_at(blockIdx.x, v), n);
#pragma unroll
  for (int v = 0; v < SCAN_V; v++) {
    const unsigned t = q[v].x + q[v].y + q[v].z + q[v].w;
    const unsigned inc = warp_scan(t);
    before[v] = run + inc - t;
    run += __shfl_sync(0xffffffffu, inc, 31);
  }
  if (lane == 0) s[warp] = run;
  __syncthreads();
  unsigned base = bsum[blockIdx.x];
  for (int w = 0; w < warp; w++) base += s[w];
#pragma unroll
  for (int v = 0; v < SCAN_V; v++) {
    const long long i = scan_at(blockIdx.x, v);
    uint4 o;
    o.x = base + before[v];
    o.y = o.x + q[v].x;
    o.z = o.y + q[v].y;
    o.w = o.z + q[v].z;
    if (i + 4 <= n) {
      *reinterpret_cast<uint4*>(out + i) = o;
    } else {
      if (i < n) out[i] = o.x;
      if (i + 1 < n) out[i + 1] = o.y;
      if (i + 2 < n) out[i + 2] = o.z;
    }
  }
}

}  // namespace

// Entries of block-sum scratch that exclusive() needs for n values.
inline long long scratch_entries(long long n) { return (n + SCAN_B - 1) / SCAN_B; }

// out[i] = in[0] + .. + in[i-1] (out may be in); bsum: scratch_entries(n)
// entries; *total (device, may be NULL) receives the sum.  in and out are
// 16-byte aligned.  Launches are counted under `stage`.
//
// Reduce, scan the totals, scan: two reads and one write of the counts, all in
// 16-byte vectors with the partial sums in registers (134M counts: 0.30 ms at
// the copy bandwidth against 1.5 ms for one element per thread, scanned in
// shared memory and corrected in a further pass).
inline void exclusive(const unsigned* in, unsigned* out, long long n, unsigned* bsum,
                      unsigned* total, int stage, cudaStream_t st) {
  const long long nb = scratch_entries(n);
  if (nb == 0) {
    if (total) cudaMemsetAsync(total, 0, sizeof(unsigned), st);
    return;
  }
  prof_mark(st, stage);
  k_scan_totals<<<(unsigned)nb, SCAN_T, 0, st>>>(in, n, bsum);
  prof_mark(st, stage);
  k_scan_sums<<<1, SUMS_T, 0, st>>>(bsum, nb, total);
  prof_mark(st, stage);
  k_scan_apply<<<(unsigned)nb, SCAN_T, 0, st>>>(in, out, n, bsum);
}

}  // namespace cgscan
