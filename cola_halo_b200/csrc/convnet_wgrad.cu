// Weight gradient of the 3x3x3 periodic convolution on tensor cores:
//   dW[t][ci][co] += sum_v in[v + off(t)][ci] g[v][co],   db[co] += sum_v g[v][co]
// with bf16 activations and float32 gradients, summed in float32.
//
// For one z run of up to 128 voxels of a line (x, y) this is, per tap, a
// 16 x 16 product over the run, D[ci][co] = A^T g with A the run of the tap's
// input line: m16n8k16 tensor-core products whose operands ldmatrix.trans
// reads in place, since both lie in shared memory as [z][channel] (two
// 8-channel halves of 16-byte rows: any 8 rows are conflict-free, and the z
// shift of a tap is a start one row on).
//
// g keeps its float32 value: it is split into three bf16 terms (8 + 8 + 8
// bits, each the rounded rest of the one before), which multiply the same
// bf16 activations exactly, so the products are those of the float32 sum.
// The leading term and the two small ones accumulate apart, and every run's
// sums are added to float32 totals in registers (round to nearest), so no
// tensor-core accumulation chain is longer than 16 products of 16.
//
// Nine warps, one per (dx, dy) input line, three dz taps each: the three taps
// share the g operands, 6 ldmatrix.x4 for 18 products.  A CTA walks runs of
// consecutive y: the three lines of a row sit in a ring of four slots, so a
// run loads one new row of three lines, by cp.async
// while the previous run multiplies.  2 CTAs per SM (80 KB, <= 112
// registers).  The last layer's gradient has three live channels of 16: its
// form (NT = 1) takes the eight columns that hold them.
//
// The first layer's input has two live channels: k_wgrad_in, below.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "convnet.h"

namespace {

constexpr int C = CNET_C;
constexpr int RUN = 128;                          // voxels of a run at most
constexpr int ROWS = RUN + 2;
constexpr int HALF_BYTES = ROWS * 16;
constexpr int LINE_BYTES = 2 * HALF_BYTES;
constexpr int RING_BYTES = 12 * LINE_BYTES;       // 4 rows of 3 lines
constexpr int G_BYTES = RUN * C * 4;              // one run of g, float32
constexpr int PLANE_BYTES = RUN * C * 2;          // one bf16 term of it
constexpr int SMEM_BYTES = RING_BYTES + 2 * G_BYTES + 3 * PLANE_BYTES;
constexpr int THREADS = 288;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void cp16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(dst), "l"(src) : "memory");
}

__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}

__device__ __forceinline__ void ldsm2t(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0, %1}, [%2];"
               : "=r"(r[0]), "=r"(r[1]) : "r"(a));
}

__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                    uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Row y (periodic) of the lines x-1, x, x+1, voxels z0 - 1 .. z0 + len, into a
// ring slot.
__device__ __forceinline__ void gather_row(const __nv_bfloat16* __restrict__ in, int N, int x,
                                           int y, int z0, int len, uint32_t slot) {
  y = y < 0 ? y + N : (y >= N ? y - N : y);
  const int rows = len + 2;
  for (int i = threadIdx.x; i < 6 * rows; i += THREADS) {
    const int h = i & 1, j = (i >> 1) % rows, l = (i >> 1) / rows;
    int xx = x + l - 1, zz = z0 + j - 1;
    xx = xx < 0 ? xx + N : (xx >= N ? xx - N : xx);
    zz = zz < 0 ? zz + N : (zz >= N ? zz - N : zz);
    cp16(slot + l * LINE_BYTES + h * HALF_BYTES + j * 16,
         in + (((size_t)xx * N + y) * N + zz) * C + h * 8);
  }
}

// Two gradients split into three bf16 pairs: the rounded value, the rounded
// rest, and what that leaves.
__device__ __forceinline__ void split2(float2 g, __nv_bfloat162 (&t)[3]) {
#pragma unroll
  for (int s = 0; s < 3; s++) {
    t[s] = __floats2bfloat162_rn(g.x, g.y);
    g.x -= __low2float(t[s]);
    g.y -= __high2float(t[s]);
  }
}

// A CTA's bias sums into db: each thread holds those of the channels 2 (tid %
// PAIRS), + 1; bred (shared) was set to zero.
template <int PAIRS>
__device__ __forceinline__ void add_bias(double2 bsum, float* bred, float* __restrict__ db) {
  const int lane = threadIdx.x & 31;
  __syncthreads();
#pragma unroll
  for (int o = PAIRS; o < 32; o <<= 1) {
    bsum.x += __shfl_xor_sync(0xffffffffu, bsum.x, o);
    bsum.y += __shfl_xor_sync(0xffffffffu, bsum.y, o);
  }
  if (lane < PAIRS) {
    atomicAdd(bred + 2 * lane, (float)bsum.x);
    atomicAdd(bred + 2 * lane + 1, (float)bsum.y);
  }
  __syncthreads();
  if (threadIdx.x < 2 * PAIRS) atomicAdd(db + threadIdx.x, bred[threadIdx.x]);
}

// NT: 8-channel halves of g that are not zero throughout (the first NT).
template <int NT>
__global__ void __launch_bounds__(THREADS, 2)
    k_conv_wgrad_tc(const __nv_bfloat16* __restrict__ in, const float* __restrict__ g, int N,
                    float* __restrict__ dw, float* __restrict__ db) {
  extern __shared__ __align__(128) uint8_t sm[];
  const uint32_t ring = smem_u32(sm);
  float* const stage = reinterpret_cast<float*>(sm + RING_BYTES);     // [2][RUN][C]
  uint8_t* const planes = sm + RING_BYTES + 2 * G_BYTES;              // [3][half][RUN] x 16 B
  const uint32_t pl = smem_u32(planes);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int lx = warp / 3, ly = warp % 3;          // this warp's input line (dx + 1, dy + 1)
  // ldmatrix row addresses: A's four 8x8 blocks are (half 0, z 0-7), (half 1,
  // z 0-7), (half 0, z 8-15), (half 1, z 8-15); B's (half 0, z 0-7), (half 0,
  // z 8-15), (half 1, z 0-7), (half 1, z 8-15)
  const uint32_t offA =
      (uint32_t)(((lane >> 3) & 1) * HALF_BYTES + ((lane & 7) + ((lane >> 4) & 1) * 8) * 16);
  const uint32_t offB = (uint32_t)(((lane >> 4) & 1) * (PLANE_BYTES / 2) +
                                   ((lane & 7) + ((lane >> 3) & 1) * 8) * 16);
  constexpr int PAIRS = 4 * NT;                    // channel pairs of a voxel of g
  float tot[3][NT][4];
#pragma unroll
  for (int d = 0; d < 3; d++)
#pragma unroll
    for (int h = 0; h < NT; h++)
#pragma unroll
      for (int q = 0; q < 4; q++) tot[d][h][q] = 0.0f;
  double2 bsum = make_double2(0.0, 0.0);           // channels 2 (tid % PAIRS), + 1
  __shared__ float bred[C];
  if (tid < C) bred[tid] = 0.0f;

  // runs in the order (x, z run, y); a CTA takes a contiguous range
  const int nz = (N + RUN - 1) / RUN;
  const int nruns = N * nz * N;
  const int per = (nruns + (int)gridDim.x - 1) / (int)gridDim.x;
  const int r1 = min(nruns, ((int)blockIdx.x + 1) * per);
  for (int r = (int)blockIdx.x * per; r < r1;) {
    const int y0 = r % N, z0 = (r / N) % nz * RUN, x = r / (N * nz);
    const int len = min(RUN, N - z0);              // a multiple of 16
    const int cnt = min(r1 - r, N - y0);           // runs of this (x, z0)
    const auto load_g = [&](int i) {
      const float* src = g + (((size_t)x * N + y0 + i) * N + z0) * C;
      const uint32_t dst = smem_u32(stage + (i & 1) * RUN * C);
      for (int k = tid; k < len * 2 * NT; k += THREADS) {
        const int at = NT == 2 ? k : (k >> 1) * 4 + (k & 1);
        cp16(dst + 16 * at, src + 4 * at);
      }
    };
    for (int j = 0; j < 3; j++)
      gather_row(in, N, x, y0 - 1 + j, z0, len, ring + j * 3 * LINE_BYTES);
    load_g(0);
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int i = 0; i < cnt; i++) {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      // rows i .. i+2 and this run's g are there, and every warp is done with
      // run i - 1: its row i - 1, the other stage and the planes are free
      __syncthreads();
      if (i + 1 < cnt) {
        gather_row(in, N, x, y0 + i + 2, z0, len, ring + ((i + 3) & 3) * 3 * LINE_BYTES);
        load_g(i + 1);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      const float2* sg = reinterpret_cast<const float2*>(stage + (i & 1) * RUN * C);
      float2 bs = make_float2(0.0f, 0.0f);
      for (int k = tid; k < len * PAIRS; k += THREADS) {
        const int z = NT == 2 ? k >> 3 : k >> 2, c = 2 * (k & (PAIRS - 1));
        const float2 v = sg[NT == 2 ? k : z * (C / 2) + c / 2];
        bs.x += v.x;
        bs.y += v.y;
        __nv_bfloat162 t[3];
        split2(v, t);
        uint8_t* d = planes + (c >> 3) * (PLANE_BYTES / 2) + z * 16 + (c & 7) * 2;
#pragma unroll
        for (int s = 0; s < 3; s++) *reinterpret_cast<__nv_bfloat162*>(d + s * PLANE_BYTES) = t[s];
      }
      bsum.x += bs.x;
      bsum.y += bs.y;
      __syncthreads();
      const uint32_t a0 = ring + (uint32_t)((((i + ly) & 3) * 3 + lx) * LINE_BYTES) + offA;
      float hi[3][NT][4], lo[3][NT][4];
#pragma unroll
      for (int d = 0; d < 3; d++)
#pragma unroll
        for (int h = 0; h < NT; h++)
#pragma unroll
          for (int q = 0; q < 4; q++) hi[d][h][q] = lo[d][h][q] = 0.0f;
#pragma unroll 1
      for (int z = 0; z < len; z += 16) {
        uint32_t a[3][4], b[4];
#pragma unroll
        for (int d = 0; d < 3; d++) ldsm4t(a[d], a0 + (uint32_t)((z + d) * 16));
#pragma unroll
        for (int s = 2; s >= 0; s--) {
          const uint32_t at = pl + (uint32_t)(s * PLANE_BYTES + z * 16) + offB;
          if (NT == 2) ldsm4t(b, at);
          else ldsm2t(b, at);
#pragma unroll
          for (int d = 0; d < 3; d++)
#pragma unroll
            for (int h = 0; h < NT; h++) mma(s ? lo[d][h] : hi[d][h], a[d], b[2 * h], b[2 * h + 1]);
        }
      }
#pragma unroll
      for (int d = 0; d < 3; d++)
#pragma unroll
        for (int h = 0; h < NT; h++)
#pragma unroll
          for (int q = 0; q < 4; q++) tot[d][h][q] += hi[d][h][q] + lo[d][h][q];
    }
    r += cnt;
    __syncthreads();                               // the ring is refilled for the next x
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  // accumulator q of a lane: ci = lane / 4 (+ 8 for q >= 2), co = 2 (lane % 4) + q % 2
#pragma unroll
  for (int d = 0; d < 3; d++)
#pragma unroll
    for (int h = 0; h < NT; h++)
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int ci = (lane >> 2) + (q >> 1) * 8, co = h * 8 + 2 * (lane & 3) + (q & 1);
        atomicAdd(dw + ((warp * 3 + d) * C + ci) * C + co, tot[d][h][q]);
      }
  // THREADS is a multiple of PAIRS, so a thread kept to one channel pair; the
  // CTA's sums meet in shared memory, then one atomic per channel
  add_bias<PAIRS>(bsum, bred, db);
}

// The first layer's weight gradient from the features as pairs.  The 27 taps'
// pairs of a voxel are gathered in shared memory into seven 16-byte groups of
// four taps (an eighth of zeros), as the forward first layer does, so that two
// groups are the 16 rows of a product: 4 products per 16 voxels, half of g and
// term where the 16-channel form does 27.  One warp per two groups; the next
// run's lines and gradients arrive by cp.async meanwhile.  128^3: 102 us,
// where the 16-channel form took 300; 182 us for the last layer's eight columns.
constexpr int IN_THREADS = 128;
constexpr int IN_LINE = (RUN + 8) * 4;             // z0 - 4 .. z0 + len + 3, 4 bytes a voxel
constexpr int IN_ROWS = 8 * RUN * 16;
constexpr int IN_CPS = 4;
constexpr int IN_SMEM = 2 * 9 * IN_LINE + 2 * G_BYTES + 3 * PLANE_BYTES + IN_ROWS;

__global__ void __launch_bounds__(IN_THREADS, IN_CPS)
    k_wgrad_in(const __nv_bfloat162* __restrict__ in, const float* __restrict__ g, int N,
               float* __restrict__ dw, float* __restrict__ db) {
  extern __shared__ __align__(128) uint8_t sm[];
  uint8_t* const lines = sm;                                          // [2][9] lines
  float* const stage = reinterpret_cast<float*>(lines + 2 * 9 * IN_LINE);   // [2][RUN][C]
  uint8_t* const planes = sm + 2 * 9 * IN_LINE + 2 * G_BYTES;         // [3][half][RUN] x 16 B
  uint8_t* const rows = planes + 3 * PLANE_BYTES;                     // [8 groups][RUN] x 16 B
  __shared__ float bred[C];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t offA = (uint32_t)((2 * warp + ((lane >> 3) & 1)) * (RUN * 16) +
                                   ((lane & 7) + ((lane >> 4) & 1) * 8) * 16);
  const uint32_t offB = (uint32_t)(((lane >> 4) & 1) * (PLANE_BYTES / 2) +
                                   ((lane & 7) + ((lane >> 3) & 1) * 8) * 16);
  const uint32_t a0 = smem_u32(rows) + offA, pl = smem_u32(planes) + offB;
  if (tid < C) bred[tid] = 0.0f;
  *reinterpret_cast<uint4*>(rows + 7 * RUN * 16 + tid * 16) = make_uint4(0, 0, 0, 0);
  float tot[2][4];
#pragma unroll
  for (int h = 0; h < 2; h++)
#pragma unroll
    for (int q = 0; q < 4; q++) tot[h][q] = 0.0f;
  double2 bsum = make_double2(0.0, 0.0);           // channels 2 (tid % 8), + 1

  const int nz = (N + RUN - 1) / RUN;
  const int nruns = N * nz * N;
  const auto load = [&](int r, int buf) {
    const int y = r % N, z0 = (r / N) % nz * RUN, x = r / (N * nz);
    const int len = min(RUN, N - z0), chunks = (len + 8) / 4;
    const uint32_t dst = smem_u32(lines + buf * 9 * IN_LINE);
    for (int i = tid; i < 9 * chunks; i += IN_THREADS) {
      const int l = i / chunks, q = i % chunks;
      int xx = x + l / 3 - 1, yy = y + l % 3 - 1, zz = z0 - 4 + 4 * q;
      xx = xx < 0 ? xx + N : (xx >= N ? xx - N : xx);
      yy = yy < 0 ? yy + N : (yy >= N ? yy - N : yy);
      zz = zz < 0 ? zz + N : (zz >= N ? zz - N : zz);
      cp16(dst + l * IN_LINE + q * 16, in + ((size_t)xx * N + yy) * N + zz);
    }
    const float* src = g + (((size_t)x * N + y) * N + z0) * C;
    const uint32_t gd = smem_u32(stage + buf * RUN * C);
    for (int k = tid; k < len * C / 4; k += IN_THREADS) cp16(gd + 16 * k, src + 4 * k);
  };
  const int per = (nruns + (int)gridDim.x - 1) / (int)gridDim.x;
  const int r0 = (int)blockIdx.x * per, r1 = min(nruns, r0 + per);
  if (r0 < r1) load(r0, 0);
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (int r = r0; r < r1; r++) {
    const int buf = (r - r0) & 1;
    const int len = min(RUN, N - (r / N) % nz * RUN);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    // this run is there, and every warp is done with the last one's rows and planes
    __syncthreads();
    if (r + 1 < r1) load(r + 1, buf ^ 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float2* sg = reinterpret_cast<const float2*>(stage + buf * RUN * C);
    float2 bs = make_float2(0.0f, 0.0f);
    for (int k = tid; k < len * C / 2; k += IN_THREADS) {
      const float2 v = sg[k];
      bs.x += v.x;
      bs.y += v.y;
      __nv_bfloat162 t[3];
      split2(v, t);
      const int z = k >> 3, c = 2 * (k & 7);
      uint8_t* d = planes + (c >> 3) * (PLANE_BYTES / 2) + z * 16 + (c & 7) * 2;
#pragma unroll
      for (int s = 0; s < 3; s++) *reinterpret_cast<__nv_bfloat162*>(d + s * PLANE_BYTES) = t[s];
    }
    bsum.x += bs.x;
    bsum.y += bs.y;
    if (tid < len) {
      const uint32_t* src =
          reinterpret_cast<const uint32_t*>(lines + buf * 9 * IN_LINE) + tid + 3;
#pragma unroll
      for (int q = 0; q < 7; q++) {
        uint32_t v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const int t = 4 * q + j;
          v[j] = t < 27 ? src[(t / 3) * (IN_LINE / 4) + t % 3] : 0u;
        }
        *reinterpret_cast<uint4*>(rows + q * (RUN * 16) + tid * 16) =
            make_uint4(v[0], v[1], v[2], v[3]);
      }
    }
    __syncthreads();
    float hi[2][4], lo[2][4];
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int q = 0; q < 4; q++) hi[h][q] = lo[h][q] = 0.0f;
#pragma unroll 2
    for (int z = 0; z < len; z += 16) {
      uint32_t a[4], b[4];
      ldsm4t(a, a0 + (uint32_t)(z * 16));
#pragma unroll
      for (int s = 2; s >= 0; s--) {
        ldsm4t(b, pl + (uint32_t)(s * PLANE_BYTES + z * 16));
#pragma unroll
        for (int h = 0; h < 2; h++) mma(s ? lo[h] : hi[h], a, b[2 * h], b[2 * h + 1]);
      }
    }
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int q = 0; q < 4; q++) tot[h][q] += hi[h][q] + lo[h][q];
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  // accumulator q of a lane: entry lane / 4 of group 2 warp (+ 1 for q >= 2),
  // which is tap 4 group + entry / 2, channel entry % 2
#pragma unroll
  for (int h = 0; h < 2; h++)
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int t = 4 * (2 * warp + (q >> 1)) + (lane >> 3), ci = (lane >> 2) & 1;
      const int co = h * 8 + 2 * (lane & 3) + (q & 1);
      if (t < 27) atomicAdd(dw + (t * C + ci) * C + co, tot[h][q]);
    }
  add_bias<8>(bsum, bred, db);
}

}  // namespace

cudaError_t conv_wgrad_set_smem() {
  constexpr auto kMax = cudaFuncAttributeMaxDynamicSharedMemorySize;
  cudaError_t e = cudaFuncSetAttribute(k_wgrad_in, kMax, IN_SMEM);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_conv_wgrad_tc<1>, kMax, SMEM_BYTES);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_conv_wgrad_tc<2>, kMax, SMEM_BYTES);
  return e;
}

cudaError_t conv_wgrad_in(const __nv_bfloat162* in, const float* g, int N, float* dw, float* db,
                          cudaStream_t st) {
  if (N % 16) return cudaErrorNotSupported;
  const int nruns = N * N * ((N + RUN - 1) / RUN), cap = IN_CPS * cg_sm_count();
  prof_mark(st, CG_ST_OTHER);
  k_wgrad_in<<<nruns < cap ? nruns : cap, IN_THREADS, IN_SMEM, st>>>(in, g, N, dw, db);
  return cudaGetLastError();
}

cudaError_t conv_wgrad_tc(const __nv_bfloat16* in, const float* g, int N, bool last, float* dw,
                          float* db, cudaStream_t st) {
  if (N % 16) return cudaErrorNotSupported;
  const int nruns = N * N * ((N + RUN - 1) / RUN);
  const int cap = 2 * cg_sm_count();
  prof_mark(st, CG_ST_OTHER);
  const auto kernel = last ? k_conv_wgrad_tc<1> : k_conv_wgrad_tc<2>;
  kernel<<<nruns < cap ? nruns : cap, THREADS, SMEM_BYTES, st>>>(in, g, N, dw, db);
  return cudaGetLastError();
}
