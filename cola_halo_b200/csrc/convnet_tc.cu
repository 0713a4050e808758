// 3x3x3 periodic convolution, 16 -> 16 channels, bf16 x bf16 -> fp32, on the
// fifth-generation tensor cores (tcgen05.mma, accumulator in tensor memory).
//
// Implicit GEMM per tile of 128 consecutive z voxels of one (x, y) line:
//   D[128 voxels][16 co] = sum over 27 taps of A_t[128][16 ci] . B_t[16 ci][16 co]
// The 27 taps read only 9 input lines -- the (x +- 1, y +- 1) neighbours --
// each over z0 - 1 .. z0 + 128.  A CTA copies those 9 lines (130 rows of
// 32 bytes) into shared memory once, in a row-contiguous K-major layout:
// per line, the 8-channel half h of row j sits at h * 2080 + j * 16 bytes.
// Read with core-matrix strides SBO = 128 B (8-row groups) and LBO = 2080 B
// (the two 8-channel halves), the operand of tap (dx, dy, dz) is the same
// buffer started dz rows further on: the z shift costs no copy.  B_t are the
// tap weights in the no-swizzle core-matrix layout (LBO 128 B, SBO 256 B).
//
// k_conv_sweep, the default, reuses the lines along x (below).  In k_conv_tc
// CTAs are persistent over tiles, 4 per SM with one line buffer each: one
// thread issues the tile's 27 MMAs (M=128, N=16, K=16), tcgen05.commit
// arrives on an mbarrier, the cp.async gather of the next tile starts, and
// the four warps read their 32 accumulator lanes with tcgen05.ld for bias +
// activation while it runs.  (A two-buffer form, 2 CTAs per SM, prefetches
// during the MMAs instead.)  Every mbarrier wait is bounded and reports through an error
// word; on a timeout the CTA drains its copies, frees its tensor memory and
// returns.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>

#include "convnet.h"

namespace {

constexpr int C = CNET_C;
constexpr int TILE_M = 128;
constexpr int ROWS = TILE_M + 2;                 // z0 - 1 .. z0 + 128
constexpr int HALF_BYTES = ROWS * 16;            // 2080: one 8-channel half of a line
constexpr int LINE_BYTES = 2 * HALF_BYTES;       // 4160
constexpr int STAGE_BYTES = 9 * LINE_BYTES;      // 37440: the 9 neighbour lines
constexpr int B_BYTES = C * C * 2;               // 512: one tap's B operand
constexpr int THREADS = 128;
__host__ __device__ constexpr int smem_bytes(int stages) {
  return stages * STAGE_BYTES + 27 * B_BYTES + 64;
}
constexpr long long kWaitLimit = 1LL << 24;

__device__ unsigned g_tc_err = 0;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// Shared-memory matrix descriptor: no swizzle, K-major, version 1.  LBO is
// the byte offset between the core matrices of the two K halves, SBO the
// offset between 8-row groups; the start address is 16-byte aligned.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr & 0x3FFFF) >> 4) | ((uint64_t)(lbo >> 4) << 16) |
         ((uint64_t)(sbo >> 4) << 32) | (1ULL << 46);
}

// Instruction descriptor, kind::f16: D f32, A bf16, B bf16, both K-major,
// N = 16, M = 128.
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((16u >> 3) << 17) |
                            ((128u >> 4) << 24);

// offset of element (row, k) of a [rows][16] bf16 operand in core-matrix layout
__device__ __forceinline__ int cm_off(int row, int k) {
  return (((row >> 3) * 2 + (k >> 3)) << 7) + ((row & 7) << 4) + ((k & 7) << 1);
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t phase) {
  for (long long i = 0; i < kWaitLimit; i++) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(bar), "r"(phase)
        : "memory");
    if (done) return true;
  }
  return false;
}

// cp.async of the 9 neighbour lines of tile `tile` into stage buffer `st`:
// element (line L, row j, half h) <- voxel (x + L/3 - 1, y + L%3 - 1,
// z0 - 1 + j), channels 8h .. 8h+7 (periodic).
__device__ __forceinline__ void gather(const __nv_bfloat16* __restrict__ in, int N, int tile,
                                       uint8_t* stage) {
  const int tiles_per_line = N / TILE_M;
  const int line = tile / tiles_per_line;
  const int z0 = (tile % tiles_per_line) * TILE_M;
  const int x = line / N, y = line % N;
  for (int i = threadIdx.x; i < 9 * ROWS * 2; i += THREADS) {
    const int h = i & 1, j = (i >> 1) % ROWS, L = (i >> 1) / ROWS;
    int xx = x + L / 3 - 1, yy = y + L % 3 - 1, zz = z0 - 1 + j;
    xx = xx < 0 ? xx + N : (xx >= N ? xx - N : xx);
    yy = yy < 0 ? yy + N : (yy >= N ? yy - N : yy);
    zz = zz < 0 ? zz + N : (zz >= N ? zz - N : zz);
    const __nv_bfloat16* src = in + (((size_t)xx * N + yy) * N + zz) * C + h * 8;
    const uint32_t dst = smem_u32(stage + L * LINE_BYTES + h * HALF_BYTES + j * 16);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(dst), "l"(src) : "memory");
  }
}

// STAGES = 2: the next tile's gather runs during this tile's MMAs (2 CTAs
// per SM fit).  STAGES = 1: the next gather starts once this tile's MMAs
// are done and runs during its epilogue (4 CTAs per SM fit).
template <bool FLIP, int STAGES, int CPS>
__global__ void __launch_bounds__(THREADS, CPS)
    k_conv_tc(const __nv_bfloat16* __restrict__ in, int N, const __nv_bfloat16* __restrict__ w,
              const float* __restrict__ bias, int act, const __nv_bfloat16* __restrict__ gate,
              float* __restrict__ out_f, __nv_bfloat16* __restrict__ out_b,
              float4* __restrict__ out4) {
  extern __shared__ __align__(1024) uint8_t sm[];
  uint8_t* const stage0 = sm;
  uint8_t* const stage1 = sm + (STAGES - 1) * STAGE_BYTES;
  uint8_t* sB = sm + STAGES * STAGE_BYTES;
  uint64_t* mbar = reinterpret_cast<uint64_t*>(sB + 27 * B_BYTES);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(mbar + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(smem_u32(tslot)), "r"(32) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(mbar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // B_t: element (n = output channel, k = input channel) of tap t
  for (int i = tid; i < 27 * C * C; i += THREADS) {
    const int t = i / (C * C), n = (i / C) % C, k = i % C;
    const __nv_bfloat16 v = FLIP ? w[((26 - t) * C + n) * C + k]   // W[26-t][ci=n][co=k]
                                 : w[(t * C + k) * C + n];         // W[t][ci=k][co=n]
    *reinterpret_cast<__nv_bfloat16*>(sB + t * B_BYTES + cm_off(n, k)) = v;
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tslot;
  const uint32_t bar = smem_u32(mbar);
  const int tiles_per_line = N / TILE_M;
  const int ntiles = N * N * tiles_per_line;
  uint32_t phase = 0;
  bool ok = true;

  int tile = blockIdx.x;
  if (tile < ntiles) gather(in, N, tile, stage0);
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (int it = 0; tile < ntiles && ok; tile += gridDim.x, it++) {
    const int next = tile + gridDim.x;
    const uint8_t* s = (it & 1) ? stage1 : stage0;
    if (STAGES == 2) {
      // the next tile's lines load while this tile multiplies; that buffer's
      // previous MMAs completed before the last iteration's epilogue
      if (next < ntiles) gather(in, N, next, (it & 1) ? stage0 : stage1);
      asm volatile("cp.async.commit_group;" ::: "memory");
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (tid == 0) {
      for (int t = 0; t < 27; t++) {
        // tap (dx, dy, dz): line t / 3, started dz = t % 3 rows on
        const uint64_t da =
            umma_desc(smem_u32(s + (t / 3) * LINE_BYTES + (t % 3) * 16), HALF_BYTES, 128);
        const uint64_t db = umma_desc(smem_u32(sB + t * B_BYTES), 128, 256);
        const uint32_t acc = t > 0 ? 1u : 0u;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
            :: "r"(tmem), "l"(da), "l"(db), "r"(kIdesc), "r"(acc)
            : "memory");
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                   :: "r"(bar) : "memory");
    }
    // every thread waits (bounded); the CTA agrees on the outcome so that all
    // threads take the same path through the barriers below
    const bool got = mbar_wait(bar, phase);
    ok = __syncthreads_and(got ? 1 : 0) != 0;
    if (!ok && tid == 0) atomicOr(&g_tc_err, 1u);
    phase ^= 1u;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (STAGES == 1) {
      // the MMAs have read the buffer: the next tile's lines load during
      // this tile's epilogue
      if (ok && next < ntiles) gather(in, N, next, stage0);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    if (ok) {
      const int line = tile / tiles_per_line;
      const int z0 = (tile % tiles_per_line) * TILE_M;
      uint32_t r[16];
      const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16);
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
          "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
          : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
            "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
            "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
          : "r"(taddr));
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      const size_t v = (size_t)line * N + z0 + warp * 32 + lane;
      float o[C];
#pragma unroll
      for (int c = 0; c < C; c++) {
        float a = __uint_as_float(r[c]) + (bias ? bias[c] : 0.0f);
        if (act) a = a > 0.0f ? a : 0.1f * a;
        if (gate && __bfloat162float(gate[v * C + c]) <= 0.0f) a *= 0.1f;
        o[c] = a;
      }
      if (out_f) {
        float4* d = reinterpret_cast<float4*>(out_f + v * C);
#pragma unroll
        for (int q = 0; q < 4; q++)
          d[q] = make_float4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
      }
      if (out_b) {
        __nv_bfloat16 hb[C];
#pragma unroll
        for (int c = 0; c < C; c++) hb[c] = __float2bfloat16_rn(o[c]);
        uint4* d = reinterpret_cast<uint4*>(out_b + v * C);
        d[0] = *reinterpret_cast<const uint4*>(&hb[0]);
        d[1] = *reinterpret_cast<const uint4*>(&hb[8]);
      }
      if (out4) out4[v] = make_float4(o[0], o[1], o[2], o[3]);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
  }
  // copies still in flight (a prefetch after a timeout) finish before exit
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(32)
                 : "memory");
}

// The same convolution, sweeping along x with every input row used once.  A
// CTA owns the z tiles (x, y0, z0) and (x, y0 + 1, z0) for a run of x.  Input
// row x' (the four lines y0-1 .. y0+2) adds to the outputs of rows x'-1, x'
// and x'+1 at once: one MMA of M = 128 voxels, N = 48 columns (the three
// rows' 16 output channels, with the weights of dx = +1, 0, -1) and K = 16
// per output line, dy and dz.  So the A operand (128 rows of 32 bytes from
// shared memory) is read 9 times per output line where one tile at a time
// (N = 16) reads it 27 times, and the lines come from L2 twice per output line
// instead of nine times.  128^3: 79-90 us a layer under ncu.  The operand reads
// (32 clocks each) come to about 19 us of that and the layer's bytes to 20; the
// rest is the chain of a row: wait for its copy, issue, commit, wait, drain,
// zero, barrier, which four CTAs per SM overlap in part (tensor pipe active 20 %
// of the time).
//
// The three accumulators of an output column y sit in tensor-memory slots o
// mod 3 (o the output row counted from the run's start).  The rows x'-1, x',
// x'+1 take every slot once, in a cyclic order that moves by one per row, so
// the B operand of a tap pair (dy, dz) is stored as five blocks of 16 channels, dx
// = +1, 0, -1, +1, 0, and the row's window of three starts at block 2, 1 or 0.
// After a row's MMAs the slot of output o = i - 2 (i the row) is complete: its
// threads read it, set it to zero for output o + 3 and hand the tensor memory
// back; bias, activation and stores then run beside the next row's MMAs.  The
// next row's lines arrive by cp.async meanwhile.  4 CTAs per SM (57 KB, 128
// tensor-memory columns each).
//
// Per output the products are added in the order dx, dy, dz, as in k_conv_tc:
// bit-identical.  (A sweep along y is as fast but adds in another order.)
constexpr int SROW_BYTES = 4 * LINE_BYTES;       // four lines of one input row
constexpr int SB_BYTES = 5 * B_BYTES;            // five 16-channel blocks per (dy, dz)
constexpr int SLOTS = 3;
__host__ __device__ constexpr int sweep_smem_bytes() {
  return 2 * SROW_BYTES + 9 * SB_BYTES + 64;
}
constexpr int SWEEP_CPS = 4;
constexpr uint32_t kIdesc48 = (kIdesc & ~(0x3Fu << 17)) | ((48u >> 3) << 17);

// cp.async of row x (periodic) of the lines y0-1 .. y0+2, voxels z0 - 1 ..
// z0 + 128, into a row buffer.
__device__ __forceinline__ void gather_row(const __nv_bfloat16* __restrict__ in, int N, int y0,
                                           int x, int z0, uint8_t* row) {
  x = x < 0 ? x + N : (x >= N ? x - N : x);
  for (int i = threadIdx.x; i < 4 * ROWS * 2; i += THREADS) {
    const int h = i & 1, j = (i >> 1) % ROWS, L = (i >> 1) / ROWS;
    int yy = y0 + L - 1, zz = z0 + j - 1;
    yy = yy < 0 ? yy + N : (yy >= N ? yy - N : yy);
    zz = zz < 0 ? zz + N : (zz >= N ? zz - N : zz);
    const __nv_bfloat16* src = in + (((size_t)x * N + yy) * N + zz) * C + h * 8;
    const uint32_t dst = smem_u32(row + L * LINE_BYTES + h * HALF_BYTES + j * 16);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(dst), "l"(src) : "memory");
  }
}

// 16 accumulator columns of this warp's 32 lanes.
__device__ __forceinline__ void tmem_ld16(uint32_t (&r)[16], uint32_t a) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(a));
}
__device__ __forceinline__ void tmem_zero16(uint32_t a) {
  const uint32_t z = 0;
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1};"
      :: "r"(a), "r"(z) : "memory");
}

// Bias, activation or gate, and the stores of one voxel's 16 channels.
__device__ __forceinline__ void store_voxel(const uint32_t (&r)[16], size_t v,
                                            const float* __restrict__ bias, int act,
                                            const __nv_bfloat16* __restrict__ gate,
                                            float* __restrict__ out_f,
                                            __nv_bfloat16* __restrict__ out_b,
                                            float4* __restrict__ out4) {
  float o[C];
#pragma unroll
  for (int c = 0; c < C; c++) {
    float a = __uint_as_float(r[c]) + (bias ? bias[c] : 0.0f);
    if (act) a = a > 0.0f ? a : 0.1f * a;
    o[c] = a;
  }
  if (gate) {
    uint4 gq[2] = {reinterpret_cast<const uint4*>(gate + v * C)[0],
                   reinterpret_cast<const uint4*>(gate + v * C)[1]};
    const __nv_bfloat16* gv = reinterpret_cast<const __nv_bfloat16*>(gq);
#pragma unroll
    for (int c = 0; c < C; c++)
      if (__bfloat162float(gv[c]) <= 0.0f) o[c] *= 0.1f;
  }
  if (out_f) {
    float4* d = reinterpret_cast<float4*>(out_f + v * C);
#pragma unroll
    for (int q = 0; q < 4; q++)
      d[q] = make_float4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
  }
  if (out_b) {
    __nv_bfloat16 hb[C];
#pragma unroll
    for (int c = 0; c < C; c++) hb[c] = __float2bfloat16_rn(o[c]);
    uint4* d = reinterpret_cast<uint4*>(out_b + v * C);
    d[0] = *reinterpret_cast<const uint4*>(&hb[0]);
    d[1] = *reinterpret_cast<const uint4*>(&hb[8]);
  }
  if (out4) out4[v] = make_float4(o[0], o[1], o[2], o[3]);
}

template <bool FLIP>
__global__ void __launch_bounds__(THREADS, SWEEP_CPS)
    k_conv_sweep(const __nv_bfloat16* __restrict__ in, int N, const __nv_bfloat16* __restrict__ w,
                 const float* __restrict__ bias, int act, const __nv_bfloat16* __restrict__ gate,
                 float* __restrict__ out_f, __nv_bfloat16* __restrict__ out_b,
                 float4* __restrict__ out4) {
  extern __shared__ __align__(1024) uint8_t sm[];
  uint8_t* sB = sm + 2 * SROW_BYTES;
  uint64_t* mbar = reinterpret_cast<uint64_t*>(sB + 9 * SB_BYTES);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(mbar + 1);
  const int tid = threadIdx.x, warp = tid >> 5;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(smem_u32(tslot)), "r"(128) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(mbar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // B of (dy, dz): blocks dx = +1, 0, -1, +1, 0; element (n = output channel,
  // k = input channel) of tap t
  for (int i = tid; i < 9 * 5 * C * C; i += THREADS) {
    const int k = i % C, n = i / C % C, b = i / (C * C) % 5, p = i / (5 * C * C);
    const int t = (2 - b % 3) * 9 + p;
    const __nv_bfloat16 v = FLIP ? w[((26 - t) * C + n) * C + k] : w[(t * C + k) * C + n];
    *reinterpret_cast<__nv_bfloat16*>(sB + p * SB_BYTES + cm_off(b * C + n, k)) = v;
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tslot;
  const uint32_t mine = tmem + ((uint32_t)(warp * 32) << 16);
  const uint32_t bar = smem_u32(mbar);
  // output rows in the order (y pair, z tile, x); a CTA takes a contiguous range
  const int nz = N / TILE_M;
  const int nrows = N / 2 * nz * N;
  const int per = (nrows + (int)gridDim.x - 1) / (int)gridDim.x;
  const int l1 = min(nrows, ((int)blockIdx.x + 1) * per);
  uint32_t phase = 0;
  bool ok = true;
  for (int l = (int)blockIdx.x * per; l < l1 && ok;) {
    const int x0 = l % N, z0 = (l / N) % nz * TILE_M, y0 = l / (N * nz) * 2;
    const int run = min(l1 - l, N - x0);
    gather_row(in, N, y0, x0 - 1, z0, sm);
    asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
    for (int q = 0; q < 2 * SLOTS; q++) tmem_zero16(mine + 16 * q);
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    uint32_t r[2][16];
    // row i holds x' = x0 - 1 + i
    for (int i = 0; i <= run + 1 && ok; i++) {
      // the other buffer's row i - 1 has been multiplied
      if (i <= run) gather_row(in, N, y0, x0 + i, z0, sm + ((i + 1) & 1) * SROW_BYTES);
      asm volatile("cp.async.commit_group;" ::: "memory");
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncthreads();
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (tid == 0) {
        const uint32_t row = smem_u32(sm + (i & 1) * SROW_BYTES);
        const uint32_t b0 = smem_u32(sB) + (uint32_t)((2 - i % 3) * B_BYTES);
        for (int yo = 0; yo < 2; yo++) {
          for (int p = 0; p < 9; p++) {
            // (dy, dz) = (p / 3, p % 3): line yo + dy, started dz rows on
            const uint64_t da = umma_desc(
                row + (uint32_t)((yo + p / 3) * LINE_BYTES + (p % 3) * 16), HALF_BYTES, 128);
            const uint64_t db = umma_desc(b0 + (uint32_t)(p * SB_BYTES), 128, 256);
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "setp.ne.b32 p, %4, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
                :: "r"(tmem + (uint32_t)(16 * SLOTS * yo)), "l"(da), "l"(db), "r"(kIdesc48),
                   "r"(1u)
                : "memory");
          }
        }
        asm volatile(
            "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
            :: "r"(bar) : "memory");
      }
      // the output that row i - 1 completed, beside this row's MMAs
      if (i >= 3) {
        const size_t v = ((size_t)(x0 + i - 3) * N + y0) * N + z0 + tid;
        store_voxel(r[0], v, bias, act, gate, out_f, out_b, out4);
        store_voxel(r[1], v + N, bias, act, gate, out_f, out_b, out4);
      }
      const bool got = mbar_wait(bar, phase);
      ok = __syncthreads_and(got ? 1 : 0) != 0;
      if (!ok && tid == 0) atomicOr(&g_tc_err, 1u);
      phase ^= 1u;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t slot = mine + (uint32_t)(16 * ((i + 1) % SLOTS));
      tmem_ld16(r[0], slot);
      tmem_ld16(r[1], slot + 16 * SLOTS);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      tmem_zero16(slot);
      tmem_zero16(slot + 16 * SLOTS);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    if (ok) {
      const size_t v = ((size_t)(x0 + run - 1) * N + y0) * N + z0 + tid;
      store_voxel(r[0], v, bias, act, gate, out_f, out_b, out4);
      store_voxel(r[1], v + N, bias, act, gate, out_f, out_b, out4);
    }
    // every copy has landed and every MMA has completed: the buffers are free
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    l += run;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(128)
                 : "memory");
}

template <bool FLIP>
cudaError_t launch_sweep(const __nv_bfloat16* in, int N, const __nv_bfloat16* w,
                         const float* bias, int act, const __nv_bfloat16* gate, float* of,
                         __nv_bfloat16* ob, float4* o4, cudaStream_t st) {
  const int nrows = N / 2 * (N / TILE_M) * N;
  const int cap = SWEEP_CPS * cg_sm_count();
  prof_mark(st, CG_ST_OTHER);
  k_conv_sweep<FLIP><<<nrows < cap ? nrows : cap, THREADS, sweep_smem_bytes(), st>>>(
      in, N, w, bias, act, gate, of, ob, o4);
  return cudaGetLastError();
}

// The first layer, whose input has two live channels (density, potential):
// the 27 taps' pairs of one voxel are gathered into one row of 54 + 10 zeros, so
// a tile of 128 voxels is 4 MMAs of K = 16 on a 128 x 64 operand where the
// 16-channel layout needs 27 (9 in the sweep) of mostly zeros; and the features
// take 4 bytes a voxel instead of 32.  Thread r copies voxel r's 27 words from
// the nine input lines in shared memory (consecutive lanes, consecutive words)
// into seven 16-byte groups of four taps, K-major: group g of row r sits at g *
// 2048 + r * 16.  The next tile's lines arrive by cp.async meanwhile.
constexpr int IN_LINE = (TILE_M + 8) * 4;        // z0 - 4 .. z0 + 131, 4 bytes a voxel
constexpr int IN_LINES = 9 * IN_LINE;
constexpr int IN_A = 8 * TILE_M * 16;            // 64 K values
constexpr int IN_B = 8 * C * 16;
constexpr int IN_CPS = 6;
constexpr int in_smem_bytes() { return 2 * IN_LINES + IN_A + IN_B + 64; }

__device__ __forceinline__ void gather_in(const __nv_bfloat162* __restrict__ in, int N, int tile,
                                          uint8_t* dst) {
  const int per_line = N / TILE_M;
  const int line = tile / per_line, z0 = tile % per_line * TILE_M;
  const int x = line / N, y = line % N;
  for (int i = threadIdx.x; i < 9 * (IN_LINE / 16); i += THREADS) {
    const int L = i / (IN_LINE / 16), q = i % (IN_LINE / 16);
    int xx = x + L / 3 - 1, yy = y + L % 3 - 1, zz = z0 - 4 + 4 * q;
    xx = xx < 0 ? xx + N : (xx >= N ? xx - N : xx);
    yy = yy < 0 ? yy + N : (yy >= N ? yy - N : yy);
    zz = zz < 0 ? zz + N : (zz >= N ? zz - N : zz);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                 :: "r"(smem_u32(dst + L * IN_LINE + q * 16)),
                    "l"(in + ((size_t)xx * N + yy) * N + zz) : "memory");
  }
}

__global__ void __launch_bounds__(THREADS, IN_CPS)
    k_conv_in(const __nv_bfloat162* __restrict__ in, int N, const __nv_bfloat16* __restrict__ w,
              const float* __restrict__ bias, int act, __nv_bfloat16* __restrict__ out_b) {
  extern __shared__ __align__(1024) uint8_t sm[];
  uint8_t* const sA = sm;
  uint8_t* const sB = sA + IN_A;
  uint8_t* const lines = sB + IN_B;
  uint64_t* mbar = reinterpret_cast<uint64_t*>(lines + 2 * IN_LINES);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(mbar + 1);
  const int tid = threadIdx.x, warp = tid >> 5;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(smem_u32(tslot)), "r"(32) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(mbar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // B: element (n = output channel, k = 2 tap + input channel); zeros past tap 26
  for (int i = tid; i < 64 * C; i += THREADS) {
    const int n = i / 64, k = i % 64;
    const __nv_bfloat16 v =
        k < 54 ? w[(k / 2 * C + k % 2) * C + n] : __float2bfloat16_rn(0.0f);
    *reinterpret_cast<__nv_bfloat16*>(sB + (k / 8) * (C * 16) + n * 16 + (k % 8) * 2) = v;
  }
  *reinterpret_cast<uint4*>(sA + 7 * TILE_M * 16 + tid * 16) = make_uint4(0, 0, 0, 0);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tslot;
  const uint32_t bar = smem_u32(mbar);
  const int ntiles = N * N * (N / TILE_M);
  uint32_t phase = 0;
  bool ok = true;
  int tile = blockIdx.x;
  if (tile < ntiles) gather_in(in, N, tile, lines);
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (int it = 0; tile < ntiles && ok; tile += gridDim.x, it++) {
    const int next = tile + gridDim.x;
    // the other line buffer was read before the last tile's MMAs
    if (next < ntiles) gather_in(in, N, next, lines + ((it + 1) & 1) * IN_LINES);
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    const uint32_t* src = reinterpret_cast<const uint32_t*>(lines + (it & 1) * IN_LINES) + tid + 3;
#pragma unroll
    for (int g = 0; g < 7; g++) {
      uint32_t q[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int t = 4 * g + j;
        q[j] = t < 27 ? src[(t / 3) * (IN_LINE / 4) + t % 3] : 0u;
      }
      *reinterpret_cast<uint4*>(sA + g * (TILE_M * 16) + tid * 16) =
          make_uint4(q[0], q[1], q[2], q[3]);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (tid == 0) {
      for (int k = 0; k < 4; k++) {
        const uint64_t da = umma_desc(smem_u32(sA) + (uint32_t)(2 * k * TILE_M * 16),
                                      TILE_M * 16, 128);
        const uint64_t db = umma_desc(smem_u32(sB) + (uint32_t)(2 * k * C * 16), C * 16, 128);
        const uint32_t acc = k > 0 ? 1u : 0u;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
            :: "r"(tmem), "l"(da), "l"(db), "r"(kIdesc), "r"(acc)
            : "memory");
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                   :: "r"(bar) : "memory");
    }
    const bool got = mbar_wait(bar, phase);
    ok = __syncthreads_and(got ? 1 : 0) != 0;
    if (!ok && tid == 0) atomicOr(&g_tc_err, 1u);
    phase ^= 1u;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (ok) {
      const int per_line = N / TILE_M;
      uint32_t r[16];
      tmem_ld16(r, tmem + ((uint32_t)(warp * 32) << 16));
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      store_voxel(r, (size_t)(tile / per_line) * N + tile % per_line * TILE_M + tid, bias, act,
                  nullptr, nullptr, out_b, nullptr);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  // copies still in flight (a prefetch after a timeout) finish before exit
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(32)
                 : "memory");
}

template <bool FLIP, int STAGES, int CPS>
cudaError_t launch_v(const __nv_bfloat16* in, int N, const __nv_bfloat16* w, const float* bias,
                     int act, const __nv_bfloat16* gate, float* of, __nv_bfloat16* ob, float4* o4, cudaStream_t st) {
  const int ntiles = N * N * (N / TILE_M);
  const int sms = cg_sm_count();
  const int grid = ntiles < CPS * sms ? ntiles : CPS * sms;
  prof_mark(st, CG_ST_OTHER);
  k_conv_tc<FLIP, STAGES, CPS><<<grid, THREADS, smem_bytes(STAGES), st>>>(in, N, w, bias, act,
                                                                         gate, of, ob, o4);
  return cudaGetLastError();
}

// pipeline variant: 2 (the default) = the sweep along x (k_conv_sweep); 1 =
// one tile at a time, one stage, 4 CTAs/SM; 0 = two stages, 2 CTAs/SM.
// COLAGPU_CONV_VARIANT=0/1/2 selects one.
int g_conv_variant = -1;      // conv_tc_set_variant

int conv_variant() {
  static const int forced = [] {
    const char* e = getenv("COLAGPU_CONV_VARIANT");
    return e ? atoi(e) : -1;
  }();
  const int v = forced >= 0 ? forced : g_conv_variant;
  return v == 0 || v == 1 ? v : 2;
}

template <bool FLIP>
cudaError_t launch(const __nv_bfloat16* in, int N, const __nv_bfloat16* w, const float* bias,
                   int act, const __nv_bfloat16* gate, float* of, __nv_bfloat16* ob, float4* o4, cudaStream_t st) {
  if (N < TILE_M || N % TILE_M) return cudaErrorNotSupported;
  const int v = conv_variant();
  if (v == 2) return launch_sweep<FLIP>(in, N, w, bias, act, gate, of, ob, o4, st);
  if (v == 1) return launch_v<FLIP, 1, 4>(in, N, w, bias, act, gate, of, ob, o4, st);
  return launch_v<FLIP, 2, 2>(in, N, w, bias, act, gate, of, ob, o4, st);
}

// The kernels of one direction.
template <bool FLIP>
cudaError_t set_smem() {
  constexpr auto kMax = cudaFuncAttributeMaxDynamicSharedMemorySize;
  cudaError_t e = cudaFuncSetAttribute(k_conv_sweep<FLIP>, kMax, sweep_smem_bytes());
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_conv_tc<FLIP, 1, 4>, kMax, smem_bytes(1));
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_conv_tc<FLIP, 2, 2>, kMax, smem_bytes(2));
  return e;
}

}  // namespace

cudaError_t conv_tc_set_smem() {
  cudaError_t e = cudaFuncSetAttribute(k_conv_in, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       in_smem_bytes());
  if (e == cudaSuccess) e = set_smem<false>();
  if (e == cudaSuccess) e = set_smem<true>();
  return e;
}

cudaError_t conv_tc_forward(const __nv_bfloat16* in, int N, const __nv_bfloat16* w,
                            const float* bias, int act, float* out_f, __nv_bfloat16* out_b,
                            float4* out4, cudaStream_t st) {
  return launch<false>(in, N, w, bias, act, nullptr, out_f, out_b, out4, st);
}

cudaError_t conv_tc_features(const __nv_bfloat162* in, int N, const __nv_bfloat16* w,
                             const float* bias, int act, __nv_bfloat16* out_b, cudaStream_t st) {
  if (N < TILE_M || N % TILE_M) return cudaErrorNotSupported;
  const int ntiles = N * N * (N / TILE_M), cap = IN_CPS * cg_sm_count();
  prof_mark(st, CG_ST_OTHER);
  k_conv_in<<<ntiles < cap ? ntiles : cap, THREADS, in_smem_bytes(), st>>>(in, N, w, bias, act,
                                                                          out_b);
  return cudaGetLastError();
}

cudaError_t conv_tc_backward_data(const __nv_bfloat16* g, int N, const __nv_bfloat16* w,
                                  const __nv_bfloat16* gate, float* out_f, __nv_bfloat16* out_b,
                                  cudaStream_t st) {
  return launch<true>(g, N, w, nullptr, 0, gate, out_f, out_b, nullptr, st);
}

int conv_tc_set_variant(int v) {
  return v >= -1 && v <= 2 ? (g_conv_variant = v, 0) : -1;
}

unsigned conv_tc_error_word() {
  unsigned v = 0;
  cudaMemcpyFromSymbol(&v, g_tc_err, sizeof(v));
  return v;
}
