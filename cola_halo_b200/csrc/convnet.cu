// Learned small-scale force correction (no reference counterpart).
//
// A coarse PM mesh (factor 1) loses force at the mesh scale.  A three-layer
// 3x3x3 periodic convolutional net on the coarse mesh maps
//   input  (2 ch):  CIC density contrast delta, potential phi (lap phi = delta)
//   hidden (16 ch): leaky-ReLU(0.1)
//   output (3 ch):  force residual, added to the coarse PM force after CIC
//                   interpolation to the particles
// and is trained on pairs generated by the PM method itself: the residual
// target is the factor-3 (fine) PM force minus the coarse PM force at the
// same particles, CIC-deposited onto the coarse mesh and divided by the
// deposited mass.  Loss: mass-weighted mean squared error on the mesh.
//
// Storage: activations channels-last [x][y][z][16] in bf16 (16 channels =
// 32 B per voxel; unused channels are zero), weights W[tap][ci][co] in bf16
// with float32 master copies and Adam moments, float32 accumulation.
// The convolution has two implementations selected at run time:
//   * k_conv_tc: tcgen05 tensor cores (convnet_tc.cu), the default
//   * k_conv_simt: CUDA cores, used as the device-side cross-check
// Backward: data gradient = the same convolution with flipped taps and
// transposed channels; weight gradient = tensor-core products per voxel line
// (convnet_wgrad.cu), register totals per CTA, one float atomic per weight
// per CTA (k_conv_wgrad: the same on CUDA cores, with k_conv_simt).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <vector>

#include "../../include/colagpu.h"
#include "convnet.h"
#include "internal.h"

extern int cg_set_error_from_lpt(int code, const char* msg);

namespace {

constexpr int T = CG_THREADS;
constexpr int C = CNET_C;           // 16 channels
constexpr int NT = 27;              // taps
constexpr int WSZ = NT * C * C;     // weights per layer

__device__ __forceinline__ int wrapi(int i, int N) { return i < 0 ? i + N : (i >= N ? i - N : i); }

// ------------------------------------------------------------- SIMT conv
// out[v][co] = act(b[co] + sum_t sum_ci W[t][ci][co] in[v + off(t)][ci]),
// off(t) = (t/9 - 1, (t/3)%3 - 1, t%3 - 1); FLIP uses -off(t) and W[t][co][ci]
// (the data gradient of the forward convolution).  gate (NULL: none): the
// leaky-ReLU backward of the layer below, out *= (gate > 0 ? 1 : 0.1), with
// that layer's output (same sign as its pre-activation).
template <bool FLIP>
__global__ void __launch_bounds__(T) k_conv_simt(const __nv_bfloat16* __restrict__ in, int N,
                                                 const __nv_bfloat16* __restrict__ w,
                                                 const float* __restrict__ bias, int act,
                                                 const __nv_bfloat16* __restrict__ gate,
                                                 float* __restrict__ out_f,
                                                 __nv_bfloat16* __restrict__ out_b,
                                                 float4* __restrict__ out4) {
  __shared__ float ws[WSZ];
  for (int i = threadIdx.x; i < WSZ; i += T) {
    const int t = i / (C * C), a = (i / C) % C, b = i % C;   // ws[t][ci][co]
    ws[i] = FLIP ? __bfloat162float(w[(26 - t) * C * C + b * C + a])
                 : __bfloat162float(w[i]);
  }
  __syncthreads();
  const size_t nv = (size_t)N * N * N;
  for (size_t v = (size_t)blockIdx.x * T + threadIdx.x; v < nv; v += (size_t)gridDim.x * T) {
    const int x = (int)(v / ((size_t)N * N)), y = (int)((v / N) % N), z = (int)(v % N);
    float acc[C];
#pragma unroll
    for (int co = 0; co < C; co++) acc[co] = bias ? bias[co] : 0.0f;
    for (int t = 0; t < NT; t++) {
      const int xx = wrapi(x + t / 9 - 1, N), yy = wrapi(y + (t / 3) % 3 - 1, N),
                zz = wrapi(z + t % 3 - 1, N);
      const uint4* src = reinterpret_cast<const uint4*>(in + (((size_t)xx * N + yy) * N + zz) * C);
      const uint4 q0 = src[0], q1 = src[1];
      const __nv_bfloat16* h0 = reinterpret_cast<const __nv_bfloat16*>(&q0);
      const __nv_bfloat16* h1 = reinterpret_cast<const __nv_bfloat16*>(&q1);
      float iv[C];
#pragma unroll
      for (int c = 0; c < 8; c++) {
        iv[c] = __bfloat162float(h0[c]);
        iv[8 + c] = __bfloat162float(h1[c]);
      }
      const float* wt = ws + t * C * C;
#pragma unroll
      for (int ci = 0; ci < C; ci++)
#pragma unroll
        for (int co = 0; co < C; co++) acc[co] = fmaf(wt[ci * C + co], iv[ci], acc[co]);
    }
#pragma unroll
    for (int co = 0; co < C; co++) {
      float a = acc[co];
      if (act) a = a > 0.0f ? a : 0.1f * a;
      if (gate && __bfloat162float(gate[v * C + co]) <= 0.0f) a *= 0.1f;
      acc[co] = a;
    }
    if (out_f) {
#pragma unroll
      for (int co = 0; co < C; co++) out_f[v * C + co] = acc[co];
    }
    if (out_b) {
      __nv_bfloat16 hb[C];
#pragma unroll
      for (int co = 0; co < C; co++) hb[co] = __float2bfloat16_rn(acc[co]);
      uint4* dst = reinterpret_cast<uint4*>(out_b + v * C);
      dst[0] = *reinterpret_cast<const uint4*>(&hb[0]);
      dst[1] = *reinterpret_cast<const uint4*>(&hb[8]);
    }
    if (out4) out4[v] = make_float4(acc[0], acc[1], acc[2], acc[3]);
  }
}

// ------------------------------------------------- weight gradient (SIMT)
// dW[t][ci][co] += sum_v in[v + off(t)][ci] g[v][co];  db[co] += sum_v g[v][co].
// A CTA walks z-lines (x, y); thread j owns weights j, j + T, ... (27 each)
// and accumulates them in registers; one atomic per weight per CTA.
__global__ void __launch_bounds__(T) k_conv_wgrad(const __nv_bfloat16* __restrict__ in,
                                                  const float* __restrict__ g, int N,
                                                  float* __restrict__ dw,
                                                  float* __restrict__ db) {
  constexpr int PER = WSZ / T;   // 27
  static_assert(WSZ % T == 0, "weight count");
  extern __shared__ float sm[];
  float* sin = sm;                          // [9 lines][N + 2][C]
  float* sg = sm + 9 * (N + 2) * C;         // [N][C]
  float acc[PER];
#pragma unroll
  for (int i = 0; i < PER; i++) acc[i] = 0.0f;
  float bacc = 0.0f;
  for (int line = blockIdx.x; line < N * N; line += gridDim.x) {
    const int x = line / N, y = line % N;
    __syncthreads();
    for (int i = threadIdx.x; i < 9 * (N + 2) * C; i += T) {
      const int l = i / ((N + 2) * C), r = (i / C) % (N + 2), c = i % C;
      const int xx = wrapi(x + l / 3 - 1, N), yy = wrapi(y + l % 3 - 1, N), zz = wrapi(r - 1, N);
      sin[i] = __bfloat162float(in[(((size_t)xx * N + yy) * N + zz) * C + c]);
    }
    for (int i = threadIdx.x; i < N * C; i += T) sg[i] = g[((size_t)x * N + y) * N * C + i];
    __syncthreads();
#pragma unroll 1
    for (int q = 0; q < PER; q++) {
      const int wi = threadIdx.x + q * T;
      const int t = wi / (C * C), ci = (wi / C) % C, co = wi % C;
      const int l = (t / 9) * 3 + (t / 3) % 3, dz = t % 3;   // line and z shift (+1 halo)
      const float* a = sin + (size_t)l * (N + 2) * C + dz * C + ci;
      const float* b = sg + co;
      float s = 0.0f;
      for (int z = 0; z < N; z++) s = fmaf(a[z * C], b[z * C], s);
      acc[q] += s;
    }
    if (threadIdx.x < C) {
      float s = 0.0f;
      for (int z = 0; z < N; z++) s += sg[z * C + threadIdx.x];
      bacc += s;
    }
  }
#pragma unroll 1
  for (int q = 0; q < PER; q++) atomicAdd(dw + threadIdx.x + q * T, acc[q]);
  if (threadIdx.x < C) atomicAdd(db + threadIdx.x, bacc);
}

__global__ void k_f2b(const float* __restrict__ a, __nv_bfloat16* __restrict__ b, size_t n) {
  for (size_t i = (size_t)blockIdx.x * T + threadIdx.x; i < n; i += (size_t)gridDim.x * T)
    b[i] = __float2bfloat16_rn(a[i]);
}

// Masked mean-squared-error gradient on the 3 output channels:
// L = sum_v m_v sum_c (o_vc - r_vc)^2 / sum_v m_v;  g = dL/do, with the
// residual target r_v = inv_scale (sum of the residuals) / m_v (0 where m_v
// is 0) formed from the deposit's sums `resid` (x, y, z, mass).  Four threads per
// voxel write its 16 channels (float32 and bf16) in coalesced runs, 13 of
// them zero: HBM-bound on the 96 bytes written and 32 read (128^3: 156 us
// for the 16-channel scalar form with a separate normalisation pass).
__global__ void k_loss(const float4* __restrict__ o, const float4* __restrict__ resid, size_t nv,
                       float inv_scale, double inv_msum, float4* __restrict__ g,
                       uint2* __restrict__ gb, double* __restrict__ loss) {
  double acc = 0.0;
  for (size_t i = (size_t)blockIdx.x * T + threadIdx.x; i < 4 * nv; i += (size_t)gridDim.x * T) {
    float4 gv = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if ((i & 3) == 0) {
      const float4 ov = o[i >> 2], rs = resid[i >> 2];
      const float mv = rs.w;
      const float oc[3] = {ov.x, ov.y, ov.z}, rc[3] = {rs.x, rs.y, rs.z};
      float gc[3];
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const float d = oc[c] - (mv > 0 ? __fmul_rn(rc[c] / mv, inv_scale) : 0.0f);
        acc += (double)mv * d * d;
        gc[c] = (float)(2.0 * inv_msum) * mv * d;
      }
      gv = make_float4(gc[0], gc[1], gc[2], 0.0f);
    }
    g[i] = gv;
    const __nv_bfloat162 b0 = __floats2bfloat162_rn(gv.x, gv.y);
    const __nv_bfloat162 b1 = __floats2bfloat162_rn(gv.z, gv.w);
    gb[i] = make_uint2(*reinterpret_cast<const unsigned*>(&b0),
                       *reinterpret_cast<const unsigned*>(&b1));
  }
  for (int s = 16; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
  if ((threadIdx.x & 31) == 0) atomicAdd(loss, acc * inv_msum);
}

// Adam on float32 masters, refreshes the bf16 copies (layer weights are
// contiguous: w, then bias).
__global__ void k_adam(float* __restrict__ p, const float* __restrict__ gr, float* __restrict__ m1,
                       float* __restrict__ m2, int n, float lr, float b1, float b2, float eps,
                       float c1, float c2, const int* __restrict__ trainable) {
  for (int i = blockIdx.x * T + threadIdx.x; i < n; i += gridDim.x * T) {
    if (!trainable[i]) continue;
    const float gi = gr[i];
    m1[i] = b1 * m1[i] + (1 - b1) * gi;
    m2[i] = b2 * m2[i] + (1 - b2) * gi * gi;
    p[i] -= lr * (m1[i] / c1) / (sqrtf(m2[i] / c2) + eps);
  }
}

// Features: channel 0 = delta, channel 1 = phi (both on the coarse mesh), as
// pairs and, with wide, in the 16-channel layout.
__global__ void k_features(const float* __restrict__ delta, const float* __restrict__ phi,
                           size_t nv, float sd, float sp, __nv_bfloat162* __restrict__ f,
                           __nv_bfloat16* __restrict__ wide) {
  for (size_t v = (size_t)blockIdx.x * T + threadIdx.x; v < nv; v += (size_t)gridDim.x * T) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(delta[v] * sd, phi[v] * sp);
    f[v] = h;
    if (wide) {
      uint4* d = reinterpret_cast<uint4*>(wide + v * C);
      d[0] = make_uint4(*reinterpret_cast<const unsigned*>(&h), 0, 0, 0);
      d[1] = make_uint4(0, 0, 0, 0);
    }
  }
}

// phi_k = -delta_k / |n|^2 / N^3 on the half spectrum [kz][kx][ky]
__global__ void k_potential(float2* __restrict__ s, int N) {
  const size_t total = (size_t)(N / 2 + 1) * N * N;
  for (size_t t = (size_t)blockIdx.x * T + threadIdx.x; t < total; t += (size_t)gridDim.x * T) {
    const int kz = (int)(t / ((size_t)N * N)), i = (int)((t / N) % N), j = (int)(t % N);
    const int si = i <= N / 2 ? i : i - N, sj = j <= N / 2 ? j : j - N;
    const float n2 = (float)(si * si + sj * sj + kz * kz);
    const float f = n2 > 0 ? -1.0f / (n2 * (float)N * (float)N * (float)N) : 0.0f;
    s[t] = make_float2(s[t].x * f, s[t].y * f);
  }
}

// Periodic cells (lower, upper) and fraction of one coordinate in mesh units.
struct Axis { int i0, i1; float d; };
__device__ __forceinline__ Axis axis_cells(float X, int N) {
  const int i = (int)floorf(X);
  Axis a;
  a.d = X - i;
  a.i0 = i;
  if ((unsigned)i >= (unsigned)N) a.i0 = (i % N + N) % N;   // outside the box
  a.i1 = a.i0 + 1 == N ? 0 : a.i0 + 1;
  return a;
}

// CIC deposit of per-particle values (3 components) and mass on a periodic
// coarse mesh (plain periodic CIC: the residual target, not the PM density):
// one 16-byte atomic per corner for the three residuals and the mass (128^3
// particles: 346 us with four scalar atomics per corner).
__global__ void k_deposit_resid(const float* __restrict__ x0, const float* __restrict__ x1,
                                const float* __restrict__ x2, const float* __restrict__ fa0,
                                const float* __restrict__ fa1, const float* __restrict__ fa2,
                                const float* __restrict__ fb0, const float* __restrict__ fb1,
                                const float* __restrict__ fb2, long long n, int N, float scale,
                                float4* __restrict__ r) {
  for (long long i = (long long)blockIdx.x * T + threadIdx.x; i < n;
       i += (long long)gridDim.x * T) {
    const Axis x = axis_cells(x0[i] * scale, N), y = axis_cells(x1[i] * scale, N),
               z = axis_cells(x2[i] * scale, N);
    const float res[3] = {fa0[i] - fb0[i], fa1[i] - fb1[i], fa2[i] - fb2[i]};
#pragma unroll
    for (int c = 0; c < 8; c++) {
      const int ax = c >> 2, ay = (c >> 1) & 1, az = c & 1;
      const float w = (ax ? x.d : 1 - x.d) * (ay ? y.d : 1 - y.d) * (az ? z.d : 1 - z.d);
      const size_t v = ((size_t)(ax ? x.i1 : x.i0) * N + (ay ? y.i1 : y.i0)) * N +
                       (az ? z.i1 : z.i0);
      atomicAdd(r + v, make_float4(w * res[0], w * res[1], w * res[2], w));
    }
  }
}

// Add the CIC-interpolated network output (3 channels, scaled) to forces.
__global__ void k_apply(const float* __restrict__ x0, const float* __restrict__ x1,
                        const float* __restrict__ x2, long long n, int N, float scale,
                        const float4* __restrict__ o, float out_scale, float* __restrict__ f0,
                        float* __restrict__ f1, float* __restrict__ f2) {
  for (long long i = (long long)blockIdx.x * T + threadIdx.x; i < n;
       i += (long long)gridDim.x * T) {
    const Axis x = axis_cells(x0[i] * scale, N), y = axis_cells(x1[i] * scale, N),
               z = axis_cells(x2[i] * scale, N);
    float acc[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int c = 0; c < 8; c++) {
      const int ax = c >> 2, ay = (c >> 1) & 1, az = c & 1;
      const float w = (ax ? x.d : 1 - x.d) * (ay ? y.d : 1 - y.d) * (az ? z.d : 1 - z.d);
      const float4 ov = __ldg(o + ((size_t)(ax ? x.i1 : x.i0) * N + (ay ? y.i1 : y.i0)) * N +
                              (az ? z.i1 : z.i0));
      acc[0] += w * ov.x;
      acc[1] += w * ov.y;
      acc[2] += w * ov.z;
    }
    f0[i] += out_scale * acc[0];
    f1[i] += out_scale * acc[1];
    f2[i] += out_scale * acc[2];
  }
}

}  // namespace

// ------------------------------------------------------------- host side
cudaError_t cnet_alloc(CNet* n, int N, unsigned long long seed) {
  memset(n, 0, sizeof(*n));
  n->N = N;
  n->out_scale = 1.0f;
  n->in_scale[0] = n->in_scale[1] = 1.0f;
  const size_t nv = (size_t)N * N * N;
  const int P = CNET_PARAMS;
  cudaError_t e = cudaSuccess;
#define CN_TRY(x) do { if (e == cudaSuccess) e = (x); } while (0)
  // shared-memory limits belong to a device, so every net sets them on its own
  CN_TRY(conv_tc_set_smem());
  CN_TRY(conv_wgrad_set_smem());
  CN_TRY(cudaFuncSetAttribute(k_conv_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              200 * 1024));
  CN_TRY(cudaMalloc(&n->params, sizeof(float) * P));
  CN_TRY(cudaMalloc(&n->grads, sizeof(float) * P));
  CN_TRY(cudaMalloc(&n->m1, sizeof(float) * P));
  CN_TRY(cudaMalloc(&n->m2, sizeof(float) * P));
  CN_TRY(cudaMalloc(&n->trainable, sizeof(int) * P));
  CN_TRY(cudaMalloc(&n->wb, sizeof(__nv_bfloat16) * 3 * WSZ));
  for (int l = 0; l < 3; l++) CN_TRY(cudaMalloc(&n->act[l], sizeof(__nv_bfloat16) * nv * C));
  CN_TRY(cudaMalloc(&n->feat, sizeof(__nv_bfloat162) * nv));
  CN_TRY(cudaMalloc(&n->out, sizeof(float) * nv * C));
  CN_TRY(cudaMalloc(&n->out4, sizeof(float4) * nv));
  CN_TRY(cudaMalloc(&n->g0, sizeof(float) * nv * C));
  CN_TRY(cudaMalloc(&n->g1, sizeof(float) * nv * C));
  CN_TRY(cudaMalloc(&n->gb, sizeof(__nv_bfloat16) * nv * C));
  CN_TRY(cudaMalloc(&n->resid, sizeof(float4) * nv));
  CN_TRY(cudaMalloc(&n->loss, sizeof(double)));
  CN_TRY(cudaMalloc(&n->phi, sizeof(float) * nv));
  CN_TRY(cudaMalloc(&n->spec, sizeof(float2) * (size_t)(N / 2 + 1) * N * N));
  CN_TRY(mesh_fft_alloc(&n->fft, N));
#undef CN_TRY
  if (e != cudaSuccess) {
    cnet_free(n);
    return e;
  }
  // initial weights: He-scaled uniform for the hidden layers, small output
  // layer; channel masks: layer 0 reads channels 0-1, layer 2 writes 0-2.
  std::vector<float> p(P, 0.0f);
  std::vector<int> tr(P, 0);
  unsigned long long s = seed * 6364136223846793005ULL + 1442695040888963407ULL;
  auto rnd = [&]() {
    s = s * 6364136223846793005ULL + 1442695040888963407ULL;
    return ((s >> 11) * (1.0 / 9007199254740992.0)) * 2.0 - 1.0;
  };
  const int cin[3] = {2, C, C}, cout[3] = {C, C, 3};
  for (int l = 0; l < 3; l++) {
    const double scale = l == 2 ? 0.1 * sqrt(3.0 / (NT * cin[l])) : sqrt(6.0 / (NT * cin[l]));
    for (int t = 0; t < NT; t++)
      for (int ci = 0; ci < C; ci++)
        for (int co = 0; co < C; co++) {
          const int i = l * (WSZ + C) + (t * C + ci) * C + co;
          if (ci < cin[l] && co < cout[l]) {
            p[i] = (float)(scale * rnd());
            tr[i] = 1;
          }
        }
    for (int co = 0; co < cout[l]; co++) tr[l * (WSZ + C) + WSZ + co] = 1;
  }
  e = cudaMemcpy(n->params, p.data(), sizeof(float) * P, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(n->trainable, tr.data(), sizeof(int) * P, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(n->m1, 0, sizeof(float) * P);
  if (e == cudaSuccess) e = cudaMemset(n->m2, 0, sizeof(float) * P);
  if (e == cudaSuccess) e = cnet_sync_bf16(n, 0);
  return e;
}

void cnet_free(CNet* n) {
  cudaFree(n->params); cudaFree(n->grads); cudaFree(n->m1); cudaFree(n->m2);
  cudaFree(n->trainable); cudaFree(n->wb);
  for (int l = 0; l < 3; l++) cudaFree(n->act[l]);
  cudaFree(n->feat); cudaFree(n->out); cudaFree(n->out4); cudaFree(n->g0); cudaFree(n->g1); cudaFree(n->gb);
  cudaFree(n->resid); cudaFree(n->loss); cudaFree(n->phi);
  cudaFree(n->spec);
  mesh_fft_free(&n->fft);
  memset(n, 0, sizeof(*n));
}

cudaError_t cnet_sync_bf16(CNet* n, cudaStream_t st) {
  for (int l = 0; l < 3; l++) {
    prof_mark(st, CG_ST_OTHER);
    k_f2b<<<grid_for(WSZ), T, 0, st>>>(n->params + l * (WSZ + C), n->wb + l * WSZ, WSZ);
  }
  return cudaGetLastError();
}

static cudaError_t conv(const CNet* n, const __nv_bfloat16* in, const __nv_bfloat16* w,
                        const float* bias, int act, float* of, __nv_bfloat16* ob, bool flip,
                        cudaStream_t st, float4* o4 = nullptr,
                        const __nv_bfloat16* gate = nullptr) {
  const int N = n->N;
  const long long nv = (long long)N * N * N;
  if (n->use_tc && !flip) {
    cudaError_t e = conv_tc_forward(in, N, w, bias, act, of, ob, o4, st);
    if (e != cudaErrorNotSupported) return e;
  }
  if (n->use_tc && flip) {
    cudaError_t e = conv_tc_backward_data(in, N, w, gate, of, ob, st);
    if (e != cudaErrorNotSupported) return e;
  }
  prof_mark(st, CG_ST_OTHER);
  if (flip)
    k_conv_simt<true><<<grid_for(nv), T, 0, st>>>(in, N, w, bias, act, gate, of, ob, o4);
  else
    k_conv_simt<false><<<grid_for(nv), T, 0, st>>>(in, N, w, bias, act, gate, of, ob, o4);
  return cudaGetLastError();
}

bool cnet_narrow_input(const CNet* n) { return n->use_tc && n->N % 128 == 0; }

cudaError_t cnet_forward(CNet* n, cudaStream_t st, bool full, bool wide) {
  cudaError_t e;
  const float* P = n->params;
  if (!wide && cnet_narrow_input(n))
    e = conv_tc_features(n->feat, n->N, n->wb, P + WSZ, 1, n->act[1], st);
  else
    e = conv(n, n->act[0], n->wb, P + WSZ, 1, nullptr, n->act[1], false, st);
  if (e) return e;
  if ((e = conv(n, n->act[1], n->wb + WSZ, P + (WSZ + C) + WSZ, 1, nullptr, n->act[2], false, st)))
    return e;
  return conv(n, n->act[2], n->wb + 2 * WSZ, P + 2 * (WSZ + C) + WSZ, 0, full ? n->out : nullptr,
              nullptr, false, st, n->out4);
}

// Backward from g0 = dL/dout (3 output channels, float [v][16]); parameter
// gradients into n->grads.  Each data gradient comes out of its convolution
// with the activation below applied, in float32 for the weight gradient and in
// bf16 for the next convolution (the second bf16 buffer is the memory of the
// [v][16] output, which nothing reads once its gradient is known).
cudaError_t cnet_backward(CNet* n, cudaStream_t st, bool gb_ready) {
  const int N = n->N;
  const size_t nv = (size_t)N * N * N;
  const size_t wgrad_smem = sizeof(float) * (9 * (N + 2) * C + N * C);
  cudaMemsetAsync(n->grads, 0, sizeof(float) * CNET_PARAMS, st);
  float* g = n->g0;
  float* gnext = n->g1;
  __nv_bfloat16* gb = n->gb;
  __nv_bfloat16* gbnext = reinterpret_cast<__nv_bfloat16*>(n->out);
  if (!gb_ready) {
    prof_mark(st, CG_ST_OTHER);
    k_f2b<<<grid_for((long long)nv * C), T, 0, st>>>(g, gb, nv * C);
  }
  for (int l = 2; l >= 0; l--) {
    float* dw = n->grads + l * (WSZ + C);
    cudaError_t ew = cudaErrorNotSupported;
    if (n->use_tc)
      ew = l == 0 ? conv_wgrad_in(n->feat, g, N, dw, dw + WSZ, st)
                  : conv_wgrad_tc(n->act[l], g, N, l == 2, dw, dw + WSZ, st);
    if (ew == cudaErrorNotSupported) {
      prof_mark(st, CG_ST_OTHER);
      k_conv_wgrad<<<cg_sm_count() * 2, T, wgrad_smem, st>>>(n->act[l], g, N, dw, dw + WSZ);
      ew = cudaGetLastError();
    }
    if (ew != cudaSuccess) return ew;
    if (l == 0) break;
    // data gradient through layer l, then through the activation of layer l-1
    // (the first layer's gradient feeds its weights alone)
    cudaError_t e = conv(n, gb, n->wb + l * WSZ, nullptr, 0, gnext, l > 1 ? gbnext : nullptr,
                         true, st, nullptr, n->act[l]);
    if (e != cudaSuccess) return e;
    float* tmp = g; g = gnext; gnext = tmp;
    __nv_bfloat16* tb = gb; gb = gbnext; gbnext = tb;
  }
  return cudaGetLastError();
}

cudaError_t cnet_loss_grad(CNet* n, double inv_msum, cudaStream_t st) {
  const size_t nv = (size_t)n->N * n->N * n->N;
  cudaMemsetAsync(n->loss, 0, sizeof(double), st);
  prof_mark(st, CG_ST_OTHER);
  k_loss<<<grid_for(4 * (long long)nv), T, 0, st>>>(n->out4, n->resid, nv, 1.0f / n->out_scale,
                                                    inv_msum, reinterpret_cast<float4*>(n->g0),
                                                    reinterpret_cast<uint2*>(n->gb), n->loss);
  return cudaGetLastError();
}

cudaError_t cnet_adam(CNet* n, float lr, cudaStream_t st) {
  n->step++;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.0f - powf(b1, (float)n->step), c2 = 1.0f - powf(b2, (float)n->step);
  prof_mark(st, CG_ST_OTHER);
  k_adam<<<grid_for(CNET_PARAMS), T, 0, st>>>(n->params, n->grads, n->m1, n->m2, CNET_PARAMS, lr,
                                              b1, b2, 1e-8f, c1, c2, n->trainable);
  return cnet_sync_bf16(n, st);
}

// Input features from a coarse PM plan whose density mesh holds delta.
cudaError_t cnet_features(CNet* n, const float* delta, bool wide, cudaStream_t st) {
  const int N = n->N;
  const size_t nv = (size_t)N * N * N;
  cudaError_t e = mesh_r2c(&n->fft, delta, n->spec, st);
  if (e != cudaSuccess) return e;
  prof_mark(st, CG_ST_OTHER);
  k_potential<<<grid_for((long long)(N / 2 + 1) * N * N), T, 0, st>>>(n->spec, N);
  if ((e = mesh_c2r(&n->fft, n->spec, n->phi, st)) != cudaSuccess) return e;
  prof_mark(st, CG_ST_OTHER);
  k_features<<<grid_for((long long)nv), T, 0, st>>>(
      delta, n->phi, nv, n->in_scale[0], n->in_scale[1], n->feat,
      wide || !cnet_narrow_input(n) ? n->act[0] : nullptr);
  return cudaGetLastError();
}

cudaError_t cnet_target(CNet* n, const float* const x[3], long long np, float boxsize,
                        const float* const f_fine[3], const float* const f_coarse[3],
                        cudaStream_t st) {
  const int N = n->N;
  const size_t nv = (size_t)N * N * N;
  cudaMemsetAsync(n->resid, 0, sizeof(float4) * nv, st);
  prof_mark(st, CG_ST_OTHER);
  k_deposit_resid<<<grid_for(np), T, 0, st>>>(x[0], x[1], x[2], f_fine[0], f_fine[1], f_fine[2],
                                              f_coarse[0], f_coarse[1], f_coarse[2], np, N,
                                              (float)N / boxsize, n->resid);
  return cudaGetLastError();
}

cudaError_t cnet_apply(const CNet* n, const float* const x[3], long long np, float boxsize,
                       float* const f[3], cudaStream_t st) {
  prof_mark(st, CG_ST_OTHER);
  k_apply<<<grid_for(np), T, 0, st>>>(x[0], x[1], x[2], np, n->N, (float)n->N / boxsize, n->out4,
                                      n->out_scale, f[0], f[1], f[2]);
  return cudaGetLastError();
}
