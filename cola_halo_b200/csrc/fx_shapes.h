// Shapes of the strided x pass by mesh size and schedule variant: ky columns
// per CTA, maximum radix, threads.  Host code only reads them; pm_kernels.cu
// compiles k_fx_sw / k_fx_inv_sw (TMA gather) and k_fx (direct loads) from
// them.
#pragma once

namespace cgfx {

// Schedules of the x and Green passes.  Variant 0 is the default; the others
// are compiled for meshes from here up and chosen per mesh size by the
// autotuner (pm_autotune) or set explicitly.
constexpr int MIN_TUNED_N = 256;

// TMA form.  A variant's number keeps its shape from one build to the next (cached
// and saved schedules hold numbers): 0 the default, 1 8 columns at radix 8 (16
// from 768 up), 2 16 columns at radix 16.  Default: 16 columns (128-byte rows) from 256 to 768, where the
// twiddles sit in shared memory and the 16-column form fits 2 CTAs per SM; 8
// columns at 1024, where they do not and it would fit one; 8 below 256, where
// 16 would leave fewer CTAs than SMs have room for.  One inverse launch, ms, as
// {16 columns radix 16, 8 columns radix 16, 8 columns radix 8}:
// 256: 0.024, 0.029, 0.029; 384: 0.079, 0.084, 0.097; 512: 0.183, 0.193,
// 0.182; 768: 0.566, 0.654, 0.734; 1024: 2.04, 1.53, 1.81.
struct FxCfg { int tk, rm; };
constexpr FxCfg fx_cfg(int N, int v) {
  if (v == 1) return FxCfg{8, N >= 768 ? 16 : 8};
  return v == 2 || (N >= 256 && N < 1024) ? FxCfg{16, 16} : FxCfg{8, 16};
}
// The first variant of v's shape (the default is one of the others).
constexpr int fx_first(int N, int v) {
  const FxCfg a = fx_cfg(N, 0), b = fx_cfg(N, v);
  return a.tk == b.tk && a.rm == b.rm ? 0 : v;
}

// Threads of the TMA form by mesh size: those whose radix-16 stages (N / 16
// butterflies per column) fill them in whole rounds.  Three components of the
// inverse pass, us, with 256 threads and with these: 1024: 4709, 4408; 192: 34,
// 31; 144: 16.9, 14.8; 96: 8.3, 6.7.
constexpr int fx_threads(int N, int tk, int rm) {
  return N <= 192 || (N >= 1024 && tk == 8 && rm == 16) ? 128 : 256;
}

// Direct form (slab windows, plain transforms, batch views of a smaller mesh):
// the variant's radix, so that both forms round alike, with columns and
// threads of its own.  It reads its twiddles from the table through 64-bit
// addresses, so three radix-16 butterflies in one thread take over 200
// registers, one CTA per SM; one or two take at most 128.  minb 0: no minimum
// of CTAs per SM asked for.  One launch, ms, plain and scaled by n_x:
//   768: 8 columns on 384 threads 0.746, 0.769 (8 on 256: 0.854, 1.058; 16 on 256:
//     0.990, 1.043; 8 columns radix 8 on 256: 0.779, 0.785)
//   384: 16 on 256 0.080, 0.110 (8 on 256: 0.088, 0.097; 16 on 384: 0.087, 0.093, which
//     gains in a slab's two scaled passes of four what the plain transforms lose)
//   512: 16 on 256 0.175, 0.197 (8 on 256: 0.211, 0.213)
//   256: 16 on 256 0.0210, 0.0228 (8 on 256: 0.0257, 0.0311)
//   1024: 8 on 256 1.85, 1.95 (16 on 256: 2.26, 2.35)
struct FxDirectCfg { int tk, rm, thr, minb; };
constexpr FxDirectCfg fx_direct_cfg(int N, int v) {
  if (fx_cfg(N, v).rm == 8) return FxDirectCfg{8, 8, 256, 0};
  if (N == 768) return FxDirectCfg{8, 16, 384, 2};
  return FxDirectCfg{N >= 256 && N < 768 ? 16 : 8, 16, 256, 0};
}

}  // namespace cgfx
