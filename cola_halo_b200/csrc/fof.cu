// Friends-of-friends halos on the GPU (fof.c:427-1181 on one process).
//
// The reference builds a k-d tree and grows one group at a time from a
// FIFO; across the x faces it links through buffer particles shifted by
// -L.  On one process that is periodic friends-of-friends: particles whose
// squared distance (float32, as kdFoF forms it, fof.c:569-572) is below
// ll^2 are linked, and groups of at least 32 (fof.c:224) are halos, with
// centre = a member position + the mean minimum-image offset of all
// members, wrapped into [0, L) (fof.c:287-322, 1141-1150), and the mean
// velocity.  Here:
//   1. wrap positions (move_particles2_min, fof.c:1042) and bin them on a
//      grid of cells no smaller than ll (counting sort: count with ranks,
//      scan, scatter); from here on a particle is its slot in cell order
//   2. the particles of crowded cells are put in the order of their sub-cells,
//      and those of a block of 32 slots that hang together are joined
//   3. each particle tests the later particles of the cells within ll of it;
//      a link joins the two sets of a lock-free union-find over the slots
//      (hooking one root under the other with atomicCAS, in a scrambled order
//      of the slots, path halving)
//   4. flatten to roots, count members and find each group's smallest
//      original index, number the groups with >= nfof_min members in the
//      order of that index (a scan), accumulate the offsets from that
//      particle and the velocities in double, and finish each halo.
// So the catalogue is in a fixed order and each centre's reference member is
// fixed.  Every retry loop is bounded; running out of iterations sets an
// error word.
//
// 256^3 particles, L = 600, ll = 0.2 spacings, a third of them in halos: the
// link kernel takes 5.3 ms (12.4 with all 27 neighbour cells and a union-find
// over the original indices; 8.8 with one candidate at a time), and the whole call
// 9.5 to 10.7 ms (26.6), of which about 2 go to the allocation.  The link kernel
// is bound by its chains of dependent loads: cell starts (134M of them, four
// times L2), candidates, parents; two thirds of it are the slots outside clumps.
#include <cuda_runtime.h>
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include "../../include/colagpu.h"
#include "../../include/colagpu_dropin.h"
#include "gadget.h"
#include "internal.h"
#include "scan.cuh"

extern int cg_set_error_from_lpt(int code, const char* msg);

namespace {

constexpr int T = CG_THREADS;
constexpr int MAX_NCELL = 512;          // cells per dimension at most
constexpr int kRetryLimit = 1 << 22;    // union / find iterations per call

// Reference ParticleMinimum (particle.h:24-29): 32 bytes.
struct PMin {
  float x[3];
  float v[3];
  long long id;
};

__device__ __forceinline__ float wrap1(float x, float L) {
  // one-shot periodic wrap as move.c:34-41
  if (x < 0.0f) x += L;
  else if (x >= L) x -= L;
  return x;
}

__device__ __forceinline__ int cell_of(float x, float inv, int nc) {
  int c = (int)(x * inv);
  return c < 0 ? 0 : (c >= nc ? nc - 1 : c);
}

// Each particle's cell and its rank among the cell's arrivals.
__global__ void k_fof_bin(const PMin* __restrict__ p, long long n, float L, float inv, int nc,
                          unsigned* __restrict__ key, unsigned* __restrict__ rank,
                          unsigned* __restrict__ count) {
  for (long long i = (long long)blockIdx.x * T + threadIdx.x; i < n;
       i += (long long)gridDim.x * T) {
    const float4 q = *reinterpret_cast<const float4*>(p + i);
    const float x = wrap1(q.x, L), y = wrap1(q.y, L), z = wrap1(q.z, L);
    const unsigned k =
        ((unsigned)cell_of(x, inv, nc) * nc + cell_of(y, inv, nc)) * nc + cell_of(z, inv, nc);
    key[i] = k;
    rank[i] = atomicAdd(count + k, 1u);
  }
}

// Wrapped position and original index at the particle's slot.
__global__ void k_fof_scatter(const PMin* __restrict__ p, const unsigned* __restrict__ key,
                              const unsigned* __restrict__ rank, long long n, float L,
                              const unsigned* __restrict__ start, float4* __restrict__ pos) {
  for (long long i = (long long)blockIdx.x * T + threadIdx.x; i < n;
       i += (long long)gridDim.x * T) {
    const float4 q = *reinterpret_cast<const float4*>(p + i);
    const unsigned slot = start[key[i]] + rank[i];
    pos[slot] = make_float4(wrap1(q.x, L), wrap1(q.y, L), wrap1(q.z, L), __int_as_float((int)i));
  }
}

// ------------------------------------------------------------- union-find
// parent[] over slots; a root is parent[r] == r.
__device__ __forceinline__ int find_root(int* parent, int x, unsigned* err) {
  for (int it = 0; it < kRetryLimit; it++) {
    const int p = __ldcg(parent + x);
    if (p == x) return x;
    const int gp = __ldcg(parent + p);
    if (gp != p) atomicCAS(parent + x, p, gp);   // path halving (benign race)
    x = gp;
  }
  atomicOr(err, 1u);
  return x;
}

// Which of two roots hangs under the other: a fixed scrambling of the slots.
// With the slots' own order, threads that work through neighbouring slots at
// once would hang every particle of a halo under the one before it, a chain as
// long as the halo (256^3: the link kernel three times slower).
__device__ __forceinline__ unsigned rank_of(int slot) { return (unsigned)slot * 2654435761u; }

// Join the sets of a and b; returns the root they then share.
__device__ __forceinline__ int unite(int* parent, int a, int b, unsigned* err) {
  for (int it = 0; it < kRetryLimit; it++) {
    a = find_root(parent, a, err);
    b = find_root(parent, b, err);
    if (a == b) return a;
    if (rank_of(a) > rank_of(b)) {
      const int t = a;
      a = b;
      b = t;
    }
    // hang the later root under the earlier one if it is still a root
    if (atomicCAS(parent + b, b, a) == b) return a;
  }
  atomicOr(err, 2u);
  return a;
}

// Squared distance of two wrapped positions with the periodic image formed
// as the reference forms it: the coordinate of the particle on the far side
// is shifted by -L before the difference (fof.c:645-647, and the cell
// images of INTERSECT), float arithmetic without contraction.
__device__ __forceinline__ float dist2(float4 a, float4 b, float L, float half) {
  float d[3];
  const float pa[3] = {a.x, a.y, a.z}, pb[3] = {b.x, b.y, b.z};
#pragma unroll
  for (int k = 0; k < 3; k++) {
    float t = __fsub_rn(pa[k], pb[k]);
    if (t > half) t = __fsub_rn(__fsub_rn(pa[k], L), pb[k]);
    else if (t < -half) t = __fsub_rn(__fsub_rn(pb[k], L), pa[k]);
    d[k] = t;
  }
  return __fadd_rn(__fadd_rn(__fmul_rn(d[0], d[0]), __fmul_rn(d[1], d[1])),
                   __fmul_rn(d[2], d[2]));
}

// Cells of one axis within `reach` of [x0, x1]: lo .. hi, unwrapped (below 0 or
// above nc - 1 across the periodic face), or every cell.  reach is ll plus a
// margin over the rounding of x +- reach, and cell_of never decreases with x, so
// no particle closer than ll lies outside.
__device__ __forceinline__ void cells_within(float x0, float x1, float reach, float L, float inv,
                                             int nc, int& lo, int& hi) {
  const float a = x0 - reach, b = x1 + reach;
  lo = a < 0.0f ? cell_of(a + L, inv, nc) - nc : cell_of(a, inv, nc);
  hi = b >= L ? cell_of(b - L, inv, nc) + nc : cell_of(b, inv, nc);
  if (hi - lo + 1 >= nc) {
    lo = 0;
    hi = nc - 1;
  }
}

// Cells with more than a warp of particles (and at most kSubMax), listed by
// their first slot.
constexpr int kSubMax = 2048;
__global__ void k_fof_dense(const float4* __restrict__ pos, long long n,
                            const unsigned* __restrict__ start, int nc, float inv,
                            unsigned* __restrict__ list, unsigned* __restrict__ count) {
  for (long long i = (long long)blockIdx.x * T + threadIdx.x; i < n;
       i += (long long)gridDim.x * T) {
    const float4 a = pos[i];
    const unsigned k = ((unsigned)cell_of(a.x, inv, nc) * nc + cell_of(a.y, inv, nc)) * nc +
                       cell_of(a.z, inv, nc);
    if (start[k] != (unsigned)i) continue;
    const unsigned m = start[k + 1] - (unsigned)i;
    if (m > 32 && m <= kSubMax) list[atomicAdd(count, 1u)] = k;
  }
}

// Their particles in the order of 4^3 sub-cells (a counting sort in shared
// memory), so that 32 consecutive slots of a halo are a compact clump: the
// ranges and the blocks that k_fof_link looks at shrink with it.
constexpr int kSubThreads = 128;
__global__ void __launch_bounds__(kSubThreads) k_fof_subsort(
    float4* __restrict__ pos, const unsigned* __restrict__ start, int nc, float inv,
    const unsigned* __restrict__ list, const unsigned* __restrict__ count) {
  __shared__ float4 buf[kSubMax];
  __shared__ unsigned at[64];
  const unsigned cells = *count;
  for (unsigned c = blockIdx.x; c < cells; c += gridDim.x) {
    const unsigned k = list[c], s0 = start[k], m = start[k + 1] - s0;
    const float cx = (float)(k / nc / nc), cy = (float)(k / nc % nc), cz = (float)(k % nc);
    const auto sub = [&](const float4& a) {
      const int x = min(max((int)(4.0f * (a.x * inv - cx)), 0), 3);
      const int y = min(max((int)(4.0f * (a.y * inv - cy)), 0), 3);
      const int z = min(max((int)(4.0f * (a.z * inv - cz)), 0), 3);
      return (x * 4 + y) * 4 + z;
    };
    if (threadIdx.x < 64) at[threadIdx.x] = 0;
    __syncthreads();
    for (unsigned i = threadIdx.x; i < m; i += kSubThreads) {
      buf[i] = pos[s0 + i];
      atomicAdd(&at[sub(buf[i])], 1u);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned run = 0;
      for (int b = 0; b < 64; b++) {
        const unsigned v = at[b];
        at[b] = run;
        run += v;
      }
    }
    __syncthreads();
    for (unsigned i = threadIdx.x; i < m; i += kSubThreads)
      pos[s0 + atomicAdd(&at[sub(buf[i])], 1u)] = buf[i];
    __syncthreads();
  }
}

// Bounding boxes of the blocks of 32 slots: box[2 b] the lower corner, box[2 b +
// 1] the upper one; and their first sets.  In halos, where a block is a clump of
// at most two cells across (marked in the lower corner's w), the slots that hang
// together within it go under the first of them: 32 broadcasts and votes in
// registers, where the link kernel would join them one pair after another through
// L2 while other warps meet 32 sets in place of one (256^3: 5.8 to 5.3 ms of
// link, for 0.15 here).  Other slots start as sets of their own.
__global__ void k_fof_blocks(const float4* __restrict__ pos, long long n, float inv, float L,
                             float ll2, float4* __restrict__ box, int* __restrict__ parent) {
  constexpr unsigned kAll = 0xffffffffu;
  const float half = 0.5f * L;
  const int lane = threadIdx.x & 31;
  for (long long base = (long long)blockIdx.x * T + (threadIdx.x & ~31); base < n;
       base += (long long)gridDim.x * T) {
    const bool live = base + lane < n;
    const float4 a = pos[live ? base + lane : n - 1];
    float lo[3] = {a.x, a.y, a.z}, hi[3] = {a.x, a.y, a.z};
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int k = 0; k < 3; k++) {
        lo[k] = fminf(lo[k], __shfl_xor_sync(kAll, lo[k], o));
        hi[k] = fmaxf(hi[k], __shfl_xor_sync(kAll, hi[k], o));
      }
    // (the warp's lanes hold the same corners)
    const bool clump =
        fmaxf(fmaxf(hi[0] - lo[0], hi[1] - lo[1]), hi[2] - lo[2]) * inv <= 2.0f;
    if (lane == 0) {
      box[base / 16] = make_float4(lo[0], lo[1], lo[2], clump ? 1.0f : 0.0f);
      box[base / 16 + 1] = make_float4(hi[0], hi[1], hi[2], 0.0f);
    }
    unsigned set = 1u << lane;      // the lanes that hang together with this one
    if (clump)
      for (int j = 0; j < 32; j++) {
        float4 d;
        d.x = __shfl_sync(kAll, a.x, j);
        d.y = __shfl_sync(kAll, a.y, j);
        d.z = __shfl_sync(kAll, a.z, j);
        const bool linked = base + j < n && live && (lane == j || dist2(a, d, L, half) < ll2);
        const unsigned near = __ballot_sync(kAll, linked);
        // every set with a lane near j becomes one
        const unsigned all = __ballot_sync(kAll, (set & near) != 0);
        if (set & near) set = all;
      }
    if (live) parent[base + lane] = (int)base + __ffs(set) - 1;
  }
}

// One thread per slot: links to the later slots of the cells within ll (each
// pair once: the earlier slot tests it).  The cells of one (x, y) row are
// consecutive in z, so a row is one range of slots, or two across the
// periodic face, and rows before the particle's own hold no later slot.
//
// In a clump (k_fof_blocks), whose own pairs are done, the lanes take the same
// ranges (the cells within ll of the clump) and skip the blocks of 32 candidates
// whose box is further than ll from the clump's.  Of a block that is left each
// lane loads one candidate and finds its root.  Once the clump is one set,
// candidates of that set drop out by one vote, and a link takes all candidates
// of the set it joins out too, so that most blocks of a halo cost two loads and
// no distance.  Elsewhere the few candidates are each lane's own; their parents
// are loaded four at a time.
//
// ra is an ancestor of s: a candidate whose parent or root it is belongs to the
// set already, for sets never split.
__global__ void __launch_bounds__(T, 5) k_fof_link(const float4* __restrict__ pos, long long n,
                                                   const float4* __restrict__ box,
                                                   const unsigned* __restrict__ start, int nc,
                                                   float inv, float L, float ll2, float reach,
                                                   int* parent, unsigned* __restrict__ err) {
  constexpr unsigned kAll = 0xffffffffu;
  const float half = 0.5f * L;
  const int lane = threadIdx.x & 31;
  for (long long base = (long long)blockIdx.x * T + (threadIdx.x & ~31); base < n;
       base += (long long)gridDim.x * T) {
    // lanes past the end stand in for the last slot, which has no later one
    const unsigned s = (unsigned)min(base + lane, n - 1);
    const float4 a = pos[s];
    float4 lo = box[base / 16], hi = box[base / 16 + 1];
    unsigned own = (unsigned)cell_of(a.x, inv, nc) * nc + cell_of(a.y, inv, nc);
    const bool clump = lo.w != 0.0f;
    if (clump) own = __reduce_min_sync(kAll, own);
    else lo = hi = a;
    int xl, xh, yl, yh, zl, zh;
    cells_within(lo.x, hi.x, reach, L, inv, nc, xl, xh);
    cells_within(lo.y, hi.y, reach, L, inv, nc, yl, yh);
    cells_within(lo.z, hi.z, reach, L, inv, nc, zl, zh);
    int ra = clump ? __ldcg(parent + s) : (int)s;
    // slots t .. end - 1, each lane its own
    const auto test = [&](unsigned t, unsigned end) {
      t = max(t, s + 1);
      for (; t < end; t += 4) {
        int pr[4];
#pragma unroll
        for (int u = 0; u < 4; u++) pr[u] = t + u < end ? __ldcg(parent + t + u) : ra;
#pragma unroll
        for (int u = 0; u < 4; u++)
          if (pr[u] != ra && dist2(a, pos[t + u], L, half) < ll2)
            ra = unite(parent, ra, (int)(t + u), err);
      }
    };
    // slots t .. end - 1 of the block of 32 at `b`, the same for all lanes
    const auto test_block = [&](unsigned b, unsigned t, unsigned end) {
      const unsigned c = b + lane;
      const bool in = c >= t && c < end;
      const float4 q = pos[in ? c : s];
      const int rc = in ? find_root(parent, (int)c, err) : -1;
      ra = find_root(parent, ra, err);
      int one;
      __match_all_sync(kAll, ra, &one);
      unsigned left = __ballot_sync(kAll, in && !(one && rc == ra));
      while (left) {
        const int j = __ffs(left) - 1;
        left &= left - 1;
        float4 d;
        d.x = __shfl_sync(kAll, q.x, j);
        d.y = __shfl_sync(kAll, q.y, j);
        d.z = __shfl_sync(kAll, q.z, j);
        const int rj = __shfl_sync(kAll, rc, j);
        const bool hit = b + j > s && rj != ra && dist2(a, d, L, half) < ll2;
        if (one) {
          if (!__any_sync(kAll, hit)) continue;
          if (lane == 0) ra = unite(parent, ra, rj, err);
          ra = __shfl_sync(kAll, ra, 0);
          left &= __ballot_sync(kAll, rc != rj);
        } else if (hit) {
          ra = unite(parent, ra, rj, err);
        }
        __syncwarp();
      }
    };
    // slots of the cells z0 .. z1 of a row; `near`: no periodic face in between
    const auto range = [&](unsigned row, int z0, int z1, bool near) {
      unsigned t = max(start[row * nc + z0], (unsigned)base + (clump ? 32 : 1));
      const unsigned end = start[row * nc + z1 + 1];
      if (!clump) {
        test(t, end);
        return;
      }
      for (; t < end; t = (t & ~31u) + 32u) {
        if (near) {
          const float4 bl = box[t / 32 * 2], bh = box[t / 32 * 2 + 1];
          if (bl.x > hi.x + reach || bh.x < lo.x - reach || bl.y > hi.y + reach ||
              bh.y < lo.y - reach || bl.z > hi.z + reach || bh.z < lo.z - reach)
            continue;
        }
        test_block(t & ~31u, t, end);
      }
    };
    for (int x = xl; x <= xh; x++) {
      const int gx = x < 0 ? x + nc : (x >= nc ? x - nc : x);
      for (int y = yl; y <= yh; y++) {
        const int gy = y < 0 ? y + nc : (y >= nc ? y - nc : y);
        const unsigned row = (unsigned)gx * nc + gy;
        if (row < own) continue;
        // ranges that stand for every cell have no image of their own
        const bool near = gx == x && gy == y && xh - xl + 1 < nc && yh - yl + 1 < nc &&
                          zh - zl + 1 < nc;
        if (zl < 0) range(row, zl + nc, nc - 1, false);
        range(row, max(zl, 0), min(zh, nc - 1), near);
        if (zh >= nc) range(row, 0, zh - nc, false);
      }
    }
  }
}

// Every slot's root, and per root the members and their smallest original
// index (lowest, set to 0xffffffff before).  The members of a group sit close
// to each other in cell order: lanes with the same root add once.
__global__ void k_fof_flatten(const float4* __restrict__ pos, int* __restrict__ parent,
                              long long n, unsigned* __restrict__ size,
                              unsigned* __restrict__ lowest, unsigned* __restrict__ err) {
  const int lane = threadIdx.x & 31;
  for (long long base = (long long)blockIdx.x * T + (threadIdx.x & ~31); base < n;
       base += (long long)gridDim.x * T) {
    const long long i = base + lane;
    const unsigned live = __ballot_sync(0xffffffffu, i < n);
    if (i >= n) continue;
    const int r = find_root(parent, (int)i, err);
    parent[i] = r;
    const unsigned orig = (unsigned)__float_as_int(pos[i].w);
    const unsigned same = __match_any_sync(live, r);
    const unsigned low = __reduce_min_sync(same, orig);
    if (lane == __ffs(same) - 1) {
      atomicAdd(size + r, (unsigned)__popc(same));
      atomicMin(lowest + r, low);
    }
  }
}

// A halo's flag stands at its smallest original index.
__global__ void k_fof_flag(const int* __restrict__ root, const unsigned* __restrict__ size,
                           const unsigned* __restrict__ lowest, long long n, unsigned nmin,
                           unsigned* __restrict__ flag) {
  for (long long i = (long long)blockIdx.x * T + threadIdx.x; i < n;
       i += (long long)gridDim.x * T)
    if (root[i] == (int)i && size[i] >= nmin) flag[lowest[i]] = 1u;
}

// Wrapped position of an original particle.
__device__ __forceinline__ float3 wrapped(const PMin* __restrict__ p, unsigned i, float L) {
  const float4 q = *reinterpret_cast<const float4*>(p + i);
  return make_float3(wrap1(q.x, L), wrap1(q.y, L), wrap1(q.z, L));
}

// Per member: offset from the halo's reference particle with the minimum-image
// wrap of halo_particle (fof.c:304-313, float), summed in double with the
// velocities.  acc[6 h + 0..2] = offsets, [3..5] = velocities.  A warp whose
// lanes all belong to one halo adds its sum once.
__global__ void k_fof_accum(const PMin* __restrict__ p, const float4* __restrict__ pos,
                            const int* __restrict__ root, const unsigned* __restrict__ size,
                            const unsigned* __restrict__ lowest,
                            const unsigned* __restrict__ hid, long long n, unsigned nmin, float L,
                            double* __restrict__ acc) {
  const float half = 0.5f * L;
  const int lane = threadIdx.x & 31;
  for (long long base = (long long)blockIdx.x * T + (threadIdx.x & ~31); base < n;
       base += (long long)gridDim.x * T) {
    const long long i = base + lane;
    const int r = i < n ? root[i] : -1;
    const bool in = r >= 0 && size[r] >= nmin;
    if (!__any_sync(0xffffffffu, in)) continue;
    double v[6] = {0, 0, 0, 0, 0, 0};
    unsigned h = 0xffffffffu;
    if (in) {
      const unsigned ref = lowest[r];
      h = hid[ref];
      const float4 a = pos[i];
      const float3 b = wrapped(p, ref, L);
      const PMin& q = p[__float_as_int(a.w)];
      const float d[3] = {__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z)};
#pragma unroll
      for (int k = 0; k < 3; k++) {
        float dx = d[k];
        if (dx > half) dx = __fsub_rn(dx, L);
        else if (dx < -half) dx = __fadd_rn(dx, L);
        v[k] = (double)dx;
        v[3 + k] = (double)q.v[k];
      }
    }
    if (__all_sync(0xffffffffu, h == __shfl_sync(0xffffffffu, h, 0))) {
#pragma unroll
      for (int k = 0; k < 6; k++)
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
      if (lane < 6) {
        const double s = lane == 0 ? v[0] : lane == 1 ? v[1] : lane == 2 ? v[2]
                       : lane == 3 ? v[3] : lane == 4 ? v[4] : v[5];
        atomicAdd(acc + 6 * (size_t)h + lane, s);
      }
    } else if (in) {
#pragma unroll
      for (int k = 0; k < 6; k++) atomicAdd(acc + 6 * (size_t)h + k, v[k]);
    }
  }
}

// Halo h: centre x0 + mean offset wrapped into [0, L) as fof.c:1141-1147,
// mean velocity (fof.c:1150).
__global__ void k_fof_finish(const PMin* __restrict__ p, const int* __restrict__ root,
                             const unsigned* __restrict__ size,
                             const unsigned* __restrict__ lowest,
                             const unsigned* __restrict__ hid, long long n, unsigned nmin, float L,
                             const double* __restrict__ acc, cg_halo* __restrict__ out,
                             long long max_out) {
  for (long long r = (long long)blockIdx.x * T + threadIdx.x; r < n;
       r += (long long)gridDim.x * T) {
    if (root[r] != (int)r || size[r] < nmin) continue;
    const unsigned ref = lowest[r], h = hid[ref];
    if ((long long)h >= max_out) continue;
    const unsigned nf = size[r];
    const float3 b = wrapped(p, ref, L);
    const float x0[3] = {b.x, b.y, b.z};
    cg_halo o;
    o.nfof = (int)nf;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      float x = __fadd_rn(x0[k], (float)(acc[6 * (size_t)h + k] / (double)nf));
      if (x < 0.0f) x += L;
      if (x >= L) x -= L;
      o.x[k] = x;
      o.v[k] = (float)(acc[6 * (size_t)h + 3 + k] / (double)nf);
    }
    out[h] = o;
  }
}

// One device block cut into arrays (16-byte aligned): a call takes and gives
// back one allocation instead of a dozen, each of which costs a mapping and a
// synchronisation (256^3: 10 of 26 ms).
struct Block {
  unsigned char* base = nullptr;
  size_t used = 0;
  template <class V>
  V* cut(long long count) {
    V* p = base ? reinterpret_cast<V*>(base + used) : nullptr;
    used += (sizeof(V) * (size_t)count + 15) / 16 * 16;
    return p;
  }
};

}  // namespace

extern "C" int cg_fof(const void* pmin, long long np, float boxsize, float ll, int nfof_min,
                      cg_halo* halos, long long max_halos, long long* nhalo) {
  if (!nhalo || np < 0 || np >= (1LL << 31) - 1 || !(boxsize > 0.0f) || !(ll > 0.0f) ||
      nfof_min < 1 || (max_halos > 0 && !halos) || (np > 0 && !pmin))
    return cg_set_error_from_lpt(CG_EINVAL, "cg_fof: bad arguments");
  *nhalo = 0;
  if (np == 0) return CG_OK;
  // cells no smaller than ll (with a margin over the float rounding of the
  // cell index, so linked pairs are never two cells apart), at most
  // MAX_NCELL per side and about 8 per particle
  long long nc = (long long)floor((double)boxsize / (double)ll * 0.99999);
  const long long ncap = (long long)cbrt(8.0 * (double)np) + 1;
  if (nc > MAX_NCELL) nc = MAX_NCELL;
  if (nc > ncap) nc = ncap;
  if (nc < 1) nc = 1;
  const long long ncells = nc * nc * nc;
  const float inv = (float)nc / boxsize;
  const long long nblk = cgscan::scratch_entries(ncells > np ? ncells + 1 : np);
  // every cell of a linked pair lies within `reach`: ll, plus the rounding of
  // the sums with positions up to 2 L
  const float reach = ll * 1.0001f + boxsize * 4e-7f;

  cudaPointerAttributes attr;
  bool on_device = cudaPointerGetAttributes(&attr, pmin) == cudaSuccess &&
                   (attr.type == cudaMemoryTypeDevice || attr.type == cudaMemoryTypeManaged);
  cudaGetLastError();   // a plain host pointer may leave an error behind
  // (records are read as 16-byte vectors; a device array off that boundary,
  // like a host array, is copied first)
  const bool in_place = on_device && reinterpret_cast<uintptr_t>(pmin) % 16 == 0;
  const PMin* d_p = nullptr;
  PMin* own = nullptr;
  unsigned *key = nullptr, *rank = nullptr, *start = nullptr, *size = nullptr, *lowest = nullptr;
  unsigned *flag = nullptr, *bsum = nullptr, *word = nullptr;
  int* parent = nullptr;
  float4 *pos = nullptr, *box = nullptr;
  Block blk;
  const auto cut = [&] {
    blk.used = 0;
    word = blk.cut<unsigned>(4);              // [0] halos, [1] error, [2] dense cells
    start = blk.cut<unsigned>(ncells + 1);    // counts, then starts; [ncells] = np
    size = blk.cut<unsigned>(np);
    flag = blk.cut<unsigned>(np);             // then the halo numbers
    lowest = blk.cut<unsigned>(np);
    parent = blk.cut<int>(np);
    key = blk.cut<unsigned>(np);
    rank = blk.cut<unsigned>(np);
    pos = blk.cut<float4>(np);
    box = blk.cut<float4>((np + 31) / 32 * 2);
    bsum = blk.cut<unsigned>(nblk + 1);
    own = blk.cut<PMin>(in_place ? 0 : np);
    d_p = in_place ? (const PMin*)pmin : own;
  };
  cut();
  cudaStream_t st = 0;
  cudaError_t e = cudaMalloc(&blk.base, blk.used);
  if (e != cudaSuccess) blk.base = nullptr;
  cut();
  if (e == cudaSuccess && !in_place)
    e = cudaMemcpy(own, pmin, sizeof(PMin) * np, cudaMemcpyDefault);
  // word, counts, sizes and flags start at 0, the smallest indices at the top
  if (e == cudaSuccess)
    e = cudaMemsetAsync(word, 0, (unsigned char*)lowest - (unsigned char*)word, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(lowest, 0xff, sizeof(unsigned) * np, st);
  unsigned nh = 0, hw[2] = {0, 0};
  void* big = nullptr;
  if (e == cudaSuccess) {
    const int g = grid_for(np);
    prof_mark(st, CG_ST_OTHER);
    k_fof_bin<<<g, T, 0, st>>>(d_p, np, boxsize, inv, (int)nc, key, rank, start);
    cgscan::exclusive(start, start, ncells + 1, bsum, nullptr, CG_ST_OTHER, st);
    prof_mark(st, CG_ST_OTHER);
    k_fof_scatter<<<g, T, 0, st>>>(d_p, key, rank, np, boxsize, start, pos);
    // (the list of dense cells goes where the ranks were)
    prof_mark(st, CG_ST_OTHER);
    k_fof_dense<<<g, T, 0, st>>>(pos, np, start, (int)nc, inv, rank, word + 2);
    prof_mark(st, CG_ST_OTHER);
    k_fof_subsort<<<cg_grid(np, 4), kSubThreads, 0, st>>>(pos, start, (int)nc, inv, rank,
                                                          word + 2);
    prof_mark(st, CG_ST_OTHER);
    k_fof_blocks<<<g, T, 0, st>>>(pos, np, inv, boxsize, ll * ll, box, parent);
    prof_mark(st, CG_ST_OTHER);
    k_fof_link<<<g, T, 0, st>>>(pos, np, box, start, (int)nc, inv, boxsize, ll * ll, reach,
                                parent, word + 1);
    prof_mark(st, CG_ST_OTHER);
    k_fof_flatten<<<g, T, 0, st>>>(pos, parent, np, size, lowest, word + 1);
    prof_mark(st, CG_ST_OTHER);
    k_fof_flag<<<g, T, 0, st>>>(parent, size, lowest, np, (unsigned)nfof_min, flag);
    cgscan::exclusive(flag, flag, np, bsum, word, CG_ST_OTHER, st);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpy(hw, word, sizeof(hw), cudaMemcpyDeviceToHost);
    nh = hw[0];
    if (e == cudaSuccess && nh > 0) {
      // the sums and the catalogue go where the cell keys and ranks were,
      // unless the halos are so small that they need more
      const size_t acc_bytes = (sizeof(double) * 6 * (size_t)nh + 15) / 16 * 16;
      const size_t need = acc_bytes + sizeof(cg_halo) * (size_t)nh;
      unsigned char* room = (unsigned char*)key;
      if (need > (size_t)((unsigned char*)pos - room)) {
        e = cudaMalloc(&big, need);
        room = (unsigned char*)big;
      }
      double* acc = (double*)room;
      cg_halo* out = (cg_halo*)(room + acc_bytes);
      if (e == cudaSuccess) e = cudaMemsetAsync(acc, 0, acc_bytes, st);
      if (e == cudaSuccess) {
        prof_mark(st, CG_ST_OTHER);
        k_fof_accum<<<g, T, 0, st>>>(d_p, pos, parent, size, lowest, flag, np,
                                     (unsigned)nfof_min, boxsize, acc);
        prof_mark(st, CG_ST_OTHER);
        k_fof_finish<<<g, T, 0, st>>>(d_p, parent, size, lowest, flag, np, (unsigned)nfof_min,
                                      boxsize, acc, out, nh);
        e = cudaGetLastError();
      }
      const long long ncopy = max_halos < (long long)nh ? max_halos : (long long)nh;
      if (e == cudaSuccess && ncopy > 0)
        e = cudaMemcpy(halos, out, sizeof(cg_halo) * ncopy, cudaMemcpyDeviceToHost);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  }
  const unsigned errw = hw[1];
  cudaFree(big);
  cudaFree(blk.base);
  if (e != cudaSuccess) {
    char msg[200];
    snprintf(msg, sizeof(msg), "cg_fof: %s", cudaGetErrorString(e));
    return cg_set_error_from_lpt(e == cudaErrorMemoryAllocation ? CG_ENOMEM : CG_ECUDA, msg);
  }
  if (errw)
    return cg_set_error_from_lpt(CG_ECUDA, "cg_fof: union-find iteration limit reached");
  *nhalo = nh;
  return CG_OK;
}

// ---------------------------------------------------------------- drop-in
void cg_dropin_error(int code, const char* msg);

namespace {
cg_halo* g_halos = nullptr;
long long g_nhalo = 0;

// move_particles2_min's wrap of a snapshot (move.c:33-41, float add or
// subtract of L once per axis), in place on the device.  Particles it moves
// are listed -- index and new position, up to `cap` -- so that the host copy
// can be patched without downloading the whole snapshot.
__global__ void k_wrap_list(ParticleMinimum* __restrict__ p, long long n, float L,
                            unsigned long long* __restrict__ count, long long cap,
                            long long* __restrict__ idx, float* __restrict__ xs) {
  for (long long i = (long long)blockIdx.x * CG_THREADS + threadIdx.x; i < n;
       i += (long long)gridDim.x * CG_THREADS) {
    float x[3];
    bool moved = false;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      x[k] = p[i].x[k];
      if (x[k] < 0.0f) {
        x[k] = __fadd_rn(x[k], L);
        moved = true;
      } else if (x[k] >= L) {
        x[k] = __fsub_rn(x[k], L);
        moved = true;
      }
    }
    if (!moved) continue;
#pragma unroll
    for (int k = 0; k < 3; k++) p[i].x[k] = x[k];
    const unsigned long long slot = atomicAdd(count, 1ULL);
    if ((long long)slot < cap) {
      idx[slot] = i;
#pragma unroll
      for (int k = 0; k < 3; k++) xs[3 * slot + k] = x[k];
    }
  }
}

// Wrap the device snapshot d (n particles, after the work on st) and bring
// the host copy h to the same positions.
cudaError_t wrap_device_and_host(ParticleMinimum* d, ParticleMinimum* h, long long n, float L,
                                 cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  const long long cap = n < (1LL << 20) ? n : (1LL << 20);
  unsigned long long* d_count = nullptr;
  long long* d_idx = nullptr;
  float* d_x = nullptr;
  cudaError_t e = cudaMalloc(&d_count, sizeof(unsigned long long));
  if (e == cudaSuccess) e = cudaMalloc(&d_idx, sizeof(long long) * cap);
  if (e == cudaSuccess) e = cudaMalloc(&d_x, sizeof(float) * 3 * cap);
  if (e == cudaSuccess) e = cudaMemsetAsync(d_count, 0, sizeof(unsigned long long), st);
  if (e == cudaSuccess) {
    prof_mark(st, CG_ST_WRAP);
    k_wrap_list<<<cg_grid(n, 16), CG_THREADS, 0, st>>>(d, n, L, d_count, cap, d_idx, d_x);
    e = cudaGetLastError();
  }
  unsigned long long moved = 0;
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(&moved, d_count, sizeof(moved), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaSuccess && moved > 0) {
    if ((long long)moved <= cap) {
      long long* idx = (long long*)malloc(sizeof(long long) * moved);
      float* xs = (float*)malloc(sizeof(float) * 3 * moved);
      if (!idx || !xs) e = cudaErrorMemoryAllocation;
      if (e == cudaSuccess)
        e = cudaMemcpy(idx, d_idx, sizeof(long long) * moved, cudaMemcpyDeviceToHost);
      if (e == cudaSuccess)
        e = cudaMemcpy(xs, d_x, sizeof(float) * 3 * moved, cudaMemcpyDeviceToHost);
      if (e == cudaSuccess)
        for (unsigned long long j = 0; j < moved; j++)
          memcpy(h[idx[j]].x, xs + 3 * j, sizeof(float) * 3);
      free(idx);
      free(xs);
    } else {
      e = cudaMemcpy(h, d, sizeof(ParticleMinimum) * n, cudaMemcpyDeviceToHost);
    }
  }
  cudaFree(d_count);
  cudaFree(d_idx);
  cudaFree(d_x);
  return e;
}
}  // namespace

extern "C" size_t fof_calc_memory(const int np_alloc, const int nc) {
  (void)np_alloc;
  (void)nc;
  return 0;   // the GPU finder needs none of the caller's arena
}

extern "C" void fof_init(const int np_alloc, const int nc, void* mem, size_t mem_size) {
  (void)np_alloc;
  (void)nc;
  (void)mem;
  (void)mem_size;
}

extern "C" void fof_find_halos(Snapshot* snapshot, const float ll) {
  if (!snapshot || !(snapshot->boxsize > 0.0f) || snapshot->np_local < 0 ||
      (snapshot->np_local > 0 && !snapshot->p)) {
    cg_dropin_error(7000, "fof_find_halos: bad snapshot");
    return;
  }
  const float L = snapshot->boxsize;
  const int n = snapshot->np_local;
  const long long cap = n / 32 + 1;   // halos hold at least 32 particles each
  cg_halo* h = (cg_halo*)realloc(g_halos, sizeof(cg_halo) * cap);
  if (!h) {
    cg_dropin_error(7050, "Not enough space for halo");
    return;
  }
  g_halos = h;
  g_nhalo = 0;
  // the snapshot on the device: the copy cola_set_snapshot left, or an upload
  cudaStream_t st = 0;
  ParticleMinimum* d = dropin_device_snapshot(snapshot, &st);
  ParticleMinimum* own = nullptr;
  cudaError_t e = cudaSuccess;
  if (!d && n > 0) {
    e = cudaMalloc(&own, sizeof(ParticleMinimum) * n);
    if (e == cudaSuccess)
      e = cudaMemcpy(own, snapshot->p, sizeof(ParticleMinimum) * n, cudaMemcpyHostToDevice);
    d = own;
    st = 0;
  }
  // move_particles2_min (fof.c:1042): one-shot wrap into the box, in place,
  // on both copies
  if (e == cudaSuccess) e = wrap_device_and_host(d, snapshot->p, n, L, st);
  long long nh = 0;
  const int rc = e == cudaSuccess ? cg_fof(d, n, L, ll, 32, g_halos, cap, &nh) : CG_ECUDA;
  cudaFree(own);
  if (rc != CG_OK) {
    cg_dropin_error(7050, "fof_find_halos failed");
    return;
  }
  g_nhalo = nh;
}

extern "C" void fof_write_halos(char filename[]) {
  FILE* fp = fopen(filename, "w");
  if (!fp) {
    char msg[512];
    snprintf(msg, sizeof(msg), "Error: Unable to write halo to file %s", filename);
    cg_dropin_error(8110, msg);
    return;
  }
  for (long long i = 0; i < g_nhalo; i++) {
    const cg_halo& h = g_halos[i];
    fprintf(fp, "%d %e %e %e %e %e %e\n", h.nfof, h.x[0], h.x[1], h.x[2], h.v[0], h.v[1],
            h.v[2]);
  }
  fclose(fp);
}
