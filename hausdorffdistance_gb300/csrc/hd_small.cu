// Small 2-D and 3-D sets: the whole solve in one kernel, every pair.
//
// Up to kSmallPairs pairs per direction, all pairs cost less than the launches of
// an early break (src/hd_impl/hausdorff_distance_early_break.h:117-219 needs its seeds,
// its scan, its stragglers and the certification one after the other, twice
// for an undirected solve).  A CTA takes items of a query tile (QPT queries
// per thread) by a chunk of targets in shared memory and lowers the queries'
// minima with one atomicMin per query; the last CTA to finish takes the
// maximum, the certifying pair (lowest rows among ties) and its FP64 distance
// for both directions, writes the result straight to the context's pinned host
// memory, and leaves the minima and its ticket as it found them, so that the
// next solve needs no reset.
//
// One GB300, undirected (before: the early-break kernels): 2-D 2,000 + 2,000 points
// 115 -> 30 us, 4,000 + 5,000 135 -> 40, 12,000 + 10,000 163 -> 85; 3-D 8,000 +
// 9,000 142 -> 81, 12,000 + 10,000 180 -> 111; directed 3-D 12,500 + 12,700 98 -> 87,
// but 15,000 + 16,000 98 either way: there the early break has caught up, so
// kSmallPairs ends between the two.
//
// Bound: latency up to about 10^7 pairs (one launch, one wait), the FP32 pipe
// above it.  Two targets ride in one packed instruction for the differences and
// squares, so a chunk is stored by coordinate.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>

#include "hd_common.cuh"
#include "hd_internal.h"

namespace hdg {
namespace {

constexpr int kSmallThreads = 256;
constexpr uint32_t kChunkMax = 256;      // targets per item, at most
constexpr uint32_t kSmallPoints = 32768; // points per set, at most
constexpr double kSmallPairs = 1.6e8;    // pairs per direction, at most
constexpr int kSmallCtas = 6;            // CTAs per SM

struct SmallDir {
  const float* Q;
  const float* T;
  uint32_t nq, nt;
  uint32_t tiles, chunks;  // items: tiles x chunks
  uint32_t* qmin;          // float bits, all ones between solves
};
struct SmallArgs {
  SmallDir d[2];     // blockIdx.y
  uint32_t chunk;    // targets per item (even)
  uint32_t* ticket;  // per direction, 0 between solves
  DevScalars* out;   // pinned host memory
};

// Squared distances of one query to two targets, bit for bit d2_2 / d2_3.
template <int D>
__device__ __forceinline__ float2 d2_two(const float2* q, float2 x, float2 y, float2 z) {
  // The additions are scalar: a packed one is contracted with its product.
  const float2 dx = sub2_rn(q[0], x), dy = sub2_rn(q[1], y);
  const float2 px = __fmul2_rn(dx, dx), py = __fmul2_rn(dy, dy);
  float2 s = make_float2(__fadd_rn(px.x, py.x), __fadd_rn(px.y, py.y));
  if constexpr (D == 3) {
    const float2 dz = sub2_rn(q[2], z), pz = __fmul2_rn(dz, dz);
    s = make_float2(__fadd_rn(s.x, pz.x), __fadd_rn(s.y, pz.y));
  }
  return s;
}

template <int D, int QPT>
__global__ void __launch_bounds__(kSmallThreads, kSmallCtas) k_small(SmallArgs a) {
  __shared__ __align__(16) float s[D][kChunkMax];
  __shared__ unsigned long long red[kSmallThreads / 32];
  __shared__ bool s_last;
  const int tid = threadIdx.x;
  const SmallDir& d = a.d[blockIdx.y];
  const uint32_t items = d.tiles * d.chunks;
  if (blockIdx.x >= items) return;
  for (uint32_t item = blockIdx.x; item < items; item += gridDim.x) {
    const uint32_t tile = item % d.tiles, t0 = item / d.tiles * a.chunk;
    const uint32_t m = min(a.chunk, d.nt - t0);
    __syncthreads();
    // Targets by coordinate; an odd count repeats the last one.
    for (uint32_t j = tid; j < ((m + 1) & ~1u); j += kSmallThreads) {
      const float* t = d.T + (size_t) (t0 + min(j, m - 1)) * D;
#pragma unroll
      for (int k = 0; k < D; ++k) s[k][j] = t[k];
    }
    float2 q[QPT][D];
    float best[QPT];
#pragma unroll
    for (int u = 0; u < QPT; ++u) {
      const uint32_t e = tile * (kSmallThreads * QPT) + u * kSmallThreads + tid;
      const float* p = d.Q + (size_t) min(e, d.nq - 1) * D;
#pragma unroll
      for (int k = 0; k < D; ++k) q[u][k] = make_float2(p[k], p[k]);
      best[u] = FLT_MAX;
    }
    __syncthreads();
#pragma unroll 8
    for (uint32_t j = 0; j < m; j += 2) {
      const float2 x = *reinterpret_cast<const float2*>(&s[0][j]);
      const float2 y = *reinterpret_cast<const float2*>(&s[1][j]);
      const float2 z = *reinterpret_cast<const float2*>(&s[D - 1][j]);
#pragma unroll
      for (int u = 0; u < QPT; ++u) {
        const float2 v = d2_two<D>(q[u], x, y, z);
        best[u] = fminf(best[u], fminf(v.x, v.y));
      }
    }
#pragma unroll
    for (int u = 0; u < QPT; ++u) {
      const uint32_t e = tile * (kSmallThreads * QPT) + u * kSmallThreads + tid;
      if (e < d.nq) atomicMin(d.qmin + e, __float_as_uint(best[u]));
    }
  }
  __threadfence();
  __syncthreads();
  const uint32_t ctas = min(gridDim.x, items);
  if (tid == 0) s_last = atomicAdd(a.ticket + blockIdx.y, 1u) == ctas - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  auto block_max = [&](unsigned long long v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      const unsigned long long w = __shfl_xor_sync(0xFFFFFFFFu, v, o);
      v = w > v ? w : v;
    }
    if ((tid & 31) == 0) red[tid >> 5] = v;
    __syncthreads();
    v = red[0];
#pragma unroll
    for (int k = 1; k < kSmallThreads / 32; ++k) v = red[k] > v ? red[k] : v;
    __syncthreads();
    return v;
  };
  unsigned long long best = 0;
#pragma unroll 8
  for (uint32_t e = tid; e < d.nq; e += kSmallThreads) {
    const unsigned long long k = pack_max(__uint_as_float(__ldcg(d.qmin + e)), e);
    best = k > best ? k : best;
    d.qmin[e] = 0xFFFFFFFFu;
  }
  best = block_max(best);
  const uint32_t ia = unpack_max_index(best);
  float p[D];
#pragma unroll
  for (int k = 0; k < D; ++k) p[k] = d.Q[(size_t) ia * D + k];
  unsigned long long near = 0;  // complement of the smallest (distance, row)
#pragma unroll 8
  for (uint32_t e = tid; e < d.nt; e += kSmallThreads) {
    const float* t = d.T + (size_t) e * D;
    float v;
    if constexpr (D == 2)
      v = d2_2(p[0], p[1], t[0], t[1]);
    else
      v = d2_3(p[0], p[1], p[2], t[0], t[1], t[2]);
    const unsigned long long k = ~pack_min(v, e);
    near = k > near ? k : near;
  }
  near = ~block_max(near);
  if (tid == 0) {
    DevScalars z;
    z.max_key = best;
    z.min_key = near;
    z.status = 0;
    finalize_scalars(d.Q, d.T, D, &z);
    // The words that the host reads.
    DevScalars* o = a.out + blockIdx.y;
    o->d2_64 = z.d2_64;
    o->d2 = z.d2;
    o->ia = z.ia;
    o->ib = z.ib;
    o->status = z.status;
    o->pairs = (unsigned long long) d.nq * d.nt;
    o->nodes = o->leaves = 0;
    o->heavy_count = 0;
    a.ticket[blockIdx.y] = 0;
    __threadfence_system();
  }
}

}  // namespace

bool small_apply(uint64_t nA, uint64_t nB, int dims) {
  return (dims == 2 || dims == 3) && nA <= kSmallPoints && nB <= kSmallPoints &&
         (double) nA * (double) nB <= kSmallPairs;
}

hd_status small_solve(Ctx& c, const DirInput* ins, int ndir) {
  hd_status s;
  void* buf;
  const size_t bytes = 2 * kSmallPoints * 4 + 256;
  const bool fresh = c.bufs[kBufSmall].bytes < bytes;
  if ((s = ensure(c, kBufSmall, bytes, &buf)) != HD_OK) return s;
  cudaError_t e;
  if (fresh || !c.small_clean) {
    // The kernel keeps the minima and its ticket ready for the next solve;
    // here they are made so, at first and after a solve that failed.
    if ((e = cudaMemsetAsync(buf, 0xFF, bytes, c.stream)) != cudaSuccess ||
        (e = cudaMemsetAsync((char*) buf + bytes - 256, 0, 256, c.stream)) != cudaSuccess)
      return cuda_fail(c, e, "memset small");
  }
  c.small_clean = false;
  SmallArgs a{};
  a.ticket = (uint32_t*) ((char*) buf + bytes - 256);
  a.out = (DevScalars*) c.host_pinned;
  // Two queries per thread once that still leaves every SM a tile.
  const bool two = std::min(ins[0].nA, ins[0].nB) >= 8192;
  const uint32_t per = kSmallThreads * (two ? 2 : 1);
  uint32_t tiles = 0;
  for (int k = 0; k < ndir; ++k) {
    SmallDir& d = a.d[k];
    d.Q = ins[k].A;
    d.T = ins[k].B;
    d.nq = (uint32_t) ins[k].nA;
    d.nt = (uint32_t) ins[k].nB;
    d.tiles = (d.nq + per - 1) / per;
    d.qmin = (uint32_t*) buf + (size_t) k * kSmallPoints;
    tiles += d.tiles;
  }
  // Chunks so that the items fill the resident CTAs once, or small ones that
  // even out several turns.
  const uint32_t slots = (uint32_t) (c.num_sms * kSmallCtas);
  const uint32_t want = std::max(1u, slots / tiles);
  const uint32_t most = std::max(a.d[0].nt, ndir > 1 ? a.d[1].nt : 0u);
  a.chunk = std::min(kChunkMax, std::max(32u, ((most + want - 1) / want + 1) & ~1u));
  uint32_t items = 0;
  for (int k = 0; k < ndir; ++k) {
    a.d[k].chunks = (a.d[k].nt + a.chunk - 1) / a.chunk;
    items = std::max(items, a.d[k].tiles * a.d[k].chunks);
  }
  const dim3 grid(std::min(items, slots / (unsigned) ndir), ndir);
  void* args[] = {&a};
  static const void* const table[2][2] = {
      {(const void*) k_small<2, 1>, (const void*) k_small<2, 2>},
      {(const void*) k_small<3, 1>, (const void*) k_small<3, 2>}};
  cudaLaunchKernel(table[ins[0].dims == 3][two], grid, dim3(kSmallThreads), args, 0, c.stream);
  return after_launch(c, "small");
}

}  // namespace hdg
