// Context, device arena, the shared certification tail and the C ABI entry
// points of libhdgpu.so (declared in include/hd_gpu.h).
//
// The C ABI replaces the reference's algorithm seam
// HausdorffDistance<COORD_T,N_DIMS>::CalculateDistance
// (src/hausdorff_distance.h:21-32) and hd_exec's variant factory and
// repeat loop (src/run_hausdorff_distance.cu:220-357).  Errors never escape
// as exceptions (the reference aborts through glog CHECK or throws
// hd::Exception from CUDA_CHECK, utils/exception.h:151-160); every call
// returns an hd_status and keeps a message for hd_last_error.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <new>
#include <numeric>
#include <string>

#include "hd_common.cuh"
#include "hd_internal.h"
#include "hd_tuning.h"

namespace hdg {

hd_status fail(Ctx& c, hd_status s, const std::string& msg) {
  if (c.last_error.empty()) c.last_error = msg;
  return s;
}

hd_status cuda_fail(Ctx& c, cudaError_t e, const char* what) {
  std::string m = std::string(what) + ": " + cudaGetErrorString(e);
  if (e == cudaErrorMemoryAllocation) return fail(c, HD_ERR_OOM, m);
  if (e == cudaErrorNoKernelImageForDevice || e == cudaErrorNoDevice ||
      e == cudaErrorInsufficientDriver)
    return fail(c, HD_ERR_NO_DEVICE, m);
  return fail(c, HD_ERR_CUDA, m);
}

hd_status ensure(Ctx& c, BufSlot slot, size_t bytes, void** out) {
  DevBuf& b = c.bufs[slot];
  if (bytes == 0) bytes = 16;
  if (b.bytes < bytes) {
    if (b.p) {
      cudaError_t e = cudaStreamSynchronize(c.stream);
      if (e != cudaSuccess) return cuda_fail(c, e, "sync before realloc");
      cudaFree(b.p);
      b.p = nullptr;
      b.bytes = 0;
    }
    // Grow geometrically so that repeated solves of slightly larger inputs
    // do not reallocate every call.
    size_t want = std::max(bytes, b.bytes + b.bytes / 4);
    ++c.buf_gen;
    auto grow = [&](size_t n) {
      return c.no_room[slot] ? cudaErrorMemoryAllocation : cudaMalloc(&b.p, n);
    };
    cudaError_t e = grow(want);
    if (e != cudaSuccess) {
      (void) cudaGetLastError();
      e = grow(bytes);
      DevBuf& filter = c.bufs[kBufCells];
      if (e != cudaSuccess && slot != kBufCells && !c.cells_live && filter.p) {
        // The cell filter's bitmaps and lists are not needed any more: their
        // room goes to the index (or to the scan, which then takes its own seeds).
        (void) cudaGetLastError();
        if ((e = cudaStreamSynchronize(c.stream)) != cudaSuccess)
          return cuda_fail(c, e, "sync before realloc");
        cudaFree(filter.p);
        filter = DevBuf{};
        c.cell_seeds[0] = c.cell_seeds[1] = CellSeeds{};
        e = grow(bytes);
      }
      if (e != cudaSuccess) {
        (void) cudaGetLastError();
        b.p = nullptr;
        if (c.no_room[slot]) --c.no_room[slot];
        return fail(c, HD_ERR_OOM,
                    "device allocation of " + std::to_string(bytes) + " bytes failed");
      }
      want = bytes;
    }
    b.bytes = want;
  }
  *out = b.p;
  return HD_OK;
}

void release(Ctx& c, BufSlot slot) {
  DevBuf& b = c.bufs[slot];
  if (!b.p) return;
  cudaStreamSynchronize(c.stream);
  cudaFree(b.p);
  b = DevBuf{};
  ++c.buf_gen;
}

hd_status after_launch(Ctx& c, const char* what) {
  ++c.launches;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(c, e, what);
  return HD_OK;
}

hd_status ensure_side(Ctx& c) {
  if (c.batch_side) return HD_OK;
  cudaError_t e;
  if ((e = cudaStreamCreateWithFlags(&c.batch_side, cudaStreamNonBlocking)) != cudaSuccess ||
      (e = cudaEventCreateWithFlags(&c.batch_fork, cudaEventDisableTiming)) != cudaSuccess ||
      (e = cudaEventCreateWithFlags(&c.batch_join, cudaEventDisableTiming)) != cudaSuccess)
    return cuda_fail(c, e, "side stream");
  return HD_OK;
}

hd_status ensure_index_side(Ctx& c) {
  if (c.index_side) return HD_OK;
  cudaError_t e;
  if ((!c.index_join &&
       (e = cudaEventCreateWithFlags(&c.index_join, cudaEventDisableTiming)) != cudaSuccess) ||
      (e = cudaStreamCreateWithFlags(&c.index_side, cudaStreamNonBlocking)) != cudaSuccess)
    return cuda_fail(c, e, "index stream");
  return HD_OK;
}

DevScalars* scalars(Ctx& c, int dir) {
  return reinterpret_cast<DevScalars*>(c.bufs[kBufScalars].p) + dir;
}

void mark(Ctx& c, int k) {
  if (!c.timing || k < 0 || k >= 12) return;
  cudaEventRecord(c.ev[c.ev_base + k], c.stream);
}

static void mark_abs(Ctx& c, int idx) {
  if (c.timing) cudaEventRecord(c.ev[idx], c.stream);
}

uint64_t pick_multiplier(uint64_t n, uint64_t seed) {
  if (n <= 2) return 1;
  // Near n / golden ratio, nudged by the seed, then moved to the next value
  // coprime with n so that j -> j*mul mod n is a bijection.
  uint64_t m = (uint64_t) ((double) n * 0.6180339887498949) + (seed % 97) * 2 + 1;
  m %= n;
  if (m == 0) m = 1;
  while (std::gcd(m, n) != 1) m = (m + 1) % n ? (m + 1) % n : 1;
  return m;
}

namespace {

__global__ void k_init_scalars(DevScalars* sc, int n) {
  int i = threadIdx.x;
  if (i < n) {
    DevScalars z;
    memset(&z, 0, sizeof(z));
    z.min_key = ~0ull;
    for (int s = 0; s < 2; ++s)
      for (int d = 0; d < 4; ++d) {
        z.mbr_ord[s][0][d] = 0xFFFFFFFFu;  // lower corner: atomicMin target
        z.mbr_ord[s][1][d] = 0u;           // upper corner: atomicMax target
      }
    sc[i] = z;
  }
}

__global__ void k_restart(DevScalars* sc) {
  sc->min_key = ~0ull;
  sc->next = sc->pairs = sc->nodes = sc->leaves = 0ull;
  sc->heavy_count = sc->heavy_mark = 0u;
}

// Exact argmin over B for the certifying A point.  Scans the caller's B in
// its own order so that ib is the caller's index; among equal squared
// distances the lowest index wins (atomicMin on (d2 bits, index)).
__global__ void k_argmin(const float* __restrict__ A, const float* __restrict__ B,
                         uint64_t nB, int D, DevScalars* sc) {
  chain_wait();
  const unsigned long long key = sc->max_key;
  const uint32_t ia = unpack_max_index(key);
  if (key == 0 || ia == kInvalid) return;  // no row has completed
  float a[4] = {0, 0, 0, 0};
  const bool small = D <= 4;
  const bool vec = D > 4 && (D % 4) == 0 && ((reinterpret_cast<uintptr_t>(A) & 15) == 0) &&
                   ((reinterpret_cast<uintptr_t>(B) & 15) == 0);
  if (small)
    for (int k = 0; k < D; ++k) a[k] = A[(uint64_t) ia * D + k];
  unsigned long long best = ~0ull;
  const uint64_t tid = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x;
  const uint64_t stride = (uint64_t) gridDim.x * blockDim.x;
  uint64_t first = 0;
  if (D == 3 && ((reinterpret_cast<uintptr_t>(B) & 15) == 0)) {
    // Four 3-D points per three 16-byte loads.
    const float4* B4 = reinterpret_cast<const float4*>(B);
    const uint64_t groups = nB / 4;
    for (uint64_t g = tid; g < groups; g += stride) {
      const float4 f0 = B4[3 * g], f1 = B4[3 * g + 1], f2 = B4[3 * g + 2];
      const float d0 = d2_3(a[0], a[1], a[2], f0.x, f0.y, f0.z);
      const float d1 = d2_3(a[0], a[1], a[2], f0.w, f1.x, f1.y);
      const float e2 = d2_3(a[0], a[1], a[2], f1.z, f1.w, f2.x);
      const float d3 = d2_3(a[0], a[1], a[2], f2.y, f2.z, f2.w);
      unsigned long long k0 = pack_min(d0, (uint32_t) (4 * g));
      unsigned long long k1 = pack_min(d1, (uint32_t) (4 * g + 1));
      unsigned long long k2 = pack_min(e2, (uint32_t) (4 * g + 2));
      unsigned long long k3 = pack_min(d3, (uint32_t) (4 * g + 3));
      k0 = k1 < k0 ? k1 : k0;
      k2 = k3 < k2 ? k3 : k2;
      k0 = k2 < k0 ? k2 : k0;
      best = k0 < best ? k0 : best;
    }
    first = groups * 4;
  } else if (D == 2 && ((reinterpret_cast<uintptr_t>(B) & 15) == 0)) {
    const float4* B4 = reinterpret_cast<const float4*>(B);
    const uint64_t groups = nB / 2;
    for (uint64_t g = tid; g < groups; g += stride) {
      const float4 f = B4[g];
      unsigned long long k0 = pack_min(d2_2(a[0], a[1], f.x, f.y), (uint32_t) (2 * g));
      unsigned long long k1 = pack_min(d2_2(a[0], a[1], f.z, f.w), (uint32_t) (2 * g + 1));
      k0 = k1 < k0 ? k1 : k0;
      best = k0 < best ? k0 : best;
    }
    first = groups * 2;
  }
  for (uint64_t j = first + tid; j < nB; j += stride) {
    float d2;
    if (D == 2) {
      d2 = d2_2(a[0], a[1], B[2 * j], B[2 * j + 1]);
    } else if (D == 3) {
      d2 = d2_3(a[0], a[1], a[2], B[3 * j], B[3 * j + 1], B[3 * j + 2]);
    } else if (vec) {
      // Same left-to-right formula, 16-byte loads.
      const float4* b4 = reinterpret_cast<const float4*>(B + j * D);
      const float4* a4 = reinterpret_cast<const float4*>(A + (uint64_t) ia * D);
      float s = 0.0f;
      for (int k4 = 0; k4 < D / 4; ++k4) {
        const float4 b = __ldg(b4 + k4), a = __ldg(a4 + k4);
        const float d0 = __fsub_rn(a.x, b.x), d1 = __fsub_rn(a.y, b.y);
        const float dd2 = __fsub_rn(a.z, b.z), d3 = __fsub_rn(a.w, b.w);
        s = k4 == 0 ? __fmul_rn(d0, d0) : __fadd_rn(s, __fmul_rn(d0, d0));
        s = __fadd_rn(s, __fmul_rn(d1, d1));
        s = __fadd_rn(s, __fmul_rn(dd2, dd2));
        s = __fadd_rn(s, __fmul_rn(d3, d3));
      }
      d2 = s;
    } else {
      d2 = d2_n(A + (uint64_t) ia * D, B + j * D, D);
    }
    unsigned long long k = pack_min(d2, (uint32_t) j);
    best = k < best ? k : best;
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    unsigned long long v = __shfl_xor_sync(0xFFFFFFFFu, best, o);
    best = v < best ? v : best;
  }
  if ((threadIdx.x & 31) == 0 && best != ~0ull) atomicMin(&sc->min_key, best);
}

__global__ void k_finalize(const float* __restrict__ A, const float* __restrict__ B,
                           int D, DevScalars* sc) {
  chain_wait();
  finalize_scalars(A, B, D, sc);
}

}  // namespace

hd_status certify(Ctx& c, const DirInput& in) {
  mark(c, 5);
  DevScalars* sc = scalars(c, in.dir);
  int grid = (int) std::min<uint64_t>((in.nB + 255) / 256, (uint64_t) c.num_sms * 4);
  grid = std::max(grid, 1);
  launch_next(c.stream, true, k_argmin, grid, 256, in.A, in.B, in.nB, in.dims, sc);
  hd_status s = after_launch(c, "argmin");
  if (s != HD_OK) return s;
  launch_next(c.stream, true, k_finalize, 1, 1, in.A, in.B, in.dims, sc);
  return after_launch(c, "finalize");
}

namespace {

// The same argmin over the cell filter's targets (x, y, z, row).
template <int D>
__global__ void k_argmin_left(const float* __restrict__ A, const float4* __restrict__ T, uint32_t n,
                              DevScalars* sc) {
  const unsigned long long key = sc->max_key;
  if (key == 0 || unpack_max_index(key) == kInvalid) return;  // no row has completed
  const float* q = A + (uint64_t) unpack_max_index(key) * D;
  const float4 a = make_float4(q[0], q[1], D == 3 ? q[2] : 0.0f, 0.0f);
  unsigned long long best = ~0ull;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float4 t = T[i];
    const unsigned long long k = pack_min(d2_pt<D>(a, t), __float_as_uint(t.w));
    best = k < best ? k : best;
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    unsigned long long v = __shfl_xor_sync(0xFFFFFFFFu, best, o);
    best = v < best ? v : best;
  }
  if ((threadIdx.x & 31) == 0 && best != ~0ull) atomicMin(&sc->min_key, best);
}

}  // namespace

hd_status certify_left(Ctx& c, const DirInput& in, const CellsLeft& left) {
  mark(c, 5);
  DevScalars* sc = scalars(c, in.dir);
  const int grid = (int) std::max<uint64_t>(
      1, std::min<uint64_t>((left.nt + 255) / 256, (uint64_t) c.num_sms * 4));
  if (in.dims == 2)
    k_argmin_left<2><<<grid, 256, 0, c.stream>>>(in.A, left.t, (uint32_t) left.nt, sc);
  else
    k_argmin_left<3><<<grid, 256, 0, c.stream>>>(in.A, left.t, (uint32_t) left.nt, sc);
  hd_status s = after_launch(c, "argmin");
  if (s != HD_OK) return s;
  launch_next(c.stream, true, k_finalize, 1, 1, in.A, in.B, in.dims, sc);
  return after_launch(c, "finalize");
}

// Stream-level forms of the certification tail and the scalar reset, for
// callers that run without a context (hd_solve_eb_noalloc).
cudaError_t certify_on_stream(cudaStream_t st, int num_sms, const float* A, const float* B,
                              uint64_t nB, int dims, DevScalars* sc) {
  int grid = (int) std::min<uint64_t>((nB + 255) / 256, (uint64_t) num_sms * 4);
  grid = std::max(grid, 1);
  k_argmin<<<grid, 256, 0, st>>>(A, B, nB, dims, sc);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  k_finalize<<<1, 1, 0, st>>>(A, B, dims, sc);
  return cudaGetLastError();
}

cudaError_t init_scalars_on_stream(cudaStream_t st, DevScalars* sc, int n) {
  k_init_scalars<<<1, 32, 0, st>>>(sc, n);
  return cudaGetLastError();
}

hd_status init_scalars(Ctx& c) {
  void* p = nullptr;
  hd_status s = ensure(c, kBufScalars, scalars_bytes(), &p);
  if (s != HD_OK) return s;
  k_init_scalars<<<1, 32, 0, c.stream>>>((DevScalars*) p, 2);
  return after_launch(c, "init_scalars");
}

hd_status restart_direction(Ctx& c, int dir) {
  k_restart<<<1, 1, 0, c.stream>>>(scalars(c, dir));
  return after_launch(c, "restart");
}

}  // namespace hdg

using namespace hdg;

namespace {

// Host staging of the two DevScalars.
struct HostScalars {
  DevScalars s[2];
};

hd_status copy_in(Ctx& c, const float* src, uint64_t n, int dims, BufSlot slot,
                  const float** out) {
  void* p = nullptr;
  size_t bytes = (size_t) n * dims * sizeof(float);
  hd_status s = ensure(c, slot, bytes, &p);
  if (s != HD_OK) return s;
  cudaError_t e = cudaMemcpyAsync(p, src, bytes, cudaMemcpyHostToDevice, c.stream);
  if (e != cudaSuccess) return cuda_fail(c, e, "copy inputs to device");
  *out = (const float*) p;
  return HD_OK;
}

hd_status run_direction(Ctx& c, const DirInput& in, int variant, int* used,
                        DirResult* extra) {
  int v = variant;
  hd_status s;
  if (v == HD_VARIANT_AUTO) {
    if ((s = select_variant(c, in, &v)) != HD_OK) return s;
  }
  *used = v;
  switch (v) {
  case HD_VARIANT_EB: return run_eb(c, in);
  case HD_VARIANT_BRUTE: return run_brute(c, in);
  case HD_VARIANT_LBVH: return run_lbvh(c, in);
  case HD_VARIANT_GRID: return run_grid(c, in);
  case HD_VARIANT_BF16: return run_bf16(c, in, extra);
  default: return fail(c, HD_ERR_INVALID_ARG, "unknown variant");
  }
}

// Early-break scans of at least this many points (|A| + |B|, times the
// directions, which share the cost) start from the cell filter's lower bound (30
// us) instead of 152 seed rows scanned in full (20 us).  Without it and with it,
// us, three inputs each: directed 3-D planes 20,000 x 15,000 187 and 163, 2-D
// uniform 19,000 x 18,000 173 and 143, clusters 18,000 x 18,000 134 and 130, 20,000
// x 18,000 from the host 139 and 109, 20,000 x 20,000 126 and 126, 25,000 x 25,000
// 161 and 139, 1M x 1M 2500 and 1020; undirected clusters 15,000 x 15,000 218 and
// 188; below, directed clusters 13,000 x 13,000 108 and 132.
// A scan of a small set is over before that: 20 x 60,000 54 and 83, 100 x 1M 168
// and 602, 1 x 1M 71 and 245.
constexpr uint64_t kSeedMinPoints = 35000, kSeedMinSet = 8000;

// A is sorted while B is copied, before it is known that the sort is of use, when
// it ends with the copy: about 100 us and 35 ps a point, against 19 ps a float over
// the host link.  Sets that the filter gives up, us without the early sort, with it,
// and before there was a filter: 3-D planes 5M + 5M 1745, 1600 and 1638, 15M + 15M
// 4290, 3615 and 3706, jittered copies 10M + 10M 7366, 7000 and 6700.  Where the sort
// outlasts the copy, sets that the filter settles pay for it: clusters 5M + 3.2M 754
// and 862, 2-D with outliers 4M + 4M 846 and 860 (10M clusters 1495 and 1492).
bool sort_first(uint64_t nA, uint64_t nB, int dims) {
  return 19e-6 * (double) nB * dims >= 100.0 + 35e-6 * (double) nA;
}

// LBVH and EB solves launch a fixed kernel sequence with no host read-back
// before the result: the second identical one in a row is captured into a CUDA
// graph and later ones replay it (no per-kernel launch cost).  The index beside the
// cell filter is such a sequence too: planes 100k x 120k directed on the same buffers
// 311 -> 266 us (260 before there was a filter), 600k x 700k 382 -> 343 (338).
template <class F>
hd_status replayed(Ctx& c, const SolveKey& key, F run) {
  const bool same = std::memcmp(key.v, c.solve_key.v, sizeof(key.v)) == 0;
  hd_status s;
  cudaError_t e;
  if (same && c.solve_graph_valid) {
    if ((e = cudaGraphLaunch(c.solve_graph, c.stream)) != cudaSuccess)
      return cuda_fail(c, e, "solve graph launch");
    c.launches += c.solve_graph_launches;
    return HD_OK;
  }
  if (!same || !c.solve_key_seen) {
    if ((s = run()) != HD_OK) return s;
    // The run may have (re)allocated buffers: key the graph on the
    // generation they now have.
    c.solve_key = key;
    c.solve_key.v[9] = c.buf_gen;
    c.solve_key_seen = true;
    c.solve_graph_valid = false;
    return HD_OK;
  }
  // Second identical run: capture it (buffers are already allocated by
  // the first, so the sequence makes no allocation), then launch.
  const uint64_t l0 = c.launches;
  const bool sorted = c.sorted_valid, first = c.first_sorted;
  cudaGraph_t graph = nullptr;
  if ((e = cudaStreamBeginCapture(c.stream, cudaStreamCaptureModeThreadLocal)) != cudaSuccess)
    return cuda_fail(c, e, "begin solve capture");
  s = run();
  e = cudaStreamEndCapture(c.stream, &graph);
  cudaGraphExec_t exec = nullptr;
  if (s == HD_OK && e == cudaSuccess) e = cudaGraphInstantiate(&exec, graph, 0);
  if (graph) cudaGraphDestroy(graph);
  if (s != HD_OK || e != cudaSuccess) {
    // Something in the sequence cannot be captured (for example a buffer
    // that has to grow): nothing ran, so run it directly and stop trying.
    cudaGetLastError();
    c.last_error.clear();
    c.launches = l0;
    c.solve_key_seen = false;
    c.solve_graph_valid = false;
    c.sorted_valid = sorted;
    c.first_sorted = first;
    return run();
  }
  if (c.solve_graph) cudaGraphExecDestroy(c.solve_graph);
  c.solve_graph = exec;
  c.solve_graph_valid = true;
  c.solve_graph_launches = c.launches - l0;
  if ((e = cudaGraphLaunch(c.solve_graph, c.stream)) != cudaSuccess)
    return cuda_fail(c, e, "solve graph launch");
  return HD_OK;
}

hd_status check_status(Ctx& c, const HostScalars& h, int ndir) {
  for (int d = 0; d < ndir; ++d) {
    uint32_t st = h.s[d].status;
    if (st & kErrWaitTimeout)
      return fail(c, HD_ERR_DEVICE_TIMEOUT, "a bounded device wait ran out");
    if (st & kErrQueueOverflow) return fail(c, HD_ERR_CUDA, "device queue overflow");
    if (st & kErrInternal)
      return fail(c, HD_ERR_CUDA, "internal consistency check failed");
  }
  return HD_OK;
}

}  // namespace

extern "C" {

void hd_default_options(hd_options* opt) {
  if (!opt) return;
  memset(opt, 0, sizeof(*opt));
  opt->device = 0;
  opt->variant = HD_VARIANT_AUTO;
  opt->seed = 0;
  opt->sample_rate = 0.01;
  opt->n_points_cell = 8;
  opt->leaf_size = 16;
  opt->eb_only_threshold = 0;
}

hd_status hd_create(hd_ctx** out, const hd_options* opt) {
  if (!out) return HD_ERR_INVALID_ARG;
  *out = nullptr;
  hd_ctx* c = new (std::nothrow) hd_ctx();
  if (!c) return HD_ERR_OOM;
  if (opt)
    c->opt = *opt;
  else
    hd_default_options(&c->opt);
  if (c->opt.leaf_size == 0 || c->opt.leaf_size > 32) c->opt.leaf_size = 16;
  if (c->opt.n_points_cell == 0) c->opt.n_points_cell = 8;
  if (!(c->opt.sample_rate > 0.0)) c->opt.sample_rate = 0.01;
  if (c->opt.batch_small_rows == 0) c->opt.batch_small_rows = tuning().batch_small_rows;
  c->opt.batch_small_rows = std::min<uint32_t>(c->opt.batch_small_rows, 65536);
  if (c->opt.batch_chunk == 0) c->opt.batch_chunk = tuning().batch_chunk;
  c->opt.batch_chunk = std::max<uint32_t>(1, std::min<uint32_t>(c->opt.batch_chunk, 64));
  if (c->opt.batch_window == 0) c->opt.batch_window = tuning().batch_window;
  c->opt.batch_window = std::max<uint32_t>(1, std::min<uint32_t>(c->opt.batch_window, 8));
  if (c->opt.lbvh_budget == 0) c->opt.lbvh_budget = tuning().lbvh_budget;
  // eb_cap_pairs 0: per solve, from |B| (see run_eb_dim).
  int n = 0;
  cudaError_t e = cudaGetDeviceCount(&n);
  if (e != cudaSuccess || n == 0 || c->opt.device < 0 || c->opt.device >= n) {
    (void) cudaGetLastError();
    delete c;
    return HD_ERR_NO_DEVICE;
  }
  c->device = c->opt.device;
  if ((e = cudaSetDevice(c->device)) != cudaSuccess) {
    delete c;
    return HD_ERR_NO_DEVICE;
  }
  cudaDeviceProp prop;
  cudaGetDeviceProperties(&prop, c->device);
  if (prop.major * 10 + prop.minor != 103) {
    // The library carries sm_103a code only.
    delete c;
    return HD_ERR_NO_DEVICE;
  }
  c->num_sms = prop.multiProcessorCount;
  if ((e = cudaStreamCreateWithFlags(&c->own_stream, cudaStreamNonBlocking)) != cudaSuccess) {
    delete c;
    return HD_ERR_CUDA;
  }
  c->stream = c->own_stream;
  for (auto& ev : c->ev) cudaEventCreate(&ev);
  if (cudaMallocHost(&c->host_pinned, 4096) != cudaSuccess) {
    hd_destroy(c);
    return HD_ERR_OOM;
  }
  c->host_pinned_bytes = 4096;
  *out = c;
  return HD_OK;
}

hd_status hd_destroy(hd_ctx* c) {
  if (!c) return HD_ERR_INVALID_ARG;
  cudaSetDevice(c->device);
  if (c->stream) cudaStreamSynchronize(c->stream);
  for (auto& b : c->bufs)
    if (b.p) cudaFree(b.p);
  for (auto& ev : c->ev)
    if (ev) cudaEventDestroy(ev);
  for (auto& gx : c->batch_graphs)
    if (gx) cudaGraphExecDestroy(gx);
  for (auto& ev : c->copy_ev)
    if (ev) cudaEventDestroy(ev);
  if (c->copy_stream) cudaStreamDestroy(c->copy_stream);
  if (c->solve_graph) cudaGraphExecDestroy(c->solve_graph);
  if (c->batch_fork) cudaEventDestroy(c->batch_fork);
  if (c->batch_join) cudaEventDestroy(c->batch_join);
  if (c->batch_side) cudaStreamDestroy(c->batch_side);
  if (c->host_pinned) cudaFreeHost(c->host_pinned);
  if (c->sel_pinned) cudaFreeHost(c->sel_pinned);
  if (c->sel_event) cudaEventDestroy(c->sel_event);
  if (c->cells_event) cudaEventDestroy(c->cells_event);
  if (c->index_side) cudaStreamDestroy(c->index_side);
  if (c->index_join) cudaEventDestroy(c->index_join);
  if (c->batch_pinned) cudaFreeHost(c->batch_pinned);
  if (c->own_stream) cudaStreamDestroy(c->own_stream);
  delete c;
  return HD_OK;
}

hd_status hd_set_stream(hd_ctx* c, void* stream) {
  if (!c) return HD_ERR_INVALID_ARG;
  c->stream = stream ? (cudaStream_t) stream : c->own_stream;
  return HD_OK;
}

hd_status hd_solve(hd_ctx* c, const float* A, uint64_t n_a, const float* B,
                   uint64_t n_b, int n_dims, uint32_t flags, int variant,
                   hd_result* out) {
  if (!c) return HD_ERR_INVALID_ARG;
  c->last_error.clear();
  if (!out || !A || !B) return fail(*c, HD_ERR_INVALID_ARG, "null pointer argument");
  if (n_a == 0 || n_b == 0) return fail(*c, HD_ERR_INVALID_ARG, "empty point set");
  if (n_a >= 0xFFFFFFFFull || n_b >= 0xFFFFFFFFull)
    return fail(*c, HD_ERR_INVALID_ARG, "point sets are limited to 2^32-2 points");
  if (n_dims < 1 || n_dims > 256)
    return fail(*c, HD_ERR_INVALID_ARG, "n_dims must be in [1, 256]");
  if (flags & ~(HD_UNDIRECTED | HD_DEVICE_PTRS | HD_COUNT_PAIRS | HD_TIMING))
    return fail(*c, HD_ERR_INVALID_ARG, "unknown flag bits");
  if (variant < 0) variant = c->opt.variant;
  if (variant > HD_VARIANT_BRUTE)
    return fail(*c, HD_ERR_INVALID_ARG, "unknown variant");
  const bool spatial = variant == HD_VARIANT_GRID || variant == HD_VARIANT_LBVH;
  if (spatial && n_dims != 2 && n_dims != 3)
    return fail(*c, HD_ERR_UNSUPPORTED, "grid and LBVH variants need n_dims 2 or 3");
  if (variant == HD_VARIANT_BF16 && (n_dims % 16) != 0)
    return fail(*c, HD_ERR_UNSUPPORTED, "the BF16 variant needs n_dims % 16 == 0");
  cudaSetDevice(c->device);
  memset(out, 0, sizeof(*out));
  out->hd_ba = -1.0;
  c->timing = (flags & HD_TIMING) != 0;
  c->sorted_valid = c->first_sorted = c->first_running = false;
  c->boxes_known = false;
  c->cells_live = false;
  c->ev_base = 0;
  c->last_p80[0] = c->last_p80[1] = 0.0;
  c->last_mean[0] = c->last_mean[1] = 0.0;
  c->last_outside[0] = c->last_outside[1] = 0.0;
  c->seeded[0] = c->seeded[1] = false;
  c->cell_seeds[0] = c->cell_seeds[1] = CellSeeds{};
  c->last_skew[0] = c->last_skew[1] = 0.0;

  hd_status s;
  struct Join {  // whatever ends the call, its stream is behind an early sort
    Ctx& c;
    ~Join() {
      join_first(c);
      c.first_sorted = false;
    }
  } join{*c};
  const float* dA = A;
  const float* dB = B;
  mark_abs(*c, 24);  // start of the whole call (copies included)
  const bool undirected = (flags & HD_UNDIRECTED) != 0;
  // Small sets that take the early-break scan by their sizes or by name (with
  // its deferral cap left to the table).
  bool small = small_apply(n_a, n_b, n_dims) && c->opt.eb_cap_pairs == 0;
  if (small && variant != HD_VARIANT_EB) {
    int va = variant, vb = variant;
    small = variant == HD_VARIANT_AUTO && select_variant_by_size(*c, n_a, n_b, n_dims, &va) &&
            va == HD_VARIANT_EB && select_variant_by_size(*c, n_b, n_a, n_dims, &vb);
  }
  // The cell filter runs before the indexes (not before an early-break scan,
  // which eb_only_threshold may ask for).  It does not wait for the selector:
  // its kernels follow the sample's, and the host evaluates the sample while
  // they run.
  bool cells = !small && cells_apply(*c, n_a, n_b, n_dims, undirected) &&
               (variant == HD_VARIANT_LBVH ||
                (variant == HD_VARIANT_AUTO && c->opt.eb_only_threshold == 0));
  if (!small && (s = init_scalars(*c)) != HD_OK) return s;
  if (!(flags & HD_DEVICE_PTRS)) {
    // An undirected solve known (from the sizes alone) to take the LBVH in
    // both directions sorts A while B is still being copied; one that the cell
    // filter takes first as well, in case the index follows.
    int v0 = variant, v1 = variant;
    bool known = variant != HD_VARIANT_AUTO;
    if (!known)
      known = select_variant_by_size(*c, n_a, n_b, n_dims, &v0) &&
              select_variant_by_size(*c, n_b, n_a, n_dims, &v1);
    const bool index = undirected && known && v0 == HD_VARIANT_LBVH && v1 == HD_VARIANT_LBVH &&
                       n_a + n_b >= kSplitMinPoints;
    if (index && !cells) {
      if ((s = spatial_upload_sort(*c, A, n_a, B, n_b, n_dims, &dA, &dB)) != HD_OK) return s;
    } else if (index && sort_first(n_a, n_b, n_dims)) {
      if ((s = spatial_upload_first(*c, A, n_a, B, n_b, n_dims, &dA, &dB)) != HD_OK) return s;
    } else {
      if ((s = copy_in(*c, A, n_a, n_dims, kBufA, &dA)) != HD_OK) return s;
      if ((s = copy_in(*c, B, n_b, n_dims, kBufB, &dB)) != HD_OK) return s;
    }
  }
  const bool count = (flags & HD_COUNT_PAIRS) != 0;
  const int ndir = undirected ? 2 : 1;
  DirResult ex[2];
  int used[2] = {variant, -1};
  DirInput ins[2];
  for (int d = 0; d < ndir; ++d) {
    ins[d] = DirInput{d == 0 ? dA : dB, d == 0 ? n_a : n_b, d == 0 ? dB : dA,
                      d == 0 ? n_b : n_a, n_dims, d, count, variant == HD_VARIANT_AUTO};
    used[d] = variant;
  }
  bool have_result = false;  // the scalars are already in the pinned staging
  CellsRun cells_state;
  const int level = cells_level(n_a + n_b, n_dims);
  auto filter = [&]() -> hd_status {
    mark(*c, 0);
    const hd_status r = cells_begin(*c, ins, ndir, level, nullptr, false, &cells_state);
    c->boxes_known = cells_state.ran;
    return r;
  };
  if (small) {
    used[0] = used[1] = HD_VARIANT_EB;
  } else if (variant == HD_VARIANT_AUTO) {
    Selection sel;
    c->ev_base = 0;
    if ((s = select_begin(*c, ins, ndir, used, &sel)) != HD_OK) return s;
    for (int d = 0; d < ndir; ++d)
      if (sel.decided[d] && used[d] != HD_VARIANT_LBVH) cells = false;
    if (cells && (s = filter()) != HD_OK) return s;
    if ((s = select_finish(*c, ins, ndir, used, sel)) != HD_OK) {
      cudaStreamSynchronize(c->stream);  // the filter still reads the caller's sets
      return s;
    }
    if (undirected) {
      // The grid only when both directions qualify; otherwise both directions
      // share the fused LBVH launches.
      auto index = [](int v) { return v == HD_VARIANT_GRID || v == HD_VARIANT_LBVH; };
      if (index(used[0]) && index(used[1]) && used[0] != used[1])
        used[0] = used[1] = HD_VARIANT_LBVH;
    }
  } else if (cells && (s = filter()) != HD_OK) {
    return s;
  }
  const bool fused = undirected && used[0] == HD_VARIANT_LBVH && used[1] == HD_VARIANT_LBVH;
  // Kernel sequences that may be replayed (timed solves always launch directly):
  // LBVH and EB ones, by everything that they are made of.
  auto graphable = [&](int v) { return v == HD_VARIANT_LBVH || v == HD_VARIANT_EB; };
  auto solve_key = [&](uint64_t part) {
    return SolveKey{{(uint64_t) dA, (uint64_t) dB, n_a, n_b, (uint64_t) n_dims, flags,
                    (uint64_t) (int64_t) used[0], (uint64_t) (int64_t) used[1],
                     (uint64_t) c->stream, c->buf_gen, part}};
  };
  auto run_all = [&]() -> hd_status {
    hd_status r;
    if (small) {
      c->ev_base = 0;
      for (int k = 0; k <= 3; ++k) mark(*c, k);
      have_result = true;
      r = small_solve(*c, ins, ndir);
      for (int k = 4; k <= 6; ++k) mark(*c, k);
      return r;
    }
    if (cells) {
      // What the cell filter left: lists go to the LBVH; a direction whose
      // answer is too few cells is filtered on a finer grid; sets that it
      // still leaves whole go to the chosen index.  (Lists are used before the
      // next filter run reuses their buffer.)
      CellsLeft left[2];
      DirInput rest[2];
      CellsLeft rest_left[2];
      int n = 0;
      // A direction that the filter's seeds already rule out (and that no finer
      // grid takes) starts on its index beside the filter's other kernels.
      bool off[2], indexed[2] = {false, false};
      float reach[2];
      if ((r = cells_hopeless(*c, ndir, n_dims, cells_state, off, reach)) != HD_OK) return r;
      for (int d = 0; d < ndir; ++d)
        indexed[d] = off[d] && cells_finer(n_a + n_b, n_dims, level, reach[d], c->first_sorted) < 0;
      auto index = [&]() -> hd_status {
        if (indexed[0] && indexed[1] && fused) return run_lbvh_pair(*c, ins[0], ins[1]);
        for (int d = 0; d < ndir; ++d)
          if (indexed[d] && (r = run_direction(*c, ins[d], used[d], &used[d], &ex[d])) != HD_OK)
            return r;
        return HD_OK;
      };
      if (indexed[0] || indexed[1]) {
        // (Part: the directions, and whether A is sorted.)
        const uint64_t part = 2 + (indexed[0] ? 4 : 0) + (indexed[1] ? 8 : 0) + (c->first_sorted ? 16 : 0);
        const bool replay = !c->timing && (!indexed[0] || used[0] == HD_VARIANT_LBVH) &&
                            (!indexed[1] || used[1] == HD_VARIANT_LBVH);
        r = index_beside(*c, [&]() {
          return replay ? replayed(*c, solve_key(part), index) : index();
        });
        c->first_sorted = false;  // a replayed sort of B took it up as well
        if (r == HD_ERR_OOM) {  // after the filter then, with its room
          c->last_error.clear();
          for (int d = 0; d < ndir; ++d)
            if (indexed[d] && (r = restart_direction(*c, d)) != HD_OK) return r;
          indexed[0] = indexed[1] = false;
        } else if (r != HD_OK) {
          return r;
        }
      }
      if (indexed[0] || indexed[1]) {  // else the filter's kernels write the results there
        const cudaError_t e = cudaMemcpyAsync(c->host_pinned, c->bufs[kBufScalars].p,
                                              sizeof(HostScalars), cudaMemcpyDeviceToHost, c->stream);
        if (e != cudaSuccess) return cuda_fail(*c, e, "copy result");
      }
      if ((r = cells_finish(*c, ndir, cells_state, left)) != HD_OK) return r;
      if ((r = join_first(*c)) != HD_OK) return r;
      have_result = cells_state.ran;
      for (int d = 0; d < ndir; ++d) left[d].done |= indexed[d];
      for (int d = 0; d < ndir; ++d)
        if (!left[d].done && left[d].narrowed) {
          rest[n] = ins[d];
          rest_left[n++] = left[d];
        }
      if (n && (r = run_lbvh_left(*c, rest, n, nullptr, rest_left)) != HD_OK) return r;
      bool lists = n > 0;
      n = 0;
      for (int d = 0; d < ndir; ++d) {
        if (left[d].done || left[d].narrowed) continue;
        const int finer = cells_finer(n_a + n_b, n_dims, level, left[d].reach, c->first_sorted);
        CellsLeft fine;
        if (finer >= 0) {
          CellsRun again;
          if ((r = cells_begin(*c, &ins[d], 1, finer, nullptr, true, &again)) != HD_OK) return r;
          if ((r = cells_finish(*c, 1, again, &fine)) != HD_OK) return r;
        }
        if (!fine.done && fine.narrowed) {
          if ((r = run_lbvh_left(*c, &ins[d], 1, nullptr, &fine)) != HD_OK) return r;
          lists = true;
        } else if (!fine.done) {
          rest[n++] = ins[d];
        }
      }
      if (lists || n) have_result = false;
      if (n == 2 && fused) {
        if ((r = run_lbvh_pair(*c, rest[0], rest[1])) != HD_OK) return r;
      } else {
        for (int i = 0; i < n; ++i) {
          const int d = rest[i].dir;
          if ((r = run_direction(*c, rest[i], used[d], &used[d], &ex[d])) != HD_OK) return r;
        }
      }
      mark(*c, 6);
    } else if (fused) {
      // Fused undirected pass: one sort of both sets, both trees and both
      // directions' queries in shared launches.
      c->ev_base = 0;
      mark(*c, 0);
      if ((r = run_lbvh_pair(*c, ins[0], ins[1])) != HD_OK) return r;
      mark(*c, 6);
    } else {
      // The early-break scan starts from the cell filter's lower bound.
      if (used[0] == HD_VARIANT_EB && (n_dims == 2 || n_dims == 3) &&
          (n_a + n_b) * ndir >= kSeedMinPoints && std::min(n_a, n_b) >= kSeedMinSet) {
        if ((r = cells_seed(*c, ins, ndir)) != HD_OK) return r;
      }
      for (int d = 0; d < ndir; ++d) {
        c->ev_base = 12 * d;
        mark(*c, 0);
        if ((r = run_direction(*c, ins[d], used[d], &used[d], &ex[d])) != HD_OK) return r;
        mark(*c, 6);
      }
    }
    return HD_OK;
  };
  const bool eligible = !c->timing && !cells && !small && graphable(used[0]) &&
                        (!undirected || graphable(used[1]));
  s = eligible ? replayed(*c, solve_key(1), run_all) : run_all();
  if (s != HD_OK) return s;
  HostScalars* h = reinterpret_cast<HostScalars*>(c->host_pinned);
  cudaError_t e = cudaSuccess;
  if (!have_result)
    e = cudaMemcpyAsync(h, c->bufs[kBufScalars].p, sizeof(HostScalars), cudaMemcpyDeviceToHost,
                        c->stream);
  if (e != cudaSuccess) return cuda_fail(*c, e, "copy result");
  mark_abs(*c, 25);
  if (!have_result || small || c->timing) e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) return cuda_fail(*c, e, "solve");
  c->small_clean |= small;
  if ((s = check_status(*c, *h, ndir)) != HD_OK) return s;

  const DevScalars& r0 = h->s[0];
  out->hd_ab = std::sqrt(r0.d2_64);
  int win = 0;
  if (undirected) {
    const DevScalars& r1 = h->s[1];
    out->hd_ba = std::sqrt(r1.d2_64);
    // The larger FP32 squared distance decides; ties keep A->B.
    if (r1.d2 > r0.d2) win = 1;
  }
  const DevScalars& w = h->s[win];
  out->hd_f32 = std::sqrt(w.d2);
  out->hd = std::sqrt(w.d2_64);
  out->direction = win;
  out->ia = w.ia;
  out->ib = w.ib;
  out->visited_pairs = r0.pairs + (undirected ? h->s[1].pairs : 0) + ex[0].pairs + ex[1].pairs;
  out->visited_nodes = r0.nodes + (undirected ? h->s[1].nodes : 0);
  out->visited_leaves = r0.leaves + (undirected ? h->s[1].leaves : 0);
  out->variant_used = used[0];
  out->variant_used_ba = undirected ? used[1] : -1;
  out->sample_p80[0] = c->last_p80[0];
  out->sample_p80[1] = undirected ? c->last_p80[1] : 0.0;
  for (int d = 0; d < 2; ++d) {
    out->grid_outside[d] = d < ndir ? c->last_outside[d] : 0.0;
    out->grid_skew[d] = d < ndir ? c->last_skew[d] : 0.0;
    out->sample_mean[d] = d < ndir ? c->last_mean[d] : 0.0;
  }
  out->err_bound = std::max(ex[0].err_bound, ex[1].err_bound);
  out->rechecked = ex[0].rechecked + ex[1].rechecked;
  // LBVH: queries whose packet ran over the traversal budget; EB: points
  // deferred past the per-point pair cap.
  for (int d = 0; d < ndir; ++d)
    if (used[d] == HD_VARIANT_LBVH || used[d] == HD_VARIANT_EB) out->rechecked += h->s[d].heavy_count;
  if (c->timing) {
    float t = 0;
    if (cudaEventElapsedTime(&t, c->ev[24], c->ev[25]) == cudaSuccess) out->ms = t;
    // Phases per direction (event k marks the end of phase k-1):
    // 0 prep/sort, 1 index build, 2 sample or seed, 3 main pass, 4 tail,
    // 5 certify.
    const int from[6] = {0, 1, 2, 3, 4, 5};
    const int to[6] = {1, 2, 3, 4, 5, 6};
    // The fused pass records its phases once, on direction 0's events.
    for (int d = 0; d < (fused || small ? 1 : ndir); ++d)
      for (int p = 0; p < 6; ++p) {
        if (cudaEventElapsedTime(&t, c->ev[12 * d + from[p]], c->ev[12 * d + to[p]]) ==
            cudaSuccess)
          out->phase_ms[p] += t;
        else
          (void) cudaGetLastError();
      }
  }
  return HD_OK;
}

hd_status hd_debug_bf16_rowmin(hd_ctx* c, const float* A, uint64_t n_a, const float* B,
                               uint64_t n_b, int n_dims, float* rowmin_out) {
  if (!c) return HD_ERR_INVALID_ARG;
  c->last_error.clear();
  if (!A || !B || !rowmin_out || n_a == 0 || n_b == 0)
    return fail(*c, HD_ERR_INVALID_ARG, "bad arguments");
  cudaSetDevice(c->device);
  c->timing = false;
  c->sorted_valid = false;
  hd_status s;
  const float *dA = nullptr, *dB = nullptr;
  if ((s = copy_in(*c, A, n_a, n_dims, kBufA, &dA)) != HD_OK) return s;
  if ((s = copy_in(*c, B, n_b, n_dims, kBufB, &dB)) != HD_OK) return s;
  if ((s = init_scalars(*c)) != HD_OK) return s;
  DirInput in{dA, n_a, dB, n_b, n_dims, 0, false};
  return bf16_rowmin_debug(*c, in, rowmin_out);
}

hd_status hd_debug_no_room(hd_ctx* c, int buffer, uint32_t times) {
  if (!c) return HD_ERR_INVALID_ARG;
  switch (buffer) {
  case HD_DEBUG_FILTER: c->no_room[kBufCells] = times; return HD_OK;
  case HD_DEBUG_TREE: c->no_room[kBufNodes0] = times; return HD_OK;
  case HD_DEBUG_TILES: c->no_room[kBufBf16B] = times; return HD_OK;
  default: return HD_ERR_INVALID_ARG;
  }
}

const char* hd_last_error(hd_ctx* c) {
  if (!c) return "null context";
  return c->last_error.c_str();
}

const char* hd_status_string(hd_status s) {
  switch (s) {
  case HD_OK: return "HD_OK";
  case HD_ERR_INVALID_ARG: return "HD_ERR_INVALID_ARG";
  case HD_ERR_OOM: return "HD_ERR_OOM";
  case HD_ERR_DEVICE_TIMEOUT: return "HD_ERR_DEVICE_TIMEOUT";
  case HD_ERR_CUDA: return "HD_ERR_CUDA";
  case HD_ERR_UNSUPPORTED: return "HD_ERR_UNSUPPORTED";
  case HD_ERR_NO_DEVICE: return "HD_ERR_NO_DEVICE";
  }
  return "HD_ERR_UNKNOWN";
}

uint64_t hd_kernel_launches(hd_ctx* c) { return c ? c->launches : 0; }

const char* hd_version(void) { return "hd-gb300 0.1 (sm_103a)"; }

}  // extern "C"
