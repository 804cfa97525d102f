// Host-side internals shared by the translation units of libhdgpu.so.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>
#include <vector>

#include "../../include/hd_gpu.h"
#ifdef __CUDACC__
#include "hd_common.cuh"
#endif

namespace hdg {

// Bits of a sorted key that hold the Morton code (bit 30 marks the set in
// the fused sort of small sets).
constexpr uint32_t kCodeMask = (1u << 30) - 1u;
// Code bits below a sorted set's low_bits are left out of its sort (three
// radix passes of 8 bits): the sorted order is exact only above them, so
// every consumer compares codes through the set's mask.  Per-set sorts of
// large sets keep 24 code bits (cells of 2^-8 of the frame per axis in 3-D,
// 2^-12 in 2-D); the fused sort of small sets keeps 23 code bits and the set
// bit 30.  Grid levels never go finer than the sorted bits.
constexpr int kSortLowBitsSplit = 6;
constexpr int kSortLowBitsFused = 7;
__host__ __device__ constexpr uint32_t sorted_mask(int low_bits) {
  return kCodeMask & ~((1u << low_bits) - 1u);
}
// From this many points (|A| + |B|) the two sets are sorted as independent
// chains, each in its own frame (and, for host inputs, A's sort overlaps
// B's copy); below it one fused chain in a common frame has fewer launches
// and aligned Morton orders.
constexpr uint64_t kSplitMinPoints = 4000000;

// Device scalars of one directed solve, zeroed with one memset per solve.
struct DevScalars {
  unsigned long long max_key;     // packed (d2 bits, ~ia) running maximum
  unsigned long long min_key;     // packed (d2 bits, ib) certifying argmin
  unsigned long long next;        // work-queue head (visit index)
  unsigned long long pairs;       // pair distances evaluated
  unsigned long long nodes;       // index nodes / cells visited
  unsigned long long leaves;      // leaf / cell visits (HD_COUNT_PAIRS)
  uint32_t heavy_count;           // deferred points
  uint32_t status;                // error bits (kErr*)
  uint32_t sample_count;
  uint32_t heavy_mark;            // EB: deferred entries already finished
  // Finalised result written by the finalize kernel.
  double d2_64;                   // FP64 squared distance of (ia, ib)
  float d2;                       // FP32 squared distance (max-min)
  uint32_t ia, ib;
  uint32_t pad2;
  uint32_t mbr_ord[2][2][4];      // [set][lo/hi][dim], order-preserving uints
};

#ifdef __CUDACC__
// A launch behind the kernel before it on the stream: chained, its CTAs are on
// their SMs when that kernel's last ones leave, if both begin with chain_wait.
template <class... P, class... T>
cudaError_t launch_next(cudaStream_t st, bool chain, void (*kernel)(P...), dim3 grid, int threads,
                        T... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned) threads);
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = chain ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

// The result words of a direction from its running maximum and argmin.
__device__ __forceinline__ void finalize_scalars(const float* __restrict__ A,
                                                 const float* __restrict__ B, int D,
                                                 DevScalars* sc) {
  const unsigned long long key = sc->max_key;
  const uint32_t ia = unpack_max_index(key);
  if (key == 0 || ia == kInvalid) {  // no row has completed
    sc->status |= kErrInternal;
    return;
  }
  const uint32_t d2bits = (uint32_t) (key >> 32);
  const unsigned long long mk = sc->min_key;
  const uint32_t ib = (uint32_t) (mk & 0xFFFFFFFFull);
  // The argmin over B of A[ia] must reproduce the maximum exactly: it is the
  // same FP32 formula over the same coordinates.
  if ((uint32_t) (mk >> 32) != d2bits) sc->status |= kErrInternal;
  double s = 0.0;
  for (int k = 0; k < D; ++k) {
    double t = (double) A[(uint64_t) ia * D + k] - (double) B[(uint64_t) ib * D + k];
    s += t * t;
  }
  sc->d2_64 = s;
  sc->d2 = __uint_as_float(d2bits);
  sc->ia = ia;
  sc->ib = ib;
}
#endif

// A growable device buffer cached in the context across solves.
struct DevBuf {
  void* p = nullptr;
  size_t bytes = 0;
};

enum BufSlot {
  kBufA = 0,      // caller's A copied to the device (host-pointer solves)
  kBufB,
  kBufPackB,      // packed / permuted B (float2, float4 or padded rows)
  kBufPackA,
  kBufHeavy,      // deferred early-break entries
  kBufScalars,    // DevScalars[2] (one per direction) + spatial frame
  kBufKeys,       // sort keys (scratch)
  kBufKeysAlt,
  kBufVals,       // sort values (scratch)
  kBufValsAlt,
  kBufSorted0,    // Morton-sorted points of set 0 / set 1 (float4 x,y,z,index)
  kBufSorted1,
  kBufCodes0,     // leaf boxes of both sorted sets
  kBufCodes1,
  kBufNodes0,     // LBVH nodes or grid cell table of set 0 / set 1
  kBufNodes1,
  kBufBoxes,      // LBVH build scratch: per-node boxes
  kBufAux,        // parents / flags / cell offsets
  kBufAux2,
  kBufCubTemp,
  kBufSample,
  kBufBf16A,      // split-BF16 operands
  kBufBf16B,
  kBufBf16Open,   // the rows still open after a round, packed together, and the seeds
  kBufNorms,      // BF16 scalars and the squared norms of both sets
  kBufRowMin,
  kBufCand,
  kBufBatch,
  kBufBatch2,
  kBufGroupOffs,  // offsets of a grouped host-input batch (device copy)
  kBufF64A,       // FP64 input path: caller's double A / B on the device
  kBufF64B,
  kBufF64Aux,     // FP64 scalars and candidate lists
  kBufSmall,      // small solves: running minima
  kBufCells,      // cell filter: bitmaps and lists
  kBufLeft,       // sorted points that the cell filter left open
  kBufF64Rows,    // FP64 nearest distance and column of every walked row
  kNumBufs
};

// Cubic Morton frame of a sorted point set (device resident, two of them
// after the two DevScalars in the scalars buffer; frame k belongs to
// c.sorted[k], or frame 0 to both sets when they share a common frame).  A
// query set's points are coded in the target set's frame (frame_code)
// wherever they meet the target's sorted codes.
struct Frame {
  float lo[3], hi[3];
  float scale, extent;  // quantisation scale (cells per unit), max extent
  int bits, dims;       // Morton bits per axis, dimensionality
};

#ifdef __CUDACC__
__device__ __forceinline__ uint32_t morton_spread2(uint32_t x) {  // 16 bits -> even bits
  x &= 0xFFFFu;
  x = (x | (x << 8)) & 0x00FF00FFu;
  x = (x | (x << 4)) & 0x0F0F0F0Fu;
  x = (x | (x << 2)) & 0x33333333u;
  x = (x | (x << 1)) & 0x55555555u;
  return x;
}
__device__ __forceinline__ uint32_t morton_spread3(uint32_t x) {  // 10 bits -> every 3rd bit
  x &= 0x3FFu;
  x = (x | (x << 16)) & 0x030000FFu;
  x = (x | (x << 8)) & 0x0300F00Fu;
  x = (x | (x << 4)) & 0x030C30C3u;
  x = (x | (x << 2)) & 0x09249249u;
  return x;
}
// Cell index of coordinate v along one axis, clamped to the frame.
__device__ __forceinline__ uint32_t frame_quant(float v, float lo, float scale, uint32_t maxq) {
  float q = (v - lo) * scale;
  q = fminf(fmaxf(q, 0.0f), (float) maxq);
  return (uint32_t) q;
}
// Morton code of a point in frame f (points outside the frame clamp to its
// border cells), D = f.dims.  D is a template parameter on purpose: one
// body that chose between the 2-D and 3-D interleave at run time produced
// wrong y bits inside one kernel on sm_103a (nvcc 13.0) while the same
// arithmetic written without the run-time branch was right, so every caller
// is instantiated per dimensionality.
template <int D>
__device__ __forceinline__ uint32_t frame_code(const Frame& f, float x, float y, float z) {
  const uint32_t maxq = (1u << f.bits) - 1u;
  const uint32_t qx = frame_quant(x, f.lo[0], f.scale, maxq);
  const uint32_t qy = frame_quant(y, f.lo[1], f.scale, maxq);
  if constexpr (D == 2) {
    (void) z;
    return morton_spread2(qx) | (morton_spread2(qy) << 1);
  } else {
    const uint32_t qz = frame_quant(z, f.lo[2], f.scale, maxq);
    return morton_spread3(qx) | (morton_spread3(qy) << 1) | (morton_spread3(qz) << 2);
  }
}
#endif

// A point set in Morton order: float4 (x, y, z|0, caller index as bits).
struct SortedSet {
  float4* pts = nullptr;
  uint32_t* codes = nullptr;   // sorted Morton codes (30 bits) in this set's frame
  const Frame* frame = nullptr;  // that frame (device)
  float4* leaf_boxes = nullptr;  // per leaf of leaf_size points: lo, hi
  uint32_t leaf_size = 16;
  uint64_t n = 0;
  int dims = 0;
  const float* src = nullptr;  // device pointer it was sorted from
  int low_bits = kSortLowBitsSplit;                // code bits left out of the sort
  uint32_t mask = sorted_mask(kSortLowBitsSplit);  // the sorted code bits
};

// What the cell filter's seeds left of a direction, on the device (null: they did
// not run), and kSeedWords zeroed words.
struct CellDirState;
constexpr int kSeedWords = 320;
struct CellSeeds {
  const CellDirState* state = nullptr;
  uint32_t* words = nullptr;
};

// What a replayed kernel sequence depends on (word 9: the buffers' generation).
struct SolveKey {
  uint64_t v[11] = {};
};

struct Ctx {
  int device = 0;
  int num_sms = 0;
  hd_options opt{};
  cudaStream_t own_stream = nullptr;
  cudaStream_t stream = nullptr;
  DevBuf bufs[kNumBufs];
  uint32_t no_room[kNumBufs] = {};  // growths yet to be refused (hd_debug_no_room)
  void* host_pinned = nullptr;   // pinned result staging
  size_t host_pinned_bytes = 0;
  void* sel_pinned = nullptr;    // pinned staging of the selector's samples
  size_t sel_pinned_bytes = 0;
  cudaEvent_t sel_event = nullptr;  // after the samples' copy
  bool small_clean = false;  // kBufSmall is ready for a small solve
  bool cells_live = false;  // kernels yet to be enqueued read kBufCells
  cudaEvent_t cells_event = nullptr;  // when the filter's seeds are in pinned memory
  // A direction's index beside the rest of the filter (index_beside).
  cudaStream_t index_side = nullptr;
  cudaEvent_t index_join = nullptr;
  void* batch_pinned = nullptr;  // pinned staging of grouped batch results
  size_t batch_pinned_bytes = 0;
  std::string last_error;
  uint64_t launches = 0;
  // Timing events (HD_TIMING): [12*dir + phase] per direction, 24/25 = the
  // whole call.  Read after the call's final synchronisation.
  cudaEvent_t ev[26] = {};
  bool timing = false;
  int ev_base = 0;
  // Batched solve: instantiated graphs and the launch shapes they were
  // captured for (reused while the shape, buffers and stream are unchanged);
  // several, because a host-input batch runs as a few groups of problems.
  static constexpr int kBatchGraphs = 16;
  cudaGraphExec_t batch_graphs[kBatchGraphs] = {};
  uint64_t batch_keys[kBatchGraphs][17] = {};
  uint64_t batch_stamp[kBatchGraphs] = {};
  uint64_t batch_clock = 0;
  // Host-input batches: group copies run on their own stream, one event per
  // group.
  static constexpr int kBatchGroups = 16;
  cudaStream_t copy_stream = nullptr;
  cudaEvent_t copy_ev[kBatchGroups] = {};
  // Side stream and fork/join events (created on first use): the batch
  // graph's second branch and the LBVH packet positions beside the build.
  cudaStream_t batch_side = nullptr;
  // Single solves: the kernel sequence of an LBVH or EB solve is captured the
  // second time the same shape runs back to back and replayed while it stays
  // the same (pointers, sizes, flags, chosen variants, stream, buffers).
  cudaGraphExec_t solve_graph = nullptr;
  SolveKey solve_key;
  bool solve_key_seen = false;      // solve_key ran once uncaptured
  bool solve_graph_valid = false;   // solve_graph replays solve_key
  uint64_t solve_graph_launches = 0;
  uint64_t buf_gen = 0;             // bumped by every (re)allocation
  cudaEvent_t batch_fork = nullptr, batch_join = nullptr;
  // Per-solve cache: the Morton-sorted sets (slot 0 = call's A, 1 = call's B)
  // are shared by both directions of an undirected solve.
  SortedSet sorted[2];
  bool sorted_valid = false;
  // Set 0 alone is sorted, or being so on index_side (spatial_upload_first), and
  // whether the call's stream has yet to wait for that.
  bool first_sorted = false, first_running = false;
  bool boxes_known = false;  // DevScalars[0].mbr_ord holds the call's boxes
  // Sampler statistic of the last AUTO decision per direction (p80 of the
  // sampled early-break iteration counts; 0 when no sample was drawn).
  double last_p80[2] = {0.0, 0.0};
  double last_mean[2] = {0.0, 0.0};
  // Grid statistics of the last AUTO decision per direction (query fraction
  // outside the target's box, target occupancy skew; 0 when not drawn).
  double last_outside[2] = {0.0, 0.0};
  // The selector's sampled scans already raised this direction's running
  // maximum (the EB variant then skips its own seed pass).
  bool seeded[2] = {false, false};
  // The cell filter's seeds did: the EB variant looks there whether it needs its
  // own.
  CellSeeds cell_seeds[2];
  double last_skew[2] = {0.0, 0.0};
};

// Result of one directed solve, on the host.
struct DirResult {
  float d2 = 0.0f;
  uint32_t ia = 0, ib = 0;
  double d2_64 = 0.0;
  uint64_t pairs = 0, nodes = 0;
  int variant = 0;
  double err_bound = 0.0;
  uint64_t rechecked = 0;
};

// Inputs of one directed solve, resident on the device (row-major floats).
struct DirInput {
  const float* A;
  uint64_t nA;
  const float* B;
  uint64_t nB;
  int dims;
  int dir;      // 0: A->B, 1: B->A (selects the DevScalars slot)
  bool count;
  bool chosen = false;  // AUTO chose the variant
};

// Records the first failure on the context and returns its status.
hd_status fail(Ctx& c, hd_status s, const std::string& msg);
hd_status cuda_fail(Ctx& c, cudaError_t e, const char* what);

// Returns the buffer, growing it (contents not kept) when smaller than bytes.
hd_status ensure(Ctx& c, BufSlot slot, size_t bytes, void** out);
// Gives a buffer back once the stream is through with it.
void release(Ctx& c, BufSlot slot);

// Counts a kernel launch and checks for launch errors.
hd_status after_launch(Ctx& c, const char* what);
// Creates the context's side stream and fork/join events on first use.
hd_status ensure_side(Ctx& c);
hd_status ensure_index_side(Ctx& c);

DevScalars* scalars(Ctx& c, int dir);

// Directed solvers; each leaves its result in DevScalars[dir] (finalized).
hd_status run_eb(Ctx& c, const DirInput& in);
hd_status run_brute(Ctx& c, const DirInput& in);
hd_status run_eb_nd(Ctx& c, const DirInput& in);  // EB for n_dims other than 2, 3
hd_status run_lbvh(Ctx& c, const DirInput& in);
// Both directions of an undirected solve with shared launches.
hd_status run_lbvh_pair(Ctx& c, const DirInput& ab, const DirInput& ba);
hd_status run_grid(Ctx& c, const DirInput& in);
constexpr int kBf16MaxDims = 64;  // tiles are built for rows of 16, 32, 48 and 64
hd_status run_bf16(Ctx& c, const DirInput& in, DirResult* extra);
// Test hook: the BF16 kernel's approximate row minima (no certification).
hd_status bf16_rowmin_debug(Ctx& c, const DirInput& in, float* rowmin_host);
hd_status select_variant(Ctx& c, const DirInput& in, int* variant);
// AUTO for the ndir directions of one call at once (ins[d].dir == d; the
// directions query and target the same two sets): one sample of each set, one
// read-back.  v[d] receives each direction's variant.
hd_status select_variants(Ctx& c, const DirInput* ins, int ndir, int* v);
// The same in two steps: begin enqueues the samples and their copy (pending:
// some direction needs them), finish waits for that copy alone and decides, so
// that kernels enqueued in between run while the host works it out.
struct Selection {
  bool pending = false, decided[2] = {false, false};
  uint32_t k[2], m[2];
  size_t o_it[2], o_smp[2];
};
hd_status select_begin(Ctx& c, const DirInput* ins, int ndir, int* v, Selection* sel);
hd_status select_finish(Ctx& c, const DirInput* ins, int ndir, int* v, const Selection& sel);
// The selector's choice when the sizes alone decide it (no sampling of the
// data); false when it needs the sample pass.
bool select_variant_by_size(const Ctx& c, uint64_t nA, uint64_t nB, int dims, int* variant);

// Small sets (hd_small.cu): the whole solve in one kernel, which writes both
// DevScalars to the pinned staging; no scalars are needed on the device.
bool small_apply(uint64_t nA, uint64_t nB, int dims);
hd_status small_solve(Ctx& c, const DirInput* ins, int ndir);

// FP64 input path (hd_f64.cu) and its hooks into the LBVH solve.
// A row of a list: the caller's row index and its FP32 nearest squared
// distance over the rounded sets (float bits).
struct RowEntry {
  uint32_t row;
  uint32_t min32;
};
// A built tree of one direction's target set: packed nodes, the root's
// index (device), the Morton-sorted points (float4 x, y, z, caller index)
// in leaves of `leaf` points.
struct LbvhTree {
  const float4* nodes;
  const uint32_t* root;
  const float4* pts;
  uint64_t n;
  uint32_t leaf;
};
// run_lbvh_f64 solves the cut sets in FP32 with a listing query pass (a row
// stops only once its minimum is at or below soft_stop(running maximum,
// soft_r[k]); rows that stay open are listed in cand[k] with their FP32
// minima, count in *cand_count[k], at most cand_cap stored), records each
// direction's tree and calls f64_seed after certification.
struct F64Plan {
  LbvhTree tree[2];
  RowEntry* cand[2];
  uint32_t* cand_count[2];
  uint32_t cand_cap;
  float soft_r[2];  // bound on |d(x, y) - d(cut x, cut y)|, rounded up
  void* state;      // the FP64 solve's own data (hd_f64.cu)
};
hd_status run_lbvh_f64(Ctx& c, const DirInput* ins, int count, F64Plan* plan);
hd_status f64_seed(Ctx& c, F64Plan& plan, int count);

// Cell filter (hd_cells.cu).  What it left of one direction: done (its result
// is in DevScalars), or narrowed to the listed queries and targets (float4 x,
// y, z, row), or neither (the whole sets have to be searched).
struct CellsLeft {
  bool done = false, narrowed = false;
  float reach = 0.0f;  // L in cells, 0 if unknown
  const float4* q = nullptr;
  const float4* t = nullptr;
  uint64_t nq = 0, nt = 0;
};
constexpr uint64_t kCellsMinPoints = 40000;
bool cells_apply(const Ctx& c, uint64_t nA, uint64_t nB, int dims, bool undirected);
// The grid (level) to start on, and the one to try again on when the filter
// neither finished nor narrowed a direction (its L: `reach` cells; sorted: a set is
// sorted already); -1: none.
int cells_level(uint64_t points, int dims);
int cells_finer(uint64_t points, int dims, int level, float reach, bool sorted);
// Filters `count` directions: the call's (ins[k].dir == k), or one of them.  With
// a plan, queries are settled by the FP64 listing pass's level, and the pair scan
// leaves the open queries' FP32 minima; no direction is finished here.
// Without a plan the results of finished directions are in the pinned staging
// (DevScalars by direction).  boxes_known: DevScalars[0].mbr_ord already holds
// the sets' boxes.
//   cells_begin enqueues the filter, cells_finish waits for the stream and
//   reads what it left (begin's `ran` false: there was no room for its lists).
// One direction of the filter, on the device (zeroed before each solve).
struct CellDirState {
  uint32_t L2;       // float bits: squared lower bound of h in cell units
  uint32_t off;      // the filter gave up
  uint32_t level;    // L2 as the seeds left it
  uint32_t wide;     // it did so because too much is far
  uint32_t cut;      // a seed met nothing in the rings it looks through
  uint32_t n_occ;    // occupied query cells, about
  uint32_t n_cells;  // cells of open blocks,
  uint32_t n_rim;    // those without a target cell near by (3-D),
  uint32_t n_far;    // and those without one twice as far
  uint32_t n_q;      // open queries
  uint32_t n_t;      // and collected targets (counts may exceed the lists)
  uint32_t done;     // the pair scan finished the direction
  uint32_t ticket;   // its CTAs that are through
  uint32_t scanned;  // with a plan: q_min holds every open query's FP32 minimum
  uint32_t max32;    // and this is the largest (float bits)
};
struct CellsRun {
  bool ran = false;
  bool wrote = false;  // the kernels write the state to the pinned staging
  const CellDirState* state = nullptr;  // device words to read back
  const float4* q[2];
  unsigned long long* q_min[2];  // per open query: (FP32 minimum's bits, target row)
  const float4* t[2];
  uint32_t cap_q[2], cap_t[2];
};
hd_status cells_begin(Ctx& c, const DirInput* ins, int count, int level, const F64Plan* plan,
                      bool boxes_known, CellsRun* run);
// The filter's seeds alone: starts the directions' running maxima at their L and
// leaves c.cell_seeds (none when there was no room).  Takes no read-back.
hd_status cells_seed(Ctx& c, const DirInput* ins, int count);
// The filter settles nothing below an L of this many cell diagonals.
constexpr float kCellsMinReach = 2.0f;
// Waits for the filter's seeds alone: off[k] where it will give direction k up
// (reach[k]: its L in cells), so that the index can be enqueued behind it.  False
// when the filter did not run: there are no seeds to wait behind.
hd_status cells_hopeless(Ctx& c, int count, int dims, const CellsRun& run, bool* off,
                         float* reach);
// Runs `index` on a stream of its own behind the filter's seeds, beside the
// filter's other kernels (which work on the other direction, or return at once);
// the call's stream waits for it.  Planes undirected, 300k x 500k 470 -> 442 us
// against the same behind those kernels, FP64 200k x 300k 524 -> 469.
// When it fails (it may find no room while the filter holds its own) nothing of
// it is left running, and the sorted sets it may have made count for nothing:
// whoever tries again will use their buffers.
template <class F>
hd_status index_beside(Ctx& c, F index) {
  hd_status s = ensure_index_side(c);
  if (s != HD_OK) return s;
  cudaError_t e = cudaStreamWaitEvent(c.index_side, c.cells_event, 0);
  if (e != cudaSuccess) return cuda_fail(c, e, "index stream");
  const cudaStream_t main = c.stream;
  c.stream = c.index_side;
  s = index();
  c.stream = main;
  if (s != HD_OK) {
    c.sorted_valid = c.first_sorted = false;
    cudaStreamSynchronize(c.index_side);
    if (c.batch_side) cudaStreamSynchronize(c.batch_side);
    return s;
  }
  e = cudaEventRecord(c.index_join, c.index_side);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(main, c.index_join, 0);
  return e != cudaSuccess ? cuda_fail(c, e, "index stream") : HD_OK;
}
// Readies a direction's scalars for another try at it (its running maximum and
// the sets' boxes hold).
hd_status restart_direction(Ctx& c, int dir);
hd_status cells_finish(Ctx& c, int count, const CellsRun& run, CellsLeft* left);
// LBVH over what the filter left of `count` directions.
hd_status run_lbvh_left(Ctx& c, const DirInput* ins, int count, F64Plan* plan,
                        const CellsLeft* left);

// Common tail: exact argmin of A[ia] over B, FP64 recomputation, written to
// DevScalars[dir].  Used by every variant.
hd_status certify(Ctx& c, const DirInput& in);

// The same with the argmin over the targets the cell filter collected: every
// target at the certifying row's distance is among them.
hd_status certify_left(Ctx& c, const DirInput& in, const CellsLeft& left);

// Resets both directions' DevScalars (allocating the scalars buffer).
hd_status init_scalars(Ctx& c);

// Context-free forms used by hd_solve_eb_noalloc.
cudaError_t certify_on_stream(cudaStream_t st, int num_sms, const float* A, const float* B,
                              uint64_t nB, int dims, DevScalars* sc);
cudaError_t init_scalars_on_stream(cudaStream_t st, DevScalars* sc, int n);

// Event-based phase timing (HD_TIMING).
void mark(Ctx& c, int phase_event);

uint64_t pick_multiplier(uint64_t n, uint64_t seed);

// Spatial preparation (hd_spatial.cu).
Frame* frame(Ctx& c, int set);
size_t scalars_bytes();
// Morton-sorts the call's two point sets (both, once per hd_solve) and
// returns the ones matching a directed input: *q = in.A, *t = in.B.
hd_status spatial_prepare(Ctx& c, const DirInput& in, const SortedSet** q,
                          const SortedSet** t);
// Host inputs: copies A, sorts it while B is copied on the side stream,
// then sorts B (sets c.sorted, c.sorted_valid); *dA, *dB = device copies.
hd_status spatial_upload_sort(Ctx& c, const float* hA, uint64_t nA, const float* hB, uint64_t nB,
                              int dims, const float** dA, const float** dB);
// Host inputs that the cell filter takes first: copies A and B, and sorts A on the
// index's stream while B arrives, for an index that may follow (plain copies when
// there is no room to sort in).
hd_status spatial_upload_first(Ctx& c, const float* hA, uint64_t nA, const float* hB, uint64_t nB,
                               int dims, const float** dA, const float** dB);
// The call's stream waits for that sort.
hd_status join_first(Ctx& c);
// Boxes of the call's two sets, into DevScalars[0].mbr_ord.
hd_status spatial_boxes(Ctx& c, const DirInput& in);
// Morton-sorts listed points in the common frame of the call's boxes: out[2k]
// = queries, out[2k + 1] = targets (with leaf boxes) of direction k.
hd_status spatial_sort_left(Ctx& c, const CellsLeft* left, int count, int dims, SortedSet* out);
// k random positions in [0, n) (with replacement), k from opt.sample_rate.
hd_status make_sample(Ctx& c, uint64_t n, uint64_t seed, uint32_t* k, uint32_t** list);

}  // namespace hdg

struct hd_ctx : public hdg::Ctx {};
