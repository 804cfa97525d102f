// Cell filter: settles most query points of a 2-D or 3-D solve on bitmaps of
// occupied cells, before anything is sorted.
//
// The reference searches an index for every point of A (its RT passes,
// src/hd_impl/hausdorff_distance_hybrid.h:203-371, shrink the list of open
// points round by round and read per-cell bounds from HdBounds,
// src/geoms/hd_bounds.h:123-156).  Here, too, a query matters only when its
// nearest neighbour may be as far as the answer, and for most that is decided
// by the cells alone:
//
//   occ      both sets set bits in a grid of 2^24 cells over their common box
//            (256^3, or 4096^2 in 2-D; 2 MB a set, so it lives in L2).  A block
//            of 64 cells (4^3, or 8^2) is one 64-bit word, and one bit per block
//            makes the coarse map (32 KB, kept in shared memory where points
//            are looked up).
//   seed     a sample of the query set's cells finds its distance to the
//            target's nearest occupied cell: the largest lower bound is L, and
//            h >= L.
//   blocks   a query block is settled when a near target block lies within L
//            at its far corner; the cells of the others are listed
//   near     a thread per listed cell looks for a target cell within L in the
//            blocks around it; most cells stop here
//   search   the other cells' lower and upper distances to the target's cells
//            (a warp per cell); L rises with the lower ones.
//   mark     cells whose upper distance still exceeds L are marked, and the
//            target cells within that distance of them:
//   collect  the points in marked cells are the open queries and the targets;
//            every nearest neighbour of an open query is among the targets.
//
// What is left is solved exactly: all pairs when they are few (k_cell_solve),
// else the LBVH over the collected points.  A settled query has a target point
// strictly nearer than L <= h and cannot be the maximum, so value, pair and
// direction are those of the full search.  The filter gives up (the whole
// sets go to the index) when L is not several cell diagonals: then the cells
// are too coarse to tell the points apart; and when too much is far to search
// (k_cell_search).
//
// What it gave (undirected, device inputs, one GB300; before: both sets sorted
// and gathered, both trees built, every query walked): 3-D clusters 10M + 10M
// 1.55 -> 0.34 ms, LiDAR planes 50M + 50M 7.7 -> 4.0 ms, 2-D uniform 200k + 200k
// with outliers 0.29 -> 0.12 ms, 4M + 4M 1.03 -> 0.47 ms; directed 1M + 0.7M
// clusters 0.43 -> 0.19 ms.  On 10M + 10M clusters 200 of 20M points stay open.
// What it costs where it gives up, by the cells or late: planes directed 3M + 4M
// 0.77 -> 0.86 ms, 12M + 20M 2.31 -> 2.45, 2-D uniform 21M + 21M 5.5 -> 6.3, shells of
// 1M points 1.36 -> 1.42.
// Its bound there: four passes over the points (box 43 us, cells 83, collect 35)
// at 5 to 6 TB/s, and a chain of eight small kernels (150 us).
//
// Geometry is in units of a cell.  A coordinate's cell unit u = (v - lo) *
// scale carries two roundings relative to at most G cells, under G 2^-23, and
// a gap compares two of them: kPad = G 2^-21 widens every cell by twice that.
// Squared bounds carry kSlack, which covers the roundings of their own arithmetic
// and of the FP32 pair formula (each a few 2^-24).
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <string>
#include <type_traits>

#include "hd_common.cuh"
#include "hd_internal.h"
#include "hd_tuning.h"

namespace hdg {
namespace {

constexpr uint32_t kNoCell = 0xFFFFFFFFu;
constexpr float kSlack = 1.0001f;
constexpr int kSearchWarps = 8, kSearchThreads = 32 * kSearchWarps;
constexpr uint32_t kSeedWarps = 2048;    // sampled words of the coarse map, a cell of each
constexpr float kMinReach = kCellsMinReach;
constexpr uint64_t kOccSplit = 1000000;  // points from which the cells are set in two launches
constexpr int kScanTile = 128;           // targets per item of the pair scan
constexpr uint64_t kScanPairs = 400000000ull;  // pairs per direction the scan takes

// A grid of 2^BITS cells per axis in D dimensions.
template <int D_, int BITS>
struct Geo {
  static constexpr int D = D_;
  static constexpr int kSub = D == 3 ? 2 : 3;              // cells per block axis: 2^kSub
  static constexpr int G = 1 << BITS, S = 1 << kSub;
  static constexpr int NB = G >> kSub;                     // blocks per axis
  static constexpr int kWords = NB / 64;                   // words per row of the coarse map
  static constexpr uint32_t kBlocks = D == 3 ? NB * NB * NB : NB * NB;
  static constexpr uint32_t kCoarse = kBlocks / 32;        // 32-bit words of the coarse map
  static constexpr float kPad = (float) G / (1 << 21);     // see the head of this file
  // Searches read the coarse map from shared memory when it is small.
  static constexpr bool kShared = kCoarse * 4 <= 32768;
  // Rings of rows that a seed looks through at most (it may stop at a lower bound).
  static constexpr int kSeedRings = D == 3 ? 16 : 128;
  // Blocks per axis of a super-block, when it is not.
  static constexpr int kTop = D == 3 ? NB / 64 : NB / 512;
};

struct CellGrid {
  float lo[3];
  float scale, side;
  bool valid;
};

// The grid over the common box of both sets (ord: their boxes as k_mbr2
// leaves them).  Not valid: an empty, unbounded or degenerate box, or
// coordinates whose squares leave the normal range.
template <class Ge>
__device__ __forceinline__ CellGrid cell_grid(const uint32_t (*ord)[2][4]) {
  constexpr int D = Ge::D;
  CellGrid g;
  float ext = 0.0f;
  g.valid = true;
#pragma unroll
  for (int k = 0; k < D; ++k) {
    const float lo = fminf(ord2f(ord[0][0][k]), ord2f(ord[1][0][k]));
    const float hi = fmaxf(ord2f(ord[0][1][k]), ord2f(ord[1][1][k]));
    g.lo[k] = lo;
    if (!(lo >= -1e15f && hi <= 1e15f)) g.valid = false;
    ext = fmaxf(ext, hi - lo);
  }
  if (!(ext >= 1e-12f)) g.valid = false;
  g.scale = (float) (Ge::G - 1) / ext;
  g.side = ext / (float) (Ge::G - 1);
  return g;
}

// A point's cell as block * 64 + bit; kNoCell for a NaN coordinate (such a
// point occupies no cell, and as a query it is never settled).
template <class Ge>
__device__ __forceinline__ uint32_t cell_of(const CellGrid& g, float x, float y, float z) {
  constexpr int D = Ge::D;
  const float u = (x - g.lo[0]) * g.scale, v = (y - g.lo[1]) * g.scale;
  const float w = D == 3 ? (z - g.lo[2]) * g.scale : 0.0f;
  if (!(u >= 0.0f && v >= 0.0f && w >= 0.0f)) return kNoCell;
  const uint32_t cx = min((uint32_t) u, (uint32_t) Ge::G - 1);
  const uint32_t cy = min((uint32_t) v, (uint32_t) Ge::G - 1);
  if constexpr (D == 3) {
    const uint32_t cz = min((uint32_t) w, (uint32_t) Ge::G - 1);
    return (((cz >> 2) * Ge::NB + (cy >> 2)) * Ge::NB + (cx >> 2)) * 64 +
           (((cz & 3) << 4) | ((cy & 3) << 2) | (cx & 3));
  } else {
    return ((cy >> 3) * Ge::NB + (cx >> 3)) * 64 + (((cy & 7) << 3) | (cx & 7));
  }
}

struct CellDir {
  const float* Q;
  const float* T;
  uint64_t nQ, nT;
  int qset;                     // which set the queries are
  unsigned long long* U;        // query cells whose upper distance exceeds L
  unsigned long long* N;        // target cells an open query may need
  unsigned long long* masks;    // per neighbour and place (3-D: of both sizes of cells)
  uint32_t* cells;              // cells of open blocks: block * 64 + bit
  uint32_t* rim;                // those without a target cell near by (3-D),
  uint32_t* far;                // and those without one twice as far,
  float* far_ub;                // their squared upper distances
  float4* q;                    // open queries (x, y, z, row)
  unsigned long long* q_min;    // their nearest (squared distance, target row)
  float4* t;                    // targets
  uint32_t cap_cells, cap_q, cap_t;
  CellDirState* st;
  DevScalars* sc;
  float soft_r;                 // >= 0: settle by soft_stop (the FP64 path's listing)
};

struct CellArgs {
  const uint32_t (*ord)[2][4];
  int swapped;                  // the sets' boxes are in ord in the other order
  unsigned long long* occ[2];
  uint32_t* coarse[2];
  unsigned long long* half[2];  // 3-D: occupied cells of twice the size
  uint32_t* code[2];            // every point's cell (block * 64 + bit), kNoCell for NaN
  uint32_t* any[2];             // blocks with a cell that U or N marks in this set
  uint32_t* top[2];             // and super-blocks with such a block (large maps only)
  int count;                    // directions
  int seeds_only;               // the seeds set the running maxima, nothing follows
  CellDirState* seen;           // pinned host memory: state after the listing of cells,
  CellDirState* left;           // and at the end
  const DevScalars* sc0;        // DevScalars of direction 0
  DevScalars* result;           // pinned host memory: results of finished directions
  CellDir d[2];
};

// The squared distance (cell units) below which a query is settled.
__device__ __forceinline__ float settle_level(const CellDir& d, const CellGrid& g, uint32_t bits) {
  const float L2 = __uint_as_float(bits);
  if (d.soft_r < 0.0f) return L2;
  const float s2 = g.side * g.side;
  return fmaxf(soft_stop(L2 * s2 * 0.9999f, d.soft_r), 0.0f) / s2 * 0.9999f;
}

__device__ __forceinline__ uint32_t ld_relaxed_u32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// A plain load that the compiler knows to be of global memory: through a pointer
// out of CellArgs it takes it for a generic one (the rows of k_cell_blocks at
// 1024^3 cells 397 us, so 360).
__device__ __forceinline__ unsigned long long ld_global_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// One slot per active lane from a counter, with one atomic per warp.
__device__ __forceinline__ uint32_t take_slot(uint32_t* counter) {
  const unsigned act = __activemask();
  const int lane = threadIdx.x & 31, lead = __ffs(act) - 1;
  uint32_t base = 0;
  if (lane == lead) base = atomicAdd(counter, (uint32_t) __popc(act));
  return __shfl_sync(act, base, lead) + __popc(act & ((1u << lane) - 1u));
}

// Occupied cells of both sets (blockIdx.y = set), and every point's cell for
// the passes that follow: they read 4 bytes a point instead of 8 or 12.  Four
// points per thread and step (three 16-byte loads in 3-D, two in 2-D, when the
// array is aligned), their four bitmap words loaded before any is tested.
// Where the points crowd, every SM reads the same few words, and L2 serves
// them one by one.  So the points are taken in two launches: the first, 1/16
// of them, reads the words from L2 and sets nearly every crowded cell; the
// second reads them through L1, which starts empty and therefore holds no word
// from before.  (A word cached in the second launch may lack bits set since:
// then a bit is set once more.)
constexpr uint32_t kOccFirst = 16;

template <class Ge, bool FIRST>
__global__ void __launch_bounds__(256) k_cell_occ(CellArgs a, const float* __restrict__ A,
                                                  uint64_t nA, const float* __restrict__ B,
                                                  uint64_t nB, uint32_t every) {
  chain_wait();
  constexpr int D = Ge::D;
  const CellGrid g = cell_grid<Ge>(a.ord);
  if (!g.valid) return;
  unsigned long long* occ = a.occ[blockIdx.y];
  uint32_t* code = a.code[blockIdx.y];
  const float* P = blockIdx.y ? B : A;
  const uint64_t n = blockIdx.y ? nB : nA;
  const bool vec = (reinterpret_cast<uintptr_t>(P) & 15) == 0;
  // Runs of 32 groups: the first launch takes every `every`-th, the second the
  // others (every = 1: the first takes all).
  const uint64_t groups = (n + 3) / 4, warps = (uint64_t) gridDim.x * blockDim.x / 32;
  for (uint64_t r = (blockIdx.x * (uint64_t) blockDim.x + threadIdx.x) / 32;; r += warps) {
    const uint64_t run = FIRST ? r * every : r + r / (every - 1) + 1;
    if (run * 32 >= groups) break;
    const uint64_t t = run * 32 + (threadIdx.x & 31);
    if (t >= groups) break;
    float v[4 * D];
    const uint32_t m = (uint32_t) min((uint64_t) 4, n - 4 * t);
    if (vec && m == 4) {
      const float4* P4 = reinterpret_cast<const float4*>(P) + D * t;
#pragma unroll
      for (int k = 0; k < D; ++k) {
        const float4 f = __ldcs(P4 + k);
        v[4 * k] = f.x;
        v[4 * k + 1] = f.y;
        v[4 * k + 2] = f.z;
        v[4 * k + 3] = f.w;
      }
    } else {
#pragma unroll
      for (int k = 0; k < 4 * D; ++k) v[k] = k < (int) m * D ? P[4 * D * t + k] : NAN;
    }
    uint32_t c[4];
    unsigned long long w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      c[k] = cell_of<Ge>(g, v[D * k], v[D * k + 1], D == 3 ? v[D * k + 2] : 0.0f);
      w[k] = c[k] == kNoCell ? ~0ull : FIRST ? __ldcg(occ + (c[k] >> 6)) : __ldca(occ + (c[k] >> 6));
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (!((w[k] >> (c[k] & 63)) & 1ull)) atomicOr(occ + (c[k] >> 6), 1ull << (c[k] & 63));
    // A query with a NaN coordinate has no cell: its direction is searched whole.
    if (blockIdx.y < a.count)
      for (uint32_t k = 0; k < m; ++k)
        if (c[k] == kNoCell) a.d[blockIdx.y].st->off = 1u;
    if (m == 4)
      *reinterpret_cast<uint4*>(code + 4 * t) = make_uint4(c[0], c[1], c[2], c[3]);
    else
      for (uint32_t k = 0; k < m; ++k) code[4 * t + k] = c[k];
  }
}

// The place of fine cell (x, y, z) of block (bx, by, bz) in its block of 3-D
// cells of twice the size.
__device__ __forceinline__ uint32_t half_cell(int bx, int by, int bz, int x, int y, int z) {
  return (uint32_t) ((((bz & 1) * 2 + (z >> 1)) << 4) | (((by & 1) * 2 + (y >> 1)) << 2) |
                     ((bx & 1) * 2 + (x >> 1)));
}

// The coarse maps, one bit per block with an occupied cell, and in 3-D the
// occupied cells of twice the size (a block of them covers 2^3 blocks).  The
// query set's cells are counted in a sixteenth of the words; counted in full by
// k_cell_blocks, which reads them again, they cost it 40 us of 400 at 1024^3 cells.
template <class Ge>
__global__ void __launch_bounds__(256) k_cell_coarse(CellArgs a) {
  chain_wait();
  const uint32_t block = blockIdx.x * 256 + threadIdx.x;
  const unsigned long long w = a.occ[blockIdx.y][block];
  const unsigned m = __ballot_sync(0xFFFFFFFFu, w != 0);
  if ((threadIdx.x & 31) == 0) a.coarse[blockIdx.y][block >> 5] = m;
  if (m && ((block >> 5) * 0x9E3779B1u >> 28) == 0 && blockIdx.y < a.count) {
    const uint32_t cells = __reduce_add_sync(0xFFFFFFFFu, (uint32_t) __popcll(w));
    if ((threadIdx.x & 31) == 0) atomicAdd(&a.d[blockIdx.y].st->n_occ, 16 * cells);
  }
  if constexpr (Ge::D == 3) {
    if (w == 0) return;
    const int bx = block % Ge::NB, by = block / Ge::NB % Ge::NB, bz = block / (Ge::NB * Ge::NB);
    unsigned long long h = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int x = i & 1, y = (i >> 1) & 1, z = i >> 2;
      if (w & (0x330033ull << (2 * x + 8 * y + 32 * z)))
        h |= 1ull << half_cell(bx, by, bz, 2 * x, 2 * y, 2 * z);
    }
    constexpr int NB = Ge::NB / 2;
    atomicOr(a.half[blockIdx.y] + (((bz >> 1) * NB + (by >> 1)) * NB + (bx >> 1)), h);
  }
}

// What a search starts from: a box in cell units (a cell, or a point) and the
// block it lies in.
template <class Ge>
struct Probe {
  static constexpr int D = Ge::D;
  float lo[D], hi[D];
  int b[D];
};

template <class Ge>
__device__ __forceinline__ Probe<Ge> probe_cell(uint32_t cell) {
  constexpr int D = Ge::D;
  Probe<Ge> p;
  const uint32_t block = cell >> 6, bit = cell & 63;
  p.b[0] = block % Ge::NB;
  p.b[1] = block / Ge::NB % Ge::NB;
  if constexpr (D == 3) p.b[2] = block / (Ge::NB * Ge::NB);
#pragma unroll
  for (int k = 0; k < D; ++k) {
    const int sub = (bit >> (k * Ge::kSub)) & (Ge::S - 1);
    p.lo[k] = (float) (p.b[k] * Ge::S + sub);
    p.hi[k] = p.lo[k] + 1.0f;
  }
  return p;
}

// The target's box in blocks: nothing of it lies outside.  (Its corners take the
// same steps as the points.)
template <class Ge>
struct BlockBox {
  int lo[Ge::D], hi[Ge::D];
};

template <class Ge>
__device__ __forceinline__ BlockBox<Ge> block_box(const CellArgs& a, const CellGrid& g, int set) {
  BlockBox<Ge> b;
  const uint32_t(*ord)[4] = a.ord[a.swapped ? 1 - set : set];
#pragma unroll
  for (int k = 0; k < Ge::D; ++k) {
    auto block = [&](float v) {
      const float u = (v - g.lo[k]) * g.scale;
      return u >= 0.0f ? (int) (min((uint32_t) u, (uint32_t) Ge::G - 1) >> Ge::kSub) : 0;
    };
    b.lo[k] = block(ord2f(ord[0][k]));
    b.hi[k] = block(ord2f(ord[1][k]));
  }
  return b;
}

// Gap between the probe and block bk along axis k, less the padding.
template <class Ge>
__device__ __forceinline__ float block_gap(const Probe<Ge>& p, int k, int bk) {
  constexpr int S = Ge::S;
  const float c = (float) (bk * S);
  return fmaxf(fmaxf(c - p.hi[k], p.lo[k] - (c + S)) - Ge::kPad, 0.0f);
}

// A row of the coarse map, walked outward from the probe's block (from the box's
// nearest to it).
template <class Ge>
struct RowWalk {
  const unsigned long long* w = nullptr;  // the row's words; null: no row
  int i_right, i_left;
  unsigned long long m_right = 0, m_left = 0;
  float g2;  // the row's squared gap in y (and z)

  __device__ __forceinline__ void open(const unsigned long long* rows, const Probe<Ge>& p,
                                       const BlockBox<Ge>& box, int by, int bz) {
    w = nullptr;
    if (by < box.lo[1] || by > box.hi[1] ||
        (Ge::D == 3 && (bz < box.lo[Ge::D - 1] || bz > box.hi[Ge::D - 1])))
      return;
    g2 = block_gap<Ge>(p, 1, by);
    g2 *= g2;
    if constexpr (Ge::D == 3) {
      const float gz = block_gap<Ge>(p, 2, bz);
      g2 += gz * gz;
    }
    w = rows + (size_t) (Ge::D == 3 ? bz * Ge::NB + by : by) * Ge::kWords;
    // (A row of one word needs no better start than the probe's place.)
    const int bx = Ge::kWords > 1 ? min(max(p.b[0], box.lo[0]), box.hi[0]) : p.b[0];
    i_right = i_left = bx >> 6;
    const unsigned long long m = w[i_right], up = ~0ull << (bx & 63);
    m_right = m & up;
    m_left = m & ~up;
  }
  // The next block along x whose squared gap from the probe is at most reach,
  // nearer side first; -1 when there is none.
  __device__ __forceinline__ int next(const Probe<Ge>& p, float reach) {
    if (w == nullptr || g2 > reach) return -1;
    if constexpr (Ge::kWords > 1) {
      while (!m_right && i_right + 1 < Ge::kWords) {
        const float gx = block_gap<Ge>(p, 0, (i_right + 1) * 64);
        if (gx * gx + g2 > reach) break;
        m_right = w[++i_right];
      }
      while (!m_left && i_left > 0) {
        const float gx = block_gap<Ge>(p, 0, i_left * 64 - 1);
        if (gx * gx + g2 > reach) break;
        m_left = w[--i_left];
      }
    }
    int x = -1;
    float g = INFINITY;
    if (m_right) {
      const int xr = i_right * 64 + __ffsll((long long) m_right) - 1;
      const float gx = block_gap<Ge>(p, 0, xr);
      if (gx * gx + g2 <= reach) {
        x = xr;
        g = gx;
      }
    }
    bool left = false;
    if (m_left) {
      const int xl = i_left * 64 + 63 - __clzll((long long) m_left);
      const float gx = block_gap<Ge>(p, 0, xl);
      if (gx < g && gx * gx + g2 <= reach) {
        x = xl;
        left = true;
      }
    }
    if (x >= 0) {
      if (left)
        m_left &= ~(1ull << (x & 63));
      else
        m_right &= m_right - 1;
    }
    return x;
  }
};

// Square rings of rows around the probe's place, moved into the target's box:
// for a probe far from the box the nearest rows come first as well, and what lies
// between takes no steps.  With rings around the probe itself, to the grid's ends,
// one far cell's search took 290 us, and two 3-D sets of 1M points 3 extents apart
// 16.6 ms undirected (the index alone 0.53, now 0.49).
template <class Ge>
struct Rings {
  int c[2];      // the first row's y (and z)
  float h[2];    // and its gaps
  int last;      // rings past this one lie outside the box

  __device__ __forceinline__ Rings(const Probe<Ge>& p, const BlockBox<Ge>& box) : last(0) {
#pragma unroll
    for (int k = 0; k < Ge::D - 1; ++k) {
      const int lo = box.lo[k + 1], hi = box.hi[k + 1];
      c[k] = min(max(p.b[k + 1], lo), hi);
      h[k] = block_gap<Ge>(p, k + 1, c[k]);
      last = max(last, max(c[k] - lo, hi - c[k]));
    }
  }
  // Squared gap of ring q's rows, at least.
  __device__ __forceinline__ float gap2(int q) const {
    const float r = fmaxf((float) (Ge::S * (q - 1)) - Ge::kPad, 0.0f);
    const float y = h[0] + r;
    if constexpr (Ge::D == 2) return y * y;
    const float z = h[1] + r;
    return fminf(y * y + h[1] * h[1], h[0] * h[0] + z * z);
  }
};

// Visits the target's occupied blocks around a probe, nearest rows first, with
// a whole warp: the rows of blocks (along x) go round the lanes in square rings
// (2-D: alternately above and below), and a lane walks a row's blocks outward
// from the probe while their squared gap is at most `reach()`, then takes its
// next row.  f(block, bx, by, bz) is called for each block.  The lanes take
// one block at a time and step() runs after each, in all lanes, so that what
// one found shortens the others' walks.
// Several warps may share a visit: `j` is the lane's first row, `stride` the
// number of lanes.  WARP = false: each thread visits alone (j = 0, stride = 1).
template <class Ge, bool WARP, class Reach, class F, class Step>
__device__ __forceinline__ void visit_blocks(const Probe<Ge>& p, const BlockBox<Ge>& box,
                                             const Rings<Ge>& rings, const uint32_t* coarse,
                                             int j, int stride, Reach reach, F f, Step step) {
  constexpr int D = Ge::D;
  const unsigned long long* rows = reinterpret_cast<const unsigned long long*>(coarse);
  RowWalk<Ge> row;
  int by = 0, bz = 0, x;
  for (;;) {
    while ((x = row.next(p, reach())) < 0 && j >= 0) {
      int q, dy, dz = 0;  // the row's ring and place
      if constexpr (D == 3) {
        q = (int) ((sqrtf((float) j) + 1.0f) * 0.5f);
        if ((2 * q - 1) * (2 * q - 1) > j && q > 0) --q;
        if (j >= (2 * q + 1) * (2 * q + 1)) ++q;
        const int i = q ? j - (2 * q - 1) * (2 * q - 1) : 0, s = q ? i / (2 * q) : 0;
        const int o = i - s * 2 * q - q;
        dy = s == 0 ? o : s == 1 ? q : s == 2 ? -o : -q;
        dz = s == 0 ? -q : s == 1 ? o : s == 2 ? q : -o;
      } else {
        q = (j + 1) / 2;
        dy = (j & 1) ? q : -q;
      }
      if (q > rings.last || rings.gap2(q) > reach()) {
        j = -1;  // every further row is out of reach
        break;
      }
      by = rings.c[0] + dy;
      bz = D == 3 ? rings.c[1] + dz : 0;
      row.open(rows, p, box, by, bz);
      j += stride;
    }
    if (WARP ? !__any_sync(0xFFFFFFFFu, x >= 0) : x < 0) return;
    if (x >= 0) f((uint32_t) ((D == 3 ? bz * Ge::NB + by : by) * Ge::NB + x), x, by, bz);
    if (WARP) __syncwarp();
    step();
  }
}

// Squared distance from a probe to the far corner of a near occupied block: the
// smallest over the nearest blocks to either side in 81 rows of blocks around
// the rings' first (33 in 2-D), spaced so that they reach about 0.6 of
// sqrt(stop); +inf when nothing lies there.
template <class Ge>
__device__ __forceinline__ float nearest_block(const Probe<Ge>& p, const Rings<Ge>& rings,
                                               const uint32_t* coarse, float stop) {
  constexpr int D = Ge::D;
  const unsigned long long* rows = reinterpret_cast<const unsigned long long*>(coarse);
  const int lane = threadIdx.x & 31;
  const int step = max(1, (int) (sqrtf(stop) * (D == 3 ? 0.15f : 0.04f) / (float) Ge::S));
  float best = INFINITY;
  auto far = [&](int k, int bk) {
    const float c = (float) (bk * Ge::S);
    return fmaxf(c + Ge::S - p.lo[k], p.hi[k] - c) + Ge::kPad;
  };
  constexpr int kRows = D == 3 ? 81 : 33;
#pragma unroll
  for (int j0 = 0; j0 < kRows; j0 += 32) {
    const int j = j0 + lane;
    const int by = rings.c[0] + (D == 3 ? j % 9 - 4 : j - 16) * step;
    const int bz = D == 3 ? rings.c[1] + (j / 9 - 4) * step : 0;
    if (j >= kRows || (uint32_t) by >= Ge::NB || (uint32_t) bz >= Ge::NB) continue;
    float r2 = far(1, by);
    r2 *= r2;
    if constexpr (D == 3) {
      const float z = far(2, bz);
      r2 += z * z;
    }
    const int bx = p.b[0], w0 = bx >> 6;
    const unsigned long long* w = rows + (size_t) (D == 3 ? bz * Ge::NB + by : by) * Ge::kWords;
    const unsigned long long m = w[w0];
    const unsigned long long right = m & (~0ull << (bx & 63)), left = m & ~(~0ull << (bx & 63));
    if (right) {
      const float x = far(0, w0 * 64 + __ffsll((long long) right) - 1);
      best = fminf(best, r2 + x * x);
    }
    if (left) {
      const float x = far(0, w0 * 64 + 63 - __clzll((long long) left));
      best = fminf(best, r2 + x * x);
    }
    if constexpr (Ge::kWords > 1) {
      for (int i = w0 + 1; !right && i < Ge::kWords; ++i)
        if (w[i]) {
          const float x = far(0, i * 64 + __ffsll((long long) w[i]) - 1);
          best = fminf(best, r2 + x * x);
          break;
        }
      for (int i = w0 - 1; !left && i >= 0; --i)
        if (w[i]) {
          const float x = far(0, i * 64 + 63 - __clzll((long long) w[i]));
          best = fminf(best, r2 + x * x);
          break;
        }
    }
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) best = fminf(best, __shfl_xor_sync(0xFFFFFFFFu, best, o));
  return best;
}

// Squared lower and upper distance (cell units) from a probe to the nearest
// of the target's occupied cells, by a warp or by each thread alone; the search
// stops once the upper one is settled against `stop`.  lb2 is +inf when it
// stopped, or found no cell.  With `most` rings it ends after them: lb2 is then
// at most the next ring's gap, ub2 of what it met.
template <class Ge, bool WARP>
__device__ __forceinline__ void cell_search(const Probe<Ge>& p, const BlockBox<Ge>& box,
                                            const unsigned long long* occ,
                                            const uint32_t* coarse, float stop,
                                            float* lb2, float* ub2, int most = Ge::NB,
                                            uint32_t* cut = nullptr) {
  constexpr int D = Ge::D;
  float lb = INFINITY, ub = INFINITY;
  Rings<Ge> rings(p, box);
  if (rings.last > most) {
    lb = rings.gap2(most + 1);
    rings.last = most;
  }
  // The coarse map first: the far corner of the nearest occupied block bounds
  // the search from the start.
  const float cap = WARP ? nearest_block<Ge>(p, rings, coarse, stop) : INFINITY;
  if (cap * kSlack < stop) {
    *lb2 = INFINITY;
    *ub2 = cap;
    return;
  }
  auto warp_min2 = [&]() {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      lb = fminf(lb, __shfl_xor_sync(0xFFFFFFFFu, lb, o));
      ub = fminf(ub, __shfl_xor_sync(0xFFFFFFFFu, ub, o));
    }
  };
  bool stopped = false;
  visit_blocks<Ge, WARP>(
      p, box, rings, coarse, WARP ? threadIdx.x & 31 : 0, WARP ? 32 : 1,
      [&]() { return fminf(lb, cap); },
      [&](uint32_t block, int bx, int by, int bz) {
        unsigned long long m = occ[block];
        while (m) {
          const int t = __ffsll((long long) m) - 1;
          m &= m - 1;
          float l2 = 0.0f, u2 = 0.0f;
#pragma unroll
          for (int k = 0; k < D; ++k) {
            const int b = k == 0 ? bx : k == 1 ? by : bz;
            const float c = (float) (b * Ge::S + ((t >> (k * Ge::kSub)) & (Ge::S - 1)));
            const float gl = fmaxf(fmaxf(c - p.hi[k], p.lo[k] - (c + 1.0f)) - Ge::kPad, 0.0f);
            const float gh = fmaxf(c + 1.0f - p.lo[k], p.hi[k] - c) + Ge::kPad;
            l2 += gl * gl;
            u2 += gh * gh;
          }
          lb = fminf(lb, l2);
          ub = fminf(ub, u2);
        }
      },
      [&]() {
        if (WARP) warp_min2();
        stopped = ub * kSlack < stop;
        if (stopped) lb = -1.0f;  // nothing is within reach any more
      });
  *lb2 = stopped ? INFINITY : lb;
  *ub2 = ub;
  // (lb still at the bound of the rings left out.)
  if (cut && !stopped && rings.last == most && lb == rings.gap2(most + 1)) *cut = 1u;
}

// Raises L from a finished search's lower distance.
__device__ __forceinline__ void raise_level(CellDirState* st, float lb2) {
  if (lb2 < INFINITY) atomicMax(&st->L2, __float_as_uint(lb2 / kSlack));
}

// The target's coarse map for a CTA's searches: copied to shared memory (a
// search is a chain of reads of it) unless it is too large.
template <class Ge>
__device__ __forceinline__ const uint32_t* search_map(const uint32_t* map) {
  if constexpr (Ge::kShared) {
    __shared__ uint4 s[Ge::kCoarse / 4];
    for (uint32_t i = threadIdx.x; i < Ge::kCoarse / 4; i += blockDim.x)
      s[i] = reinterpret_cast<const uint4*>(map)[i];
    __syncthreads();
    return reinterpret_cast<const uint32_t*>(s);
  } else {
    return map;
  }
}

// A direction's running maximum from L: a key of that distance and no row,
// below the key of any row at h, so that a scan or an index may stop its
// queries at L from the start (the FP64 listing pass at soft_stop(L)).
template <class Ge>
__device__ __forceinline__ void start_at_level(const CellDir& d, const CellGrid& g, float cells2) {
  const float L2 = cells2 * (g.side * g.side) * 0.9999f;
  if (g.valid && L2 > 0.0f)
    atomicMax(&d.sc->max_key, (unsigned long long) __float_as_uint(L2) << 32);
}

// Seeds (a warp per sampled word, 64 blocks, of the query set's coarse map):
// one cell of one of its occupied blocks.
template <class Ge>
__global__ void __launch_bounds__(kSearchThreads) k_cell_seed(CellArgs a) {
  chain_wait();
  const CellDir& d = a.d[blockIdx.y];
  const CellGrid g = cell_grid<Ge>(a.ord);
  if (!g.valid) return;
  const uint32_t* map = search_map<Ge>(a.coarse[1 - d.qset]);
  // kSeedWarps of the map's words, spread by an odd multiplier near 0.618 of
  // their number (a power of two).
  constexpr uint32_t kMapWords = Ge::kBlocks / 64;
  const uint32_t w = (blockIdx.x * kSearchWarps + (threadIdx.x >> 5)) *
                     ((uint32_t) (kMapWords * 0.618) | 1u) & (kMapWords - 1);
  const unsigned long long m =
      reinterpret_cast<const unsigned long long*>(a.coarse[d.qset])[w];
  if (!m) return;
  // The last occupied block of the word's row but one in four takes the
  // first: clusters' edges, where the far points are.
  const int bit = (w & 3) ? 63 - __clzll((long long) m) : __ffsll((long long) m) - 1;
  const uint32_t block = w * 64 + bit;
  const unsigned long long cells = a.occ[d.qset][block];
  const Probe<Ge> p = probe_cell<Ge>(block * 64 + __ffsll((long long) cells) - 1);
  const float stop = __uint_as_float(ld_relaxed_u32(&d.st->L2));
  float lb, ub;
  cell_search<Ge, true>(p, block_box<Ge>(a, g, 1 - d.qset), a.occ[1 - d.qset], map, stop, &lb, &ub,
                        Ge::kSeedRings, &d.st->cut);
  if ((threadIdx.x & 31) == 0) {
    raise_level(d.st, lb);
    if (a.seeds_only && lb < INFINITY) start_at_level<Ge>(d, g, lb / kSlack);
  }
}

// For a cell at each of the 64 places of a block, the cells of neighbour j (of
// 3^D) that lie within `stop` at the far corner, as masks of its 64 cells; the
// first 64 threads of a CTA.
template <class Ge>
__device__ __forceinline__ void near_masks(float stop, int j, unsigned long long* out) {
  constexpr int D = Ge::D, S = Ge::S;
  const int sub = threadIdx.x;
  if (sub >= 64) return;
  const int ox = (j % 3 - 1) * S - (sub & (S - 1));
  const int oy = (j / 3 % 3 - 1) * S - ((sub >> Ge::kSub) & (S - 1));
  const int oz = D == 3 ? (j / 9 - 1) * S - (sub >> (2 * Ge::kSub)) : 0;
  unsigned long long m = 0;
  for (int r = 0; r < 64 / S; ++r) {
    const float y = (float) (abs(oy + (r & (S - 1))) + 1) + Ge::kPad;
    const float z = D == 3 ? (float) (abs(oz + (r >> Ge::kSub)) + 1) + Ge::kPad : 0.0f;
    const float left = stop - y * y - z * z;
    if (!(left > 1.0f)) continue;
    const int w = (int) floorf(sqrtf(left) - 1.0f - Ge::kPad);  // cells apart along x, at most
    const int x0 = max(-ox - w, 0), x1 = min(-ox + w, S - 1);
    if (w >= 0 && x0 <= x1) m |= (unsigned long long) ((2u << x1) - (1u << x0)) << (r * S);
  }
  out[j * 64 + sub] = m;
}

// A thread per block of the query set: settled when the nearest target block
// to either side in one of the rows around it (25 rows in 3-D, 7 in 2-D, spaced
// to reach about 0.6 sqrt(stop)) lies within L at its far corner, else its cells
// are listed.  The first CTAs also write down the masks of k_cell_near.
template <class Ge>
__global__ void __launch_bounds__(256) k_cell_blocks(CellArgs a) {
  chain_wait();
  constexpr int D = Ge::D;
  const CellDir& d = a.d[blockIdx.y];
  const CellGrid g = cell_grid<Ge>(a.ord);
  const float stop = g.valid ? settle_level(d, g, d.st->L2) : 0.0f;
  if (!(stop >= kMinReach * kMinReach * D)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      d.st->off = 1u;
      start_at_level<Ge>(d, g, __uint_as_float(d.st->L2));  // for the index that takes over
      a.seen[blockIdx.y].L2 = d.st->L2;
      a.seen[blockIdx.y].off = 1u;
    }
    return;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    d.st->level = d.st->L2;
    a.seen[blockIdx.y].L2 = d.st->L2;
    a.seen[blockIdx.y].off = d.st->off;  // a query without a cell
  }
  constexpr int kN = D == 3 ? 27 : 9;
  if (blockIdx.x < kN)
    near_masks<Ge>(stop / kSlack, blockIdx.x, d.masks);
  else if (D == 3 && blockIdx.x < 2 * kN)
    near_masks<Ge>(stop / kSlack * 0.25f, blockIdx.x - kN, d.masks + kN * 64);
  // Squared reach in blocks, after the padding and slack; per row, how many
  // blocks apart along x still are within it (-1: none).
  constexpr int kRows = D == 3 ? 25 : 7;
  __shared__ int s_far[kRows];
  // (A pair settled here may lie G 2^-22 cells further apart per axis than its
  // blocks, whose far corners are at least sqrt(2) blocks apart: at 2^13 cells 0.05 %
  // of the square, under the 0.1 % taken off.)
  const float reach = (stop / kSlack) / (float) (Ge::S * Ge::S) * 0.999f;
  const int step = max(1, (int) (sqrtf(reach) * (D == 3 ? 0.3f : 0.2f)));
  if (threadIdx.x < kRows) {
    const int j = threadIdx.x;
    const int ay = abs(D == 3 ? j % 5 - 2 : j - 3) * step + 1;
    const int az = D == 3 ? abs(j / 5 - 2) * step + 1 : 0;
    const float left = reach - (float) (ay * ay + az * az);
    s_far[j] = left >= 1.0f ? (int) sqrtf(left) - 1 : -1;
  }
  __syncthreads();
  // A CTA takes runs of 256 blocks.
  __shared__ uint32_t s_sum[8], s_base;
  for (uint32_t block = blockIdx.x * 256 + threadIdx.x; block < Ge::kBlocks;
       block += gridDim.x * 256) {
    const bool some = (a.coarse[d.qset][block >> 5] >> (block & 31)) & 1u;
    if (!__syncthreads_or(some)) continue;
    const unsigned long long m = some ? a.occ[d.qset][block] : 0ull;
    bool open = m != 0;
    if (open) {
      const int bx = block % Ge::NB, by = block / Ge::NB % Ge::NB;
      const int bz = D == 3 ? block / (Ge::NB * Ge::NB) : 0;
      const unsigned long long* rows = reinterpret_cast<const unsigned long long*>(a.coarse[1 - d.qset]);
      // The row's word (3-D) or the words within reach (2-D).
      auto row = [&](int j) -> unsigned long long {
        const int y = by + (D == 3 ? j % 5 - 2 : j - 3) * step;
        const int z = D == 3 ? bz + (j / 5 - 2) * step : 0;
        const int far = s_far[j];
        if (far < 0 || (uint32_t) y >= (uint32_t) Ge::NB || (uint32_t) z >= (uint32_t) Ge::NB) return 0;
        const unsigned long long* w = rows + (size_t) (D == 3 ? z * Ge::NB + y : y) * Ge::kWords;
        const int x0 = max(bx - far, 0), x1 = min(bx + far, Ge::NB - 1);
        unsigned long long any = 0;
        for (int k = x0 >> 6; k <= x1 >> 6; ++k) {
          unsigned long long bits = ld_global_u64(w + k);
          if (k == x0 >> 6) bits &= ~0ull << (x0 & 63);
          if (k == x1 >> 6) bits &= ~0ull >> (63 - (x1 & 63));
          any |= bits;
        }
        return any;
      };
      // The middle row first, then five (2-D: three) at a time.
      open = row(kRows / 2) == 0;
      constexpr int kGroup = D == 3 ? 5 : 3;
      for (int j0 = 0; j0 < kRows && open; j0 += kGroup) {
        unsigned long long any = 0;
#pragma unroll
        for (int k = 0; k < kGroup; ++k)
          if (j0 + k < kRows) any |= row(j0 + k);
        open = any == 0;
      }
    }
    // Room for the open blocks' cells, one atomic per CTA.
    const uint32_t cnt = open ? (uint32_t) __popcll(m) : 0u;
    uint32_t incl = cnt;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) s_sum[warp] = incl;
    __syncthreads();
    uint32_t base = 0, total = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (k < warp) base += s_sum[k];
      total += s_sum[k];
    }
    if (total == 0) continue;
    if (threadIdx.x == 0) s_base = atomicAdd(&d.st->n_cells, total);
    __syncthreads();
    base += s_base + incl - cnt;
    unsigned long long rest = open ? m : 0ull;
    while (rest) {
      const int t = __ffsll((long long) rest) - 1;
      rest &= rest - 1;
      if (base < d.cap_cells) d.cells[base] = block * 64 + t;
      ++base;
    }
  }
}

// A thread per listed cell: settled when a target cell of the blocks around it
// (its own and those it touches) lies within L at the far corner, by the masks
// of k_cell_blocks, else kept for the search.
// HALF (3-D): the same once more for what is left, on cells of twice the size,
// whose blocks reach twice as far; at the rim of a cluster most cells have
// their nearest target one or two blocks beyond the touching ones.
template <class Ge, bool HALF>
__global__ void __launch_bounds__(256) k_cell_near(CellArgs a) {
  chain_wait();
  constexpr int D = Ge::D;
  constexpr int NB = HALF ? Ge::NB / 2 : Ge::NB;
  constexpr int kN = D == 3 ? 27 : 9;
  __shared__ unsigned long long mask[kN * 64];
  const CellDir& d = a.d[blockIdx.y];
  if (d.st->off) return;
  if (d.st->n_cells > d.cap_cells) {
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicExch(&d.st->off, 1u);
    return;
  }
  const uint32_t n = HALF ? d.st->n_rim : d.st->n_cells;
  if (blockIdx.x * 256 >= n) return;
  for (int i = threadIdx.x; i < kN * 64; i += 256) mask[i] = d.masks[(HALF ? kN * 64 : 0) + i];
  __syncthreads();
  const unsigned long long* occ = HALF ? a.half[1 - d.qset] : a.occ[1 - d.qset];
  // 3-D: listed cells -> rim -> far; 2-D: listed cells -> far.
  const uint32_t* in = HALF ? d.rim : d.cells;
  uint32_t* out = HALF ? d.far : D == 3 ? d.rim : d.far;
  uint32_t* out_n = HALF || D == 2 ? &d.st->n_far : &d.st->n_rim;
  for (uint32_t e = blockIdx.x * 256 + threadIdx.x; e < n; e += gridDim.x * 256) {
    const uint32_t cell = in[e];
    uint32_t block = cell >> 6, sub = cell & 63;
    int bx = block % Ge::NB, by = block / Ge::NB % Ge::NB;
    int bz = D == 3 ? block / (Ge::NB * Ge::NB) : 0;
    if constexpr (HALF) {
      sub = half_cell(bx, by, bz, sub & 3, (sub >> 2) & 3, sub >> 4);
      bx >>= 1;
      by >>= 1;
      bz >>= 1;
      block = (uint32_t) ((bz * NB + by) * NB + bx);
    }
    bool open = !(occ[block] & mask[kN / 2 * 64 + sub]);
    if (open) {
#pragma unroll
      for (int r = 0; r < kN / 3; ++r) {
        const int y = by + r % 3 - 1, z = D == 3 ? bz + r / 3 - 1 : 0;
        if (!open || (uint32_t) y >= (uint32_t) NB || (uint32_t) z >= (uint32_t) NB) continue;
        const unsigned long long* w = occ + ((size_t) (D == 3 ? z * NB + y : y) * NB + bx);
        unsigned long long hit = w[0] & mask[(3 * r + 1) * 64 + sub];
        if (bx > 0) hit |= w[-1] & mask[3 * r * 64 + sub];
        if (bx < NB - 1) hit |= w[1] & mask[(3 * r + 2) * 64 + sub];
        if (hit) open = false;
      }
    }
    if (open) out[take_slot(out_n)] = cell;
  }
}

// A warp per far cell, which shortens the chain of reads; with more than
// kManyFar of them a thread per cell, which takes a tenth of the instructions.
constexpr uint32_t kManyFar = 24576;

// The search gives a direction up when most of the query set's cells are far (one
// set around the other: hardly any is settled by the cells), or when the rows to
// look through are too many: 8 million and one per point.  1M + 1M points, given
// up and searched, and the index alone: 3-D shells of radius 1 and 1.05 1.42, 2.74
// and 1.36 ms undirected; two cubes apart (64,000 cells by 289 rows) directed 0.47,
// 0.93 and 0.47 ms; but 10M + 10M with 48,000 such cells 1.3, 0.91 and 1.12.
constexpr float kMaxRows = 8e6f;

template <class Ge>
__global__ void __launch_bounds__(kSearchThreads) k_cell_search(CellArgs a) {
  chain_wait();
  const CellDir& d = a.d[blockIdx.y];
  if (d.st->off) return;
  const uint32_t n = d.st->n_far;
  const bool many = n > kManyFar;
  if (blockIdx.x * (many ? kSearchThreads : kSearchWarps) >= n) return;
  const CellGrid g = cell_grid<Ge>(a.ord);
  const BlockBox<Ge> box = block_box<Ge>(a, g, 1 - d.qset);
  // Rows of blocks per cell, at least.  (st->level: L2 rises from here on.)
  const float r = 2.0f * ceilf(sqrtf(__uint_as_float(d.st->level)) / (float) Ge::S) + 1.0f;
  float rows = fminf(r, (float) (box.hi[1] - box.lo[1] + 1));
  if constexpr (Ge::D == 3) rows *= fminf(r, (float) (box.hi[2] - box.lo[2] + 1));
  if ((many && n > d.st->n_occ / 2) || (float) n * rows > kMaxRows + (float) (d.nQ + d.nT)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      d.st->wide = 1u;
      atomicExch(&d.st->off, 1u);
      start_at_level<Ge>(d, g, __uint_as_float(d.st->L2));  // for the index that takes over
    }
    return;
  }
  const uint32_t* map = search_map<Ge>(a.coarse[1 - d.qset]);
  const unsigned long long* occ = a.occ[1 - d.qset];
  float lb, ub;
  if (many) {
    for (uint32_t e = blockIdx.x * kSearchThreads + threadIdx.x; e < n;
         e += gridDim.x * kSearchThreads) {
      const float stop = settle_level(d, g, ld_relaxed_u32(&d.st->L2));
      cell_search<Ge, false>(probe_cell<Ge>(d.far[e]), box, occ, map, stop, &lb, &ub);
      d.far_ub[e] = ub;
      if (lb < INFINITY && lb / kSlack > __uint_as_float(ld_relaxed_u32(&d.st->L2)))
        raise_level(d.st, lb);
    }
    return;
  }
  const int lane = threadIdx.x & 31;
  for (uint32_t e = blockIdx.x * kSearchWarps + (threadIdx.x >> 5); e < n;
       e += gridDim.x * kSearchWarps) {
    const float stop = settle_level(d, g, ld_relaxed_u32(&d.st->L2));
    cell_search<Ge, true>(probe_cell<Ge>(d.far[e]), box, occ, map, stop, &lb, &ub);
    if (lane == 0) {
      d.far_ub[e] = ub;
      raise_level(d.st, lb);
    }
  }
}

// Cells whose upper distance exceeds the L that the search ended with, and the
// target cells within that distance of them.  Few cells get here: a CTA looks
// for them among kMarkChunk far cells at a time and takes each with all its
// warps.  They sit together in the list, so that a CTA's chunk is taken from all
// over it (10M clusters 53 -> 43 us against chunks of neighbours, two thirds of
// the SMs idle then; the call 350 -> 345, 1M 203 -> 195).  Of more than kManyFar far
// cells many may be marked: then a thread per cell marks whole blocks within the
// distance.
constexpr uint32_t kMarkChunk = 8;

// Where the map of blocks is too large for shared memory, a top map of 2^18
// super-blocks (of 4^3 or 4^2 blocks) stands before it.
template <class Ge>
__device__ __forceinline__ uint32_t super_block(uint32_t block) {
  if constexpr (Ge::kShared) {
    return block;
  } else {
    constexpr int N = Ge::NB / Ge::kTop;
    const uint32_t x = block % Ge::NB / Ge::kTop, y = block / Ge::NB % Ge::NB / Ge::kTop;
    return Ge::D == 3 ? (block / (Ge::NB * Ge::NB) / Ge::kTop * N + y) * N + x : y * N + x;
  }
}

// Marks a block in a set's map of blocks and in the map before it.
template <class Ge>
__device__ __forceinline__ void mark_block(uint32_t* any, uint32_t* top, uint32_t block) {
  const uint32_t bit = 1u << (block & 31);
  if (atomicOr(any + (block >> 5), bit) & bit) return;
  if constexpr (!Ge::kShared) {
    const uint32_t s = super_block<Ge>(block);
    if (!((__ldcg(top + (s >> 5)) >> (s & 31)) & 1u)) atomicOr(top + (s >> 5), 1u << (s & 31));
  }
}

template <class Ge>
__global__ void __launch_bounds__(kSearchThreads) k_cell_mark(CellArgs a) {
  chain_wait();
  constexpr int D = Ge::D;
  __shared__ uint32_t s_cell[kMarkChunk];
  __shared__ float s_ub[kMarkChunk];
  __shared__ uint32_t s_n;
  const CellDir& d = a.d[blockIdx.y];
  if (d.st->off) return;
  const uint32_t n = d.st->n_far;
  const bool many = n > kManyFar;
  if (blockIdx.x * (many ? kSearchThreads : kMarkChunk) >= n) return;
  const uint32_t* map = search_map<Ge>(a.coarse[1 - d.qset]);
  const CellGrid g = cell_grid<Ge>(a.ord);
  const BlockBox<Ge> box = block_box<Ge>(a, g, 1 - d.qset);
  const float stop = settle_level(d, g, d.st->L2);
  const unsigned long long* occ = a.occ[1 - d.qset];
  uint32_t* any_q = a.any[d.qset];
  uint32_t* any_t = a.any[1 - d.qset];
  // Squared distance within which a cell's targets are marked.
  auto reach_of = [&](float ub) {
    const float r2 = ub * kSlack;
    if (!(d.soft_r > 0.0f)) return r2;
    const float r = sqrtf(r2) * kSlack + 2.1f * d.soft_r / g.side;
    return r * r * kSlack;
  };
  auto mark_query = [&](uint32_t cell, float ub) {
    atomicOr(d.U + (cell >> 6), 1ull << (cell & 63));
    mark_block<Ge>(any_q, a.top[d.qset], cell >> 6);
    if (!(ub < INFINITY)) atomicExch(&d.st->off, 1u);  // the target has no cell at all
  };
  if (many) {
    for (uint32_t e = blockIdx.x * kSearchThreads + threadIdx.x; e < n;
         e += gridDim.x * kSearchThreads) {
      const float ub = d.far_ub[e];
      if (ub * kSlack < stop) continue;
      const uint32_t cell = d.far[e];
      mark_query(cell, ub);
      if (!(ub < INFINITY)) continue;
      const float r2 = reach_of(ub);
      const Probe<Ge> p = probe_cell<Ge>(cell);
      visit_blocks<Ge, false>(
          p, box, Rings<Ge>(p, box), map, 0, 1, [&]() { return r2; },
          [&](uint32_t block, int, int, int) {
            if (__ldcg(d.N + block) == ~0ull) return;
            d.N[block] = ~0ull;
            mark_block<Ge>(any_t, a.top[1 - d.qset], block);
          },
          []() {});
    }
    return;
  }
  const uint32_t chunks = (n + kMarkChunk - 1) / kMarkChunk;
  for (uint32_t at = blockIdx.x; at < chunks; at += gridDim.x) {
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    const uint32_t e = at + threadIdx.x * chunks;  // from all over the list
    if (threadIdx.x < kMarkChunk && e < n && !(d.far_ub[e] * kSlack < stop)) {
      const uint32_t cell = d.far[e], i = atomicAdd(&s_n, 1u);
      s_cell[i] = cell;
      s_ub[i] = d.far_ub[e];
      mark_query(cell, s_ub[i]);
    }
    __syncthreads();
    for (uint32_t i = 0; i < s_n; ++i) {
      if (!(s_ub[i] < INFINITY)) continue;
      const float r2 = reach_of(s_ub[i]);
      const Probe<Ge> p = probe_cell<Ge>(s_cell[i]);
      visit_blocks<Ge, true>(
          p, box, Rings<Ge>(p, box), map, threadIdx.x, kSearchThreads, [&]() { return r2; },
          [&](uint32_t block, int bx, int by, int bz) {
            unsigned long long m = occ[block], hit = 0ull;
            while (m) {
              const int t = __ffsll((long long) m) - 1;
              m &= m - 1;
              float l2 = 0.0f;
#pragma unroll
              for (int k = 0; k < D; ++k) {
                const int b = k == 0 ? bx : k == 1 ? by : bz;
                const float c = (float) (b * Ge::S + ((t >> (k * Ge::kSub)) & (Ge::S - 1)));
                const float gl = fmaxf(fmaxf(c - p.hi[k], p.lo[k] - (c + 1.0f)) - Ge::kPad, 0.0f);
                l2 += gl * gl;
              }
              if (l2 <= r2) hit |= 1ull << t;
            }
            if (hit && (hit & ~__ldcg(d.N + block))) {
              atomicOr(d.N + block, hit);
              mark_block<Ge>(any_t, a.top[1 - d.qset], block);
            }
          },
          []() {});
    }
    __syncthreads();
  }
}

// The points in marked cells, as (x, y, z, row): queries of the direction that
// asks for the set's points, targets of the other (blockIdx.y = set).  Four
// points per thread and step; the set's map of blocks turns most away.  Not
// chained, so that the marks are constant here.
template <class Ge>
__global__ void __launch_bounds__(256) k_cell_collect(CellArgs a, const float* __restrict__ A,
                                                      uint64_t nA, const float* __restrict__ B,
                                                      uint64_t nB) {
  constexpr int D = Ge::D;
  const int set = blockIdx.y;
  const bool ask = set < a.count && !a.d[set].st->off;               // direction `set`
  const bool give = 1 - set < a.count && !a.d[1 - set].st->off;      // direction 1 - set
  if (!ask && !give) return;
  const CellDir& dq = a.d[set];
  const CellDir& dt = a.d[1 - set];
  const float* P = set ? B : A;
  const uint64_t n = set ? nB : nA;
  const uint32_t* any = a.any[set];
  const uint32_t* top = Ge::kShared ? any : search_map<Geo<3, 8>>(a.top[set]);
  const uint4* code = reinterpret_cast<const uint4*>(a.code[set]);  // padded to whole groups
  const uint64_t groups = (n + 3) / 4, stride = (uint64_t) gridDim.x * blockDim.x;
  for (uint64_t t = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; t < groups; t += stride) {
    const uint4 c4 = __ldcs(code + t);
    const uint32_t c[4] = {c4.x, c4.y, c4.z, c4.w};
    uint32_t hit = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      // kNoCell is past the map: masked into it, and left out below.
      const uint32_t block = super_block<Ge>((c[k] >> 6) & (Ge::kBlocks - 1));
      hit |= ((top[block >> 5] >> (block & 31)) & 1u) << k;
    }
    const uint64_t left = n - 4 * t;
    if (left < 4) hit &= (1u << left) - 1u;
    while (hit) {
      const int k = __ffs(hit) - 1;
      hit &= hit - 1;
      const uint32_t ck = k == 0 ? c[0] : k == 1 ? c[1] : k == 2 ? c[2] : c[3];
      if (ck == kNoCell) continue;
      if (!Ge::kShared && !((__ldg(any + (ck >> 11)) >> ((ck >> 6) & 31)) & 1u)) continue;
      const bool q = ask && ((__ldg(dq.U + (ck >> 6)) >> (ck & 63)) & 1ull);
      const bool t2 = give && ((__ldg(dt.N + (ck >> 6)) >> (ck & 63)) & 1ull);
      if (!q && !t2) continue;
      const uint64_t i = 4 * t + k;
      const float4 p = make_float4(P[i * D], P[i * D + 1], D == 3 ? P[i * D + 2] : 0.0f,
                                   __uint_as_float((uint32_t) i));
      if (q) {
        const uint32_t slot = take_slot(&dq.st->n_q);
        if (slot < dq.cap_q) {
          dq.q[slot] = p;
          dq.q_min[slot] = ~0ull;
        }
      }
      if (t2) {
        const uint32_t slot = take_slot(&dt.st->n_t);
        if (slot < dt.cap_t) dt.t[slot] = p;
      }
    }
  }
}

__device__ __forceinline__ bool scan_takes(const CellDirState* st, uint32_t cap_q, uint32_t cap_t) {
  return !st->off && st->n_q > 0 && st->n_t > 0 && st->n_q <= cap_q && st->n_t <= cap_t &&
         (uint64_t) st->n_q * st->n_t <= kScanPairs;
}

// All pairs of open queries and collected targets, when they are few: items of
// 256 queries (one per thread) by kScanTile targets (through shared memory),
// each query's nearest target (lowest row among ties: every target at its
// distance was collected) by one 64-bit atomicMin per item.  The last CTA to
// finish takes the maximum over the queries and writes the direction's result
// (with a plan, only that maximum).
template <class Ge, bool COUNT>
__global__ void __launch_bounds__(256) k_cell_solve(CellArgs a) {
  constexpr int D = Ge::D;
  __shared__ float4 s[kScanTile];
  __shared__ unsigned long long red[2][8];
  __shared__ bool s_last;
  const CellDir& d = a.d[blockIdx.y];
  if (!scan_takes(d.st, d.cap_q, d.cap_t)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) a.left[blockIdx.y] = *d.st;
    return;
  }
  const uint32_t nq = d.st->n_q, nt = d.st->n_t;
  const uint32_t qt = (nq + 255) / 256, tt = (nt + kScanTile - 1) / kScanTile;
  const uint64_t items = (uint64_t) qt * tt;
  if (blockIdx.x >= items) return;
  for (uint64_t item = blockIdx.x; item < items; item += gridDim.x) {
    const uint32_t q0 = (uint32_t) (item % qt) * 256, t0 = (uint32_t) (item / qt) * kScanTile;
    const uint32_t m = min((uint32_t) kScanTile, nt - t0);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < m; i += 256) s[i] = d.t[t0 + i];
    __syncthreads();
    const uint32_t e = q0 + threadIdx.x;
    if (e < nq) {
      const float4 q = d.q[e];
      unsigned long long best = ~0ull;
#pragma unroll 8
      for (uint32_t i = 0; i < m; ++i) {
        const unsigned long long k = pack_min(d2_pt_packed<D>(q, s[i]), __float_as_uint(s[i].w));
        best = k < best ? k : best;
      }
      atomicMin(d.q_min + e, best);
    }
  }
  __threadfence();
  __syncthreads();
  const uint32_t ctas = (uint32_t) min((uint64_t) gridDim.x, items);
  if (threadIdx.x == 0) s_last = atomicAdd(&d.st->ticket, 1u) == ctas - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // The largest distance, the lowest query row among ties, and its target.
  unsigned long long best = 0, pair = 0;
#pragma unroll 4
  for (uint32_t e = threadIdx.x; e < nq; e += 256) {
    const unsigned long long k = __ldcg(d.q_min + e);
    const unsigned long long v = (k & 0xFFFFFFFF00000000ull) | (kInvalid - __float_as_uint(d.q[e].w));
    if (v > best) {
      best = v;
      pair = k;
    }
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const unsigned long long v = __shfl_xor_sync(0xFFFFFFFFu, best, o);
    const unsigned long long k = __shfl_xor_sync(0xFFFFFFFFu, pair, o);
    if (v > best) {
      best = v;
      pair = k;
    }
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = best;
    red[1][threadIdx.x >> 5] = pair;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 1; k < 8; ++k)
      if (red[0][k] > best) {
        best = red[0][k];
        pair = red[1][k];
      }
    if (d.soft_r >= 0.0f) {  // the FP64 path goes on from here
      d.st->max32 = (uint32_t) (best >> 32);
      d.st->scanned = 1u;
      if (COUNT) d.sc->pairs += (unsigned long long) nq * nt;
      return;
    }
    d.sc->max_key = best;
    d.sc->min_key = pair;
    if (COUNT) d.sc->pairs += (unsigned long long) nq * nt;
    finalize_scalars(d.Q, d.T, D, d.sc);
    d.st->done = 1u;
    // The words that the host reads.
    DevScalars* o = a.result + (d.sc - a.sc0);
    o->d2_64 = d.sc->d2_64;
    o->d2 = d.sc->d2;
    o->ia = d.sc->ia;
    o->ib = d.sc->ib;
    o->status = d.sc->status;
    o->pairs = d.sc->pairs;
    o->nodes = o->leaves = 0;
    o->heavy_count = 0;
    a.left[blockIdx.y].off = 0u;
    a.left[blockIdx.y].done = 1u;
    __threadfence_system();
  }
}

constexpr size_t kStateBytes = 4096;  // both directions' states and seed words
constexpr size_t kStageState = 3072, kStageSeeds = 3584;  // in the pinned staging (4 KB)

uint64_t cap_queries(uint64_t n) { return n / 8 + 8192; }
uint64_t cap_targets(uint64_t n) { return n / 4 + 8192; }
constexpr uint64_t kCapCells = 1ull << 23;

// Grids by level: 2^8 cells per axis in 3-D; 2^12 in 2-D, and 2^13 from
// kFine2Points points, whose answer is a few cells of the first.  A 3-D direction
// that is too few cells there is tried again on 2^10 (maps of 128 MB a set) if its L
// is kFinerReach diagonals there, from kFinestPoints points.  The index alone and
// that grid, us: directed planes 16M + 16M 2495 and 2487, 14M + 16M 2375 and 2460, 18M
// + 18M 2771 and 2590, undirected 21M + 21M 3310 and 2950.  With A sorted beside B's
// copy the index is ahead for longer: 21M + 21M 4770 and 5290, 30M + 30M 6700 and
// 6660.  (In 2-D a grid of 2^14 never paid: uniform 21M + 21M 6095 without it, 6990
// with it, whose lists ran over.)
constexpr int kFinest = 2;
constexpr uint64_t kFine2Points = 1500000;
constexpr uint64_t kFinestPoints = 33000000, kFinestPointsSorted = 60000000;
constexpr float kFinerReach = 2.5f;

}  // namespace

// Not for one direction against few targets: hardly a cell of the queries is near
// one.  The index alone and the filter first, us: 1M x 3,000 uniform 3-D 326 and 655,
// 10M x 100 2-D 650 and 1055, FP64 1M x 1,000 311 and 362 (undirected the other
// direction makes up for it).
constexpr uint64_t kCellsMaxRatio = 128;

bool cells_apply(const Ctx& c, uint64_t nA, uint64_t nB, int dims, bool undirected) {
  return (dims == 2 || dims == 3) && nA + nB >= kCellsMinPoints &&
         (undirected || nA / kCellsMaxRatio <= nB) && c.opt.lbvh_budget == tuning().lbvh_budget;
}

namespace {

// The filter's launches: eleven short kernels in a row (200k uniform 2-D points
// 144 -> 131 us with them chained, 1M clusters 220 -> 204, 10M 368 -> 348).  Not
// chained are the search, whose waiting CTAs hold shared memory that the level
// before needs (5M 2-D points 374 -> 439 us), the pass over the points, which ran
// slower when it started beside the marking (50M planes 3.94 -> 4.33 ms), and the
// pair scan, which delays an index that waits behind it (200k planes directed
// 294 -> 310 us).
template <class Ge>
hd_status enqueue(Ctx& c, const DirInput* ins, int count, const F64Plan* plan, CellArgs& a,
                  bool boxes_known, bool seeds_only, bool* no_room) {
  const uint64_t n[2] = {ins[0].nA, ins[0].nB};
  hd_status s;
  // Zeroed words first: state, occupied cells, U, N, maps of marked blocks.
  const size_t fine = (size_t) Ge::kBlocks * 8, coarse = (size_t) Ge::kCoarse * 4;
  size_t off = kStateBytes;
  auto take = [&](size_t bytes) {
    const size_t o = off;
    off += (bytes + 255) / 256 * 256;
    return o;
  };
  size_t o_occ[2], o_half[2], o_U[2], o_N[2], o_any[2], o_top[2];
  for (int k = 0; k < 2; ++k) {
    o_occ[k] = take(fine);
    o_half[k] = take(Ge::D == 3 ? fine / 8 : 0);
    o_any[k] = take(coarse);
    o_top[k] = take(Ge::kShared ? 0 : 32768);
  }
  const int lists = seeds_only ? 0 : count;
  for (int k = 0; k < lists; ++k) {
    o_U[k] = take(fine);
    o_N[k] = take(fine);
  }
  const size_t zero_bytes = off;
  size_t o_coarse[2], o_code[2], o_cells[2], o_masks[2], o_rim[2], o_far[2], o_fub[2];
  size_t o_q[2], o_qmin[2], o_t[2];
  for (int k = 0; k < 2; ++k) {
    o_coarse[k] = take(coarse);
    o_code[k] = take((n[k] + 3) / 4 * 16);
  }
  for (int k = 0; k < lists; ++k) {
    const uint64_t cc = std::min(n[k], kCapCells);
    const uint64_t cq = cap_queries(n[k]), ct = cap_targets(n[1 - k]);
    o_cells[k] = take(cc * 4);
    o_masks[k] = take(2 * 27 * 64 * 8);
    o_rim[k] = take(Ge::D == 3 ? cc * 4 : 0);
    o_far[k] = take(cc * 4);
    o_fub[k] = take(cc * 4);
    o_q[k] = take(cq * sizeof(float4));
    o_qmin[k] = take(cq * 8);
    o_t[k] = take(ct * sizeof(float4));
  }
  void* buf;
  const std::string before = c.last_error;
  if (ensure(c, kBufCells, off, &buf) != HD_OK) {
    c.last_error = before;
    *no_room = true;
    return HD_OK;
  }
  char* base = (char*) buf;
  a.ord = scalars(c, 0)->mbr_ord;
  a.swapped = ins[0].dir;
  for (int k = 0; k < 2; ++k) {
    a.occ[k] = (unsigned long long*) (base + o_occ[k]);
    a.half[k] = (unsigned long long*) (base + o_half[k]);
    a.coarse[k] = (uint32_t*) (base + o_coarse[k]);
    a.code[k] = (uint32_t*) (base + o_code[k]);
    a.any[k] = (uint32_t*) (base + o_any[k]);
    a.top[k] = (uint32_t*) (base + o_top[k]);
  }
  a.count = count;
  a.seeds_only = seeds_only;
  a.seen = (CellDirState*) ((char*) c.host_pinned + kStageSeeds);
  a.left = (CellDirState*) ((char*) c.host_pinned + kStageState);
  a.sc0 = scalars(c, 0);
  a.result = (DevScalars*) c.host_pinned;
  for (int k = 0; k < count; ++k) {
    CellDir& d = a.d[k];
    d.Q = ins[k].A;
    d.T = ins[k].B;
    d.nQ = ins[k].nA;
    d.nT = ins[k].nB;
    d.qset = k;
    d.st = (CellDirState*) base + k;
    d.sc = scalars(c, ins[k].dir);
    d.soft_r = plan ? plan->soft_r[k] : -1.0f;
    if (seeds_only) continue;
    d.U = (unsigned long long*) (base + o_U[k]);
    d.N = (unsigned long long*) (base + o_N[k]);
    d.cells = (uint32_t*) (base + o_cells[k]);
    d.masks = (unsigned long long*) (base + o_masks[k]);
    d.rim = (uint32_t*) (base + o_rim[k]);
    d.far = (uint32_t*) (base + o_far[k]);
    d.far_ub = (float*) (base + o_fub[k]);
    d.q = (float4*) (base + o_q[k]);
    d.q_min = (unsigned long long*) (base + o_qmin[k]);
    d.t = (float4*) (base + o_t[k]);
    d.cap_cells = (uint32_t) std::min(ins[k].nA, kCapCells);
    d.cap_q = (uint32_t) cap_queries(ins[k].nA);
    d.cap_t = (uint32_t) cap_targets(ins[k].nB);
  }
  if (count == 1) a.d[1] = a.d[0];
  cudaError_t e = cudaMemsetAsync(base, 0, zero_bytes, c.stream);
  if (e != cudaSuccess) return cuda_fail(c, e, "memset cells");
  if (!boxes_known && (s = spatial_boxes(c, ins[0])) != HD_OK) return s;
  const uint64_t most = std::max(n[0], n[1]);
  const unsigned sms = (unsigned) c.num_sms, dirs = (unsigned) count;
  // Passes over points: four points per thread.
  const unsigned gp = (unsigned) std::max<uint64_t>(
      1, std::min<uint64_t>((most / 4 + 255) / 256, (uint64_t) sms * 8));
  constexpr bool chain = true;
  const uint32_t every = n[0] + n[1] >= kOccSplit ? kOccFirst : 1u;
  launch_next(c.stream, chain, k_cell_occ<Ge, true>, dim3(gp, 2), 256, a, ins[0].A, ins[0].nA, ins[0].B,
              ins[0].nB, every);
  if ((s = after_launch(c, "cell_occ")) != HD_OK) return s;
  if (every > 1) {
    launch_next(c.stream, chain, k_cell_occ<Ge, false>, dim3(gp, 2), 256, a, ins[0].A, ins[0].nA,
                ins[0].B, ins[0].nB, every);
    if ((s = after_launch(c, "cell_occ")) != HD_OK) return s;
  }
  launch_next(c.stream, chain, k_cell_coarse<Ge>, dim3(Ge::kBlocks / 256, 2), 256, a);
  if ((s = after_launch(c, "cell_coarse")) != HD_OK) return s;
  launch_next(c.stream, chain, k_cell_seed<Ge>, dim3(kSeedWarps / kSearchWarps, dirs), kSearchThreads, a);
  if ((s = after_launch(c, "cell_seed")) != HD_OK) return s;
  if (seeds_only) return HD_OK;
  launch_next(c.stream, chain, k_cell_blocks<Ge>,
              dim3(std::min<unsigned>(Ge::kBlocks / 256, sms * 32), dirs), 256, a);
  if ((s = after_launch(c, "cell_blocks")) != HD_OK) return s;
  // What the seeds found is in pinned memory now, for the host to act on while
  // the rest runs.
  if (!c.cells_event) {
    if ((e = cudaEventCreateWithFlags(&c.cells_event, cudaEventDisableTiming)) != cudaSuccess)
      return cuda_fail(c, e, "filter event");
  }
  if ((e = cudaEventRecord(c.cells_event, c.stream)) != cudaSuccess)
    return cuda_fail(c, e, "filter event");
  const dim3 gw(sms * 6 / dirs, dirs);  // searches: six CTAs with the map per SM
  const dim3 gn(sms * 8 / dirs, dirs);
  launch_next(c.stream, chain, k_cell_near<Ge, false>, gn, 256, a);
  if ((s = after_launch(c, "cell_near")) != HD_OK) return s;
  if constexpr (Ge::D == 3) {
    launch_next(c.stream, chain, k_cell_near<Ge, true>, gn, 256, a);
    if ((s = after_launch(c, "cell_near")) != HD_OK) return s;
  }
  launch_next(c.stream, false, k_cell_search<Ge>, gw, kSearchThreads, a);
  if ((s = after_launch(c, "cell_search")) != HD_OK) return s;
  launch_next(c.stream, chain, k_cell_mark<Ge>, gw, kSearchThreads, a);
  if ((s = after_launch(c, "cell_mark")) != HD_OK) return s;
  mark(c, 1);
  launch_next(c.stream, false, k_cell_collect<Ge>, dim3(gp, 2), 256, a, ins[0].A, ins[0].nA, ins[0].B,
              ins[0].nB);
  if ((s = after_launch(c, "cell_collect")) != HD_OK) return s;
  mark(c, 2);
  mark(c, 3);
  const dim3 gs(sms * 4, dirs);
  if (ins[0].count)
    launch_next(c.stream, false, k_cell_solve<Ge, true>, gs, 256, a);
  else
    launch_next(c.stream, false, k_cell_solve<Ge, false>, gs, 256, a);
  if ((s = after_launch(c, "cell_solve")) != HD_OK) return s;
  mark(c, 4);
  mark(c, 5);
  return HD_OK;
}

}  // namespace

int cells_level(uint64_t points, int dims) { return dims == 2 && points >= kFine2Points ? 1 : 0; }

int cells_finer(uint64_t points, int dims, int level, float reach, bool sorted) {
  const bool take = dims == 3 && points >= (sorted ? kFinestPointsSorted : kFinestPoints) &&
                    reach * (float) (1 << (kFinest - level)) >= kFinerReach * 1.732f;
  return take ? kFinest : -1;
}

hd_status cells_begin(Ctx& c, const DirInput* ins, int count, int level, const F64Plan* plan,
                      bool boxes_known, CellsRun* run) {
  CellArgs a{};
  bool no_room = false;
  *run = CellsRun{};
  auto go = [&](auto grid) {
    return enqueue<decltype(grid)>(c, ins, count, plan, a, boxes_known, false, &no_room);
  };
  hd_status s;
  if (ins[0].dims == 3)
    s = level == 0 ? go(Geo<3, 8>{}) : go(Geo<3, 10>{});
  else
    s = level == 0 ? go(Geo<2, 12>{}) : go(Geo<2, 13>{});
  if (s != HD_OK || no_room) return s;
  run->ran = true;
  run->wrote = plan == nullptr;
  c.cells_live = true;
  run->state = a.d[0].st;
  for (int k = 0; k < count; ++k) {
    run->q_min[k] = a.d[k].q_min;
    run->q[k] = a.d[k].q;
    run->t[k] = a.d[k].t;
    run->cap_q[k] = a.d[k].cap_q;
    run->cap_t[k] = a.d[k].cap_t;
  }
  return HD_OK;
}

hd_status cells_seed(Ctx& c, const DirInput* ins, int count) {
  CellArgs a{};
  bool no_room = false;
  const hd_status s =
      ins[0].dims == 3 ? enqueue<Geo<3, 8>>(c, ins, count, nullptr, a, false, true, &no_room)
                       : enqueue<Geo<2, 12>>(c, ins, count, nullptr, a, false, true, &no_room);
  // Zeroed words behind the states, for the scan's own seeds.
  uint32_t* words = (uint32_t*) (a.d[0].st + 2);
  static_assert(2 * sizeof(CellDirState) + 2 * kSeedWords * 4 <= kStateBytes, "state");
  for (int k = 0; k < count; ++k)
    c.cell_seeds[ins[k].dir] = s == HD_OK && !no_room
                                   ? CellSeeds{a.d[k].st, words + k * kSeedWords}
                                   : CellSeeds{};
  return s;
}

hd_status cells_hopeless(Ctx& c, int count, int dims, const CellsRun& run, bool* off,
                         float* reach) {
  for (int k = 0; k < count; ++k) {
    off[k] = false;
    reach[k] = 0.0f;
  }
  if (!run.ran) return HD_OK;
  cudaError_t e = cudaEventSynchronize(c.cells_event);
  if (e != cudaSuccess) return cuda_fail(c, e, "filter seeds");
  const CellDirState* h =
      reinterpret_cast<const CellDirState*>((const char*) c.host_pinned + kStageSeeds);
  for (int k = 0; k < count; ++k) {
    float L2;
    memcpy(&L2, &h[k].L2, 4);
    // The test of k_cell_blocks (without a plan, whose level is lower).
    off[k] = h[k].off != 0 || !(L2 >= kMinReach * kMinReach * (float) dims);
    reach[k] = std::sqrt(L2);
  }
  return HD_OK;
}

hd_status cells_finish(Ctx& c, int count, const CellsRun& run, CellsLeft* left) {
  for (int k = 0; k < count; ++k) left[k] = CellsLeft{};
  if (!run.ran) return HD_OK;
  CellDirState* h = reinterpret_cast<CellDirState*>((char*) c.host_pinned + kStageState);
  static_assert(2 * sizeof(CellDirState) <= 512, "pinned staging");
  cudaError_t e = cudaSuccess;
  if (!run.wrote)
    e = cudaMemcpyAsync(h, run.state, 2 * sizeof(CellDirState), cudaMemcpyDeviceToHost, c.stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c.stream);
  if (e != cudaSuccess) return cuda_fail(c, e, "cell filter");
  c.cells_live = false;  // but for the lists below
  for (int k = 0; k < count; ++k) {
    CellsLeft& l = left[k];
    l.done = h[k].done != 0;
    memcpy(&l.reach, &h[k].L2, 4);
    l.reach = h[k].wide ? 0.0f : std::sqrt(l.reach);  // a finer grid is no remedy for that
    l.narrowed = !h[k].off && h[k].n_q > 0 && h[k].n_t > 0 && h[k].n_q <= run.cap_q[k] &&
                 h[k].n_t <= run.cap_t[k];
    l.q = run.q[k];
    l.nq = h[k].n_q;
    l.t = run.t[k];
    l.nt = h[k].n_t;
    c.cells_live |= !l.done && l.narrowed;
  }
  return HD_OK;
}

}  // namespace hdg
