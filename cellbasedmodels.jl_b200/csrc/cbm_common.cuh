// cbm_common.cuh — constants, the device counter block and the small
// device helpers shared by every kernel of the library.
//
// Arithmetic follows the reference's expression order with no FMA
// contraction (the library is built with -fmad=false), so float and double
// results are bit-identical to a CPU evaluation of the same expressions.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>

#include "../../include/cbm_b200.h"
#include "../../include/cbm_rng.h"

namespace cbm {

constexpr int kTile = 256;          // threads per block of the per-agent kernels
constexpr unsigned kFull = 0xffffffffu;
constexpr int kScanItems = 32;      // cells per thread in the cell scan (8192 per tile, so
                                    // the look-back spans few tiles)
constexpr int kScanTile = kTile * kScanItems;
constexpr long long kSpinLimit = 1ll << 20;  // bounded look-back wait

// Programmatic dependent launch.  A kernel launched with programmatic stream
// serialization is launched as the kernel before it on the stream completes,
// without the full gap between two launches; pdl_wait() returns once that
// kernel has completed and its writes are visible (at once for a plain
// launch), so a dependent kernel calls it before its first access to global
// memory.  No kernel here triggers its dependents early: blocks that wait
// resident for their predecessor would hold the SMs the concurrent branches
// of the step graph need.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Host side: launch kern on stream st, with programmatic stream
// serialization when `pdl` (then the operation before it on st must be a
// kernel launch, and kern calls pdl_wait() before its first global access).
// Errors are seen like those of <<<>>> launches, by cudaGetLastError.
// split: the preferred percentage of shared memory, -1 for the kernel's own.
template <typename... KP, typename... A>
inline void launch_split(cudaStream_t st, int split, bool pdl, void (*kern)(KP...), dim3 grid,
                         dim3 block, size_t smem, A&&... args) {
  cudaLaunchConfig_t lc = {};
  lc.gridDim = grid;
  lc.blockDim = block;
  lc.dynamicSmemBytes = smem;
  lc.stream = st;
  cudaLaunchAttribute at[2];
  lc.attrs = at;
  if (pdl) {
    at[lc.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[lc.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (split >= 0) {
    at[lc.numAttrs].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    at[lc.numAttrs++].val.sharedMemCarveout = (unsigned)split;
  }
  cudaLaunchKernelEx(&lc, kern, std::forward<A>(args)...);
}
template <typename... KP, typename... A>
inline void launch_serial(cudaStream_t st, bool pdl, void (*kern)(KP...), dim3 grid, dim3 block,
                          size_t smem, A&&... args) {
  launch_split(st, -1, pdl, kern, grid, block, smem, std::forward<A>(args)...);
}

// device error bits (cbm_sync reports the first as a status code)
enum : int {
  kErrAgentOverflow = 1 << 0,
  kErrNeighborOverflow = 1 << 1,
  kErrTimeout = 1 << 2,
};

// Device counters.  Values that a step both reads and produces are indexed
// by step parity p: a step of parity p reads [p] and writes [p ^ 1].
struct Counters {
  long long N[2];
  long long step[2];
  double t[2];
  long long n_add;      // NAdd_ of the step in flight
  long long n_remove;   // NRemove_
  long long id_max;     // idMax_
  long long id_base;    // idMax_ before this step's births
  long long children;   // births requested (including dropped ones)
  long long slots;      // working slots of the step that ended (N + NAdd)
  int flag[2];          // flagRecomputeNeighbors_ of the step of that parity
  int err;              // kErr* bits
  unsigned scan_ticket; // tile tickets of the cell scan
  unsigned scan_epoch;  // generation of the cell-scan tile states
  int resort;           // the step that ended re-sorts its agents (grid rebuild)
  int events;           // births or deaths in the step in flight
  int list_valid;       // the Verlet list matches the current slots
  int list_written;     // this step wrote the Verlet list lazily
  unsigned fate_ticket; // tile tickets of the fused rule / births kernel
  unsigned fate_epoch;  // generation of its tile states
  unsigned de_ticket;   // tile tickets of the force kernel (reset by its last block)
  unsigned de_done;     // blocks of the force kernel that have finished
  unsigned hist_done;   // blocks of the sort's histogram that have finished
  unsigned long long crowd;  // squares of the cells' counts, summed by the last scan (if asked)
};

// The commit of update!: the next parity's counters from those of parity p (N
// <- N + NAdd - NRemove, t += dt, step += 1: update.jl:201-298), and the
// re-sort decision of computeNeighbors!.
// One thread of one kernel of the step does it, once no other thread still
// reads the step's births, deaths and flag.
__device__ __forceinline__ void commit_counters(Counters* C, int p, double dt, bool resort) {
  C->slots = C->N[p] + C->n_add;
  C->N[p ^ 1] = C->N[p] + C->n_add - C->n_remove;
  C->n_add = 0;
  C->n_remove = 0;
  C->t[p ^ 1] = C->t[p] + dt;
  C->step[p ^ 1] = C->step[p] + 1;
  C->flag[p ^ 1] = 0;
  C->resort = resort ? 1 : 0;
  C->events = 0;
  if (C->list_written) C->list_valid = 1;
  C->list_written = 0;
}

template <typename T>
__device__ __forceinline__ T ld(const T* p) { return __ldg(p); }

// Julia's float `÷` on a >= 0: round((a - rem(a, b)) / b), which is the exact
// floor of a / b (quotients below 4e6).  Fast path: when the correctly
// rounded quotient f has a fractional part farther than m from 0 and 1, the
// exact quotient lies within half an ulp of f (< m) and so in the same unit
// interval, and floor(f) is that floor; otherwise the remainder formula runs.
__device__ __forceinline__ int floordiv(double a, double b) {
  const double f = a / b;
  const double n = floor(f);
  const double fr = f - n;  // exact below 2^52
  const double m = f * 1e-12 + 1e-14;
  if (fr > m && fr < 1.0 - m) return (int)n;
  return (int)rint((a - fmod(a, b)) / b);
}
__device__ __forceinline__ int floordiv(float a, float b) {
  const float f = a / b;
  const float n = floorf(f);
  const float fr = f - n;  // exact below 2^23
  const float m = f * 1e-5f + 1e-6f;
  if (fr > m && fr < 1.0f - m) return (int)n;
  return (int)rintf((a - fmodf(a, b)) / b);
}

// Square root and quotient of normal numbers far from the ends of the
// exponent range, without branches, so that several of them interleave (the
// general functions branch to handle zeros, subnormals and infinities, which
// keeps one pair's operations in series with the next's).  Both refine the
// hardware's approximation with fused operations and end in Markstein's
// correction step (P. Markstein, "Computation of elementary functions on the
// IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990): with h near
// 1 / (2 sqrt(x)) and g near sqrt(x), g + h (x - g^2) is the rounded root;
// with y the rounded reciprocal of b and q near a / b, q + y (a - b q) is the
// rounded quotient.
//
// They give the bits of the general operations.  Float32: every root of the
// range and the reciprocal of every divisor are compared.  Float64, with
// u = 2^-53 and an approximation good to 2^-18 (it is to 2^-20):
//  - Of the first iteration's errors, g and h share all but three roundings,
//    and the second halves what differs: both end within 2.5 u, and the last
//    step within 12 u^2 of the root before it rounds.  The result can be wrong
//    only if a midpoint of two numbers lies in between; there are 37 such x in
//    [1, 4), and these are compared at every exponent.
//  - inv is within 3.5 u of 1 / b, so y is 1 / b less at most (3.5 u)^2 of it,
//    rounded: the rounded reciprocal unless a midpoint lies in between, at
//    k u^2 / b from 1 / b with a whole k <= 12.  The quotient needs no more
//    than |b y - 1| b < 2 u (1 - u) for b in [1, 2), since a - b m is a
//    multiple of u times the spacing for every midpoint m; a y that is not the
//    rounded one keeps to that too, unless b >= 2 - 12 u.  There the k of the
//    number 2 - 2 n u is n^2 for odd n (for even n no midpoint is near), and
//    errors are below 2.5 u, which leaves n = 1, the significand of ones: its y
//    may be the power of two, and the quotient of a power of two then ends in
//    a tie.  mid_root keeps the x with that root from here.  Also, q may be off
//    by more than one place for both a and b among the last numbers of their
//    binades, and these are compared.
__device__ __forceinline__ float sqrt_mid(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  float g = x * y;
  float h = 0.5f * y;
  const float r = __fmaf_rn(-g, h, 0.5f);
  g = __fmaf_rn(g, r, g);
  h = __fmaf_rn(h, r, h);
  return __fmaf_rn(__fmaf_rn(-g, g, x), h, g);
}
__device__ __forceinline__ float div_mid(float a, float b) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
  y = __fmaf_rn(__fmaf_rn(-b, y, 1.f), y, y);
  const float q = a * y;
  return __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
}
// (the forms of the two types alike, for templates)
__device__ __forceinline__ float sqrt_mid(float x, float* inv) {
  *inv = 0.f;
  return sqrt_mid(x);
}
__device__ __forceinline__ float div_mid(float a, float b, float) { return div_mid(a, b); }
// *inv: 1 / sqrt(x) to about an ulp, from which div_mid starts
__device__ __forceinline__ double sqrt_mid(double x, double* inv) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  double g = x * y;
  double h = 0.5 * y;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const double r = __fma_rn(-g, h, 0.5);
    g = __fma_rn(g, r, g);
    h = __fma_rn(h, r, h);
  }
  *inv = h + h;
  return __fma_rn(__fma_rn(-g, g, x), h, g);
}
// y: of sqrt_mid, whose root b is, for an x that mid_root takes
__device__ __forceinline__ double div_mid(double a, double b, double y) {
  y = __fma_rn(__fma_rn(-b, y, 1.0), y, y);
  const double q = a * y;
  return __fma_rn(__fma_rn(-b, q, a), y, q);
}

// Whether div_mid takes the root of x as a divisor: a root of ones has an x of
// 4^k (4 - 2^-50) or 4^k (4 - 2^-51).  (One comparison of the low word, which
// a few other x fail: the Float64 walk of 1.5e5 agents takes 248 us with it,
// 245 without.  Setting the bit of y instead: 248, and 3 % in communities of a
// few hundred, which lose nothing so.)
__device__ __forceinline__ bool mid_root(float) { return true; }
__device__ __forceinline__ bool mid_root(double x) {
  return (unsigned)__double2loint(x) < 0xfffffffeu;
}

// cellPos, src/neighbors.jl:636-638, 0-based; a NaN coordinate goes to the
// first cell
template <typename T>
__device__ __forceinline__ int cell_pos1(T edge, T x, T lo, T hi, int n) {
  if (x > hi) return n - 1;
  if (!(x >= lo)) return 0;
  int p = floordiv(x - lo, edge) + 1;
  return p > n - 1 ? n - 1 : p;
}

// linear cell of a point, x fastest
template <typename T, int D>
__device__ __forceinline__ int cell_of(T edge, const T* lo, const T* hi, const int* nc,
                                       const T* x) {
  int lin = cell_pos1<T>(edge, x[0], lo[0], hi[0], nc[0]);
  if (D > 1) lin += nc[0] * cell_pos1<T>(edge, x[1], lo[1], hi[1], nc[1]);
  if (D > 2) lin += nc[0] * nc[1] * cell_pos1<T>(edge, x[2], lo[2], hi[2], nc[2]);
  return lin;
}

// cellInMesh, src/metrics.jl:18-20 (0-based, clamped at the top)
template <typename T>
__device__ __forceinline__ int cell_in_mesh(T dx, T x, T lo, T hi, int n) {
  if (x > hi) return n - 1;
  if (!(x >= lo)) return 0;
  int p = floordiv(x - lo, dx);
  return p > n - 1 ? n - 1 : p;
}

// cellPosNeigh, src/neighbors.jl:658-708: k-th of 3^D cells, x fastest,
// -1 outside the grid
template <int D>
__device__ __forceinline__ int cell_neigh(const int* nc, const int* q, int k) {
  int px = q[0] + (k % 3) - 1;
  if (px < 0 || px >= nc[0]) return -1;
  int lin = px;
  if (D > 1) {
    int py = q[1] + ((k / 3) % 3) - 1;
    if (py < 0 || py >= nc[1]) return -1;
    lin += nc[0] * py;
  }
  if (D > 2) {
    int pz = q[2] + (k / 9) - 1;
    if (pz < 0 || pz >= nc[2]) return -1;
    lin += nc[0] * nc[1] * pz;
  }
  return lin;
}

template <int D>
__device__ __forceinline__ void cell_coords(const int* nc, int pos, int* q) {
  q[0] = pos % nc[0];
  if (D > 1) q[1] = (pos / nc[0]) % nc[1];
  if (D > 2) q[2] = pos / (nc[0] * nc[1]);
}

// exclusive block scan of one int per thread (kTile threads)
__device__ __forceinline__ int block_exscan(int v, int* warp_sums, int* total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(kFull, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[w] = x;
  __syncthreads();
  if (w == 0) {
    int s = lane < kTile / 32 ? warp_sums[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(kFull, s, o);
      if (lane >= o) s += y;
    }
    if (lane < kTile / 32) warp_sums[lane] = s;
  }
  __syncthreads();
  int prefix = w > 0 ? warp_sums[w - 1] : 0;
  *total = warp_sums[kTile / 32 - 1];
  __syncthreads();
  return prefix + x - v;
}

// ---------------------------------------------------------------------------
// exclusive scan of per-cell counts (cumsum .- counts, src/neighbors.jl:934-937)
// in one pass with decoupled look-back.  Tiles take tickets in launch order so
// a tile only waits on tiles that are already running; the wait is bounded.
// Counts are zeroed for the next build.  The preceding histogram kernel resets
// the ticket counter and advances the tile-state epoch.
// ---------------------------------------------------------------------------
struct ScanArgs {
  int* count;                      // n counts, zeroed on exit
  int* start;                      // n + 1 exclusive offsets
  unsigned long long* state;       // n_tiles tile states: epoch | flag | value
  int n;
  int n_tiles;
  Counters* ctr;
  const int* due;                  // skip the scan when *due == 0 (nullptr: always)
  // the scan also commits the counters of a step of parity p that always
  // re-sorts, whose force kernel made the histogram
  int commit = 0;
  int crowd = 0;                   // add the squares of the counts to the counters' crowd
  int parity = 0;
  double dt = 0.0;
};

// Shared-memory index of cell k of a tile: one padding word per 32 cells, so
// that a thread reading its 32 consecutive cells hits 32 different banks.
__device__ __forceinline__ int scan_pad(int k) { return k + (k >> 5); }

static __global__ void __launch_bounds__(kTile) k_scan_cells(ScanArgs A) {
  __shared__ int warp_sums[kTile / 32];
  __shared__ unsigned s_tile;
  __shared__ int s_prefix;
  __shared__ int s_cells[kScanTile + kScanTile / 32];
  pdl_wait();
  if (A.due && *A.due == 0) return;
  Counters* C = A.ctr;
  const unsigned epoch = C->scan_epoch;
  if (threadIdx.x == 0) s_tile = atomicAdd(&C->scan_ticket, 1u);
  __syncthreads();
  const int tile = (int)s_tile;
  if (tile >= A.n_tiles) {  // tickets were not reset: never index past the tile states
    if (threadIdx.x == 0) atomicOr(&C->err, kErrTimeout);
    return;
  }
  static_assert(kScanItems % 4 == 0 && kScanItems == 32, "int4 staging, 32 cells per thread");
  const int tile_base = tile * kScanTile;
  const bool full = tile_base + kScanTile <= A.n;
  // coalesced load of the tile's counts into shared memory
  if (full) {
#pragma unroll
    for (int v = 0; v < kScanItems / 4; ++v) {
      const int q = v * kTile + threadIdx.x;  // int4 index inside the tile
      const int4 a = reinterpret_cast<const int4*>(A.count + tile_base)[q];
      s_cells[scan_pad(4 * q)] = a.x;
      s_cells[scan_pad(4 * q + 1)] = a.y;
      s_cells[scan_pad(4 * q + 2)] = a.z;
      s_cells[scan_pad(4 * q + 3)] = a.w;
    }
  } else {
    for (int k = threadIdx.x; k < kScanTile; k += kTile)
      s_cells[scan_pad(k)] = tile_base + k < A.n ? A.count[tile_base + k] : 0;
  }
  __syncthreads();
  const int first = threadIdx.x * kScanItems;  // this thread's cells inside the tile
  int vals[kScanItems];
  int sum = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    vals[k] = s_cells[scan_pad(first + k)];
    sum += vals[k];
  }
  if (A.crowd) {
    unsigned long long sq = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) sq += (unsigned long long)vals[k] * (unsigned)vals[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(kFull, sq, o);
    if ((threadIdx.x & 31) == 0 && sq) atomicAdd(&C->crowd, sq);
  }
  int total;
  int ex = block_exscan(sum, warp_sums, &total);
  const unsigned long long ep = (unsigned long long)epoch << 32;
  if (threadIdx.x < 32) {
    // warp look-back: lane l inspects tile (t - l); stop at the nearest tile
    // that has published its inclusive prefix, summing aggregates before it
    const int lane = threadIdx.x;
    if (tile == 0) {
      if (lane == 0) {
        s_prefix = 0;
        atomicExch(A.state, ep | (2ull << 30) | (unsigned)total);
      }
    } else {
      if (lane == 0) atomicExch(A.state + tile, ep | (1ull << 30) | (unsigned)total);
      int prefix = 0;
      int t = tile - 1;
      long long spins = 0;
      while (true) {
        const int idx = t - lane;
        unsigned flag = 2u, val = 0u;  // before tile 0: an inclusive prefix of 0
        if (idx >= 0) {
          unsigned long long s = atomicAdd(A.state + idx, 0ull);
          flag = ((s >> 32) == epoch) ? (unsigned)(s >> 30) & 3u : 0u;
          val = (unsigned)(s & 0x3fffffffu);
        }
        const unsigned incl = __ballot_sync(kFull, flag == 2u);
        const unsigned pend = __ballot_sync(kFull, flag == 0u);
        // lanes up to and including the first inclusive one must be ready
        const unsigned upto = incl ? ((incl & (0u - incl)) << 1) - 1u : kFull;
        if (pend & upto) {
          if (++spins > kSpinLimit) {
            if (lane == 0) atomicOr(&C->err, kErrTimeout);
            break;
          }
          continue;
        }
        unsigned mine = ((1u << lane) & upto) ? val : 0u;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(kFull, mine, o);
        prefix += (int)mine;
        if (incl) break;
        t -= 32;
      }
      if (lane == 0) {
        s_prefix = prefix;
        atomicExch(A.state + tile, ep | (2ull << 30) | (unsigned)(prefix + total));
      }
    }
  }
  __syncthreads();
  // exclusive offsets back into shared memory, then coalesced stores
  int run = s_prefix + ex;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    s_cells[scan_pad(first + k)] = run;
    run += vals[k];
  }
  // the thread holding the last cell writes the end sentinel
  if (A.n - 1 >= tile_base + first && A.n - 1 < tile_base + first + kScanItems) A.start[A.n] = run;
  __syncthreads();
  if (full) {
    // start is only 4-byte aligned for a shifted array, so it is written as
    // plain ints; counts are cleared as int4
#pragma unroll 8
    for (int k = threadIdx.x; k < kScanTile; k += kTile) A.start[tile_base + k] = s_cells[scan_pad(k)];
#pragma unroll
    for (int v = 0; v < kScanItems / 4; ++v)
      reinterpret_cast<int4*>(A.count + tile_base)[v * kTile + threadIdx.x] = make_int4(0, 0, 0, 0);
  } else {
    for (int k = threadIdx.x; k < kScanTile; k += kTile)
      if (tile_base + k < A.n) {
        A.start[tile_base + k] = s_cells[scan_pad(k)];
        A.count[tile_base + k] = 0;
      }
  }
  if (A.commit && tile == 0 && threadIdx.x == 0) commit_counters(C, A.parity, A.dt, true);
}

}  // namespace cbm
