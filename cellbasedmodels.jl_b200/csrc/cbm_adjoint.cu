// cbm_adjoint.cu — exact gradients of a trajectory loss with respect to the
// interaction parameters and the initial positions, by a hand-written
// reverse (adjoint) sweep of the force + Euler step with checkpointing.
//
// Forward map (the 3D soft-sphere ODE of the reference's agentODE with
// Euler, src/integrators.jl:465-505): x_{n+1} = x_n + dt F(x_n; theta),
//   F_i = sum_j f(r_ij),  f(r) = (F(d)/d) r,  r = x_i - x_j, d = |r|,
//   F(d) = k (rho - d) for d < rho,  -a (d - rho) for rho <= d < r_att,
// with theta = (k, a, rho = 2r) and r_att = 3r.  Loss L = mean over agents and
// axes of (x_T - x*)^2.  Adjoint (lambda_n = dL/dx_n):
//   lambda_T = 2 (x_T - x*) / (3N)
//   lambda_n = lambda_{n+1} + dt J_n^T lambda_{n+1},
//   (J^T l)_i = sum_j [ s (l_i - l_j) + c r (r . (l_i - l_j)) ],
//     s = F/d,  c = (F'(d) d - F) / d^3   (the Hessian of the pair term is
//     s I + c r r^T, symmetric, and f_ji = -f_ij)
//   dL/dtheta += dt sum_i lambda_{n+1,i} . sum_j (dF/dtheta / d) r_ij.
// The cutoff r_att is held fixed in the derivative (a pair crossing it
// changes the force discontinuously; that measure-zero event has no
// derivative), which is also what forward-mode dual numbers of the same
// program compute.
//
// Memory: checkpoints every `checkpoint_every` steps; a segment is recomputed
// from its checkpoint, keeping each step's slot positions and interacting
// pairs, and then swept backwards, so long trajectories need O(T/K + K)
// states instead of O(T).  The last segment's are kept by the forward sweep
// itself, into the same buffers, and not computed twice.
//
// Layout and launches.  States are double4/float4 in index order.  A step is
// four kernels: the scan of the cell counts, the scatter, the placement of
// the positions in slot order (cells x fastest, ascending index inside a
// cell; the agent index rides in w), and the Euler step by tiles of 32 slots
// (cbm_tile.cuh), which also files the new positions in their cells.  They
// follow one another by programmatic launches.  A backward step is one kernel
// over the recorded pairs, four lanes an agent (at 65536 agents one lane
// leaves 3.5 warps a scheduler, each in a serial chain); it reads the
// partners' lambda by their index.  All buffers of a shape (n, steps, checkpoint interval) are
// kept, and the whole device part of a run is one CUDA graph replayed by
// later runs of the same shape; host copies of the inputs and results stay
// outside the graph.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/cbm_b200.h"
#include "cbm_tile.cuh"

using namespace cbm;

namespace {

template <typename T>
struct AV4;
template <>
struct AV4<float> {
  using type = float4;
  __device__ static float enc(int i) { return __int_as_float(i); }
  __device__ static int dec(float w) { return __float_as_int(w); }
};
template <>
struct AV4<double> {
  using type = double4;
  __device__ static double enc(int i) { return __longlong_as_double((long long)i); }
  __device__ static int dec(double w) { return (int)__double_as_longlong(w); }
};

template <typename T>
struct AdjParams {
  using V4 = typename AV4<T>::type;
  const V4* x;          // state, index order
  V4* xn;               // x_{n+1}, index order (forward)
  V4* xs;               // x_n in slot order, w = agent index
  const V4* lam;        // lambda_{n+1}, index order (backward)
  V4* lam_out;          // lambda_n
  int* cell_count;
  const int* cell_start;
  int* agent_cell;      // per agent: cell of the state filed last, rank in it
  int* agent_rank;
  int* cell_tmp;        // agents by cell, in arrival order
  int* cell_of_slot;    // cell of each slot of xs
  int* pair_n;          // per slot: partners with a force term (recorded steps), or null
  int* pair_list;       // entry k of slot s at k * n + s: the partner's slot
  int cap;
  bool file;            // the step files x_{n+1} in its cells
  bool mid;             // the stiffnesses suit sqrt_mid and div_mid
  double* gpart;        // per block: running dL/dtheta partials (3 per block)
  Counters* ctr;
  int n;
  int nc[3];
  T lo[3], hi[3];
  T edge;
  T dt, k, a, rho, ratt, cut2;
};

constexpr int kLanes = 4;                // lanes an agent (backward)
constexpr int kSlots = kTile / kLanes;   // slots a block

// fresh tickets and tile states for the scan that follows
template <typename T>
__device__ __forceinline__ void adj_scan_begin(const AdjParams<T>& A) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    A.ctr->scan_ticket = 0u;
    A.ctr->scan_epoch = A.ctr->scan_epoch + 1u;
  }
}

// agent i at v filed in its cell (assignCells, neighbors.jl:763-821)
template <typename T>
__device__ __forceinline__ void adj_file(const AdjParams<T>& A, int i, const T* x) {
  const int c = cell_of<T, 3>(A.edge, A.lo, A.hi, A.nc, x);
  A.agent_cell[i] = c;
  A.agent_rank[i] = atomicAdd(A.cell_count + c, 1);
}

template <typename T>
__global__ void __launch_bounds__(kTile) k_adj_file(AdjParams<T> A) {
  pdl_wait();
  adj_scan_begin(A);
  const int i = blockIdx.x * kTile + threadIdx.x;
  if (i >= A.n) return;
  const typename AV4<T>::type v = A.x[i];
  const T x[3] = {v.x, v.y, v.z};
  adj_file(A, i, x);
}

template <typename T>
__global__ void __launch_bounds__(kTile) k_adj_scatter(AdjParams<T> A) {
  pdl_wait();
  const int i = blockIdx.x * kTile + threadIdx.x;
  if (i >= A.n) return;
  A.cell_tmp[A.cell_start[A.agent_cell[i]] + A.agent_rank[i]] = i;
}

// rank among the cell's agents with a smaller index (neighbors.jl:851-862)
template <typename T>
__global__ void __launch_bounds__(kTile) k_adj_place(AdjParams<T> A) {
  pdl_wait();
  const int i = blockIdx.x * kTile + threadIdx.x;
  if (i >= A.n) return;
  typename AV4<T>::type v = A.x[i];
  const int c = A.agent_cell[i];
  const int s0 = A.cell_start[c], s1 = A.cell_start[c + 1];
  int r = 0;
  for (int s = s0; s < s1; ++s) r += A.cell_tmp[s] < i;
  v.w = AV4<T>::enc(i);
  A.xs[s0 + r] = v;
  A.cell_of_slot[s0 + r] = c;
}

// three index-ordered arrays <-> states
template <typename T>
__global__ void __launch_bounds__(kTile) k_adj_pack(const T* x0, const T* x1, const T* x2,
                                                    typename AV4<T>::type* out, int n) {
  const int i = blockIdx.x * kTile + threadIdx.x;
  if (i >= n) return;
  typename AV4<T>::type v;
  v.x = x0[i];
  v.y = x1[i];
  v.z = x2[i];
  v.w = (T)0;
  out[i] = v;
}
template <typename T>
__global__ void __launch_bounds__(kTile) k_adj_unpack(const typename AV4<T>::type* in, T* x0, T* x1,
                                                      T* x2, int n) {
  const int i = blockIdx.x * kTile + threadIdx.x;
  if (i >= n) return;
  const typename AV4<T>::type v = in[i];
  x0[i] = v.x;
  x1[i] = v.y;
  x2[i] = v.z;
}

// a checkpoint (a kernel, so that the step after it may launch programmatically)
template <typename T>
__global__ void __launch_bounds__(kTile) k_adj_keep(const typename AV4<T>::type* x,
                                                    typename AV4<T>::type* out, int n) {
  const int i = blockIdx.x * kTile + threadIdx.x;
  if (i < n) out[i] = x[i];
}

// square root and quotient of the pair terms: the branch-free forms where
// they are exact (every recorded pair is closer than the cutoff)
template <typename T>
__device__ __forceinline__ T adj_sqrt(bool mid, T x, T* inv) {
  if (mid) {
    if constexpr (sizeof(T) == 8) return sqrt_mid(x, inv);
    else return sqrt_mid(x);
  }
  return sqrt(x);
}
template <typename T>
__device__ __forceinline__ T adj_div(bool mid, T a, T b, T inv) {
  if (mid) {
    if constexpr (sizeof(T) == 8) return div_mid(a, b, inv);
    else return div_mid(a, b);
  }
  return a / b;
}

template <typename T>
__device__ __forceinline__ T adj_diff(const T* xi, const typename AV4<T>::type& o, T* e) {
  e[0] = xi[0] - o.x;
  T s2 = e[0] * e[0];
  e[1] = xi[1] - o.y;
  s2 = s2 + e[1] * e[1];
  e[2] = xi[2] - o.z;
  return s2 + e[2] * e[2];
}

// forward Euler step by tiles of 32 slots (cbm_tile.cuh): the reference's
// expression order, cells x fastest, ascending index inside a cell (the plain
// path's CellLinked sums).  A recorded step keeps the slots of the partners
// that carry a force term, in that order.
template <typename T>
__global__ void __launch_bounds__(32, kTileWarps) k_adj_step(Params<T> P, AdjParams<T> A) {
  __shared__ TileSmem S;
  pdl_wait();
  if (A.file) adj_scan_begin(A);
  tile_begin(S);
  const int s0 = blockIdx.x * 32, s = s0 + (int)threadIdx.x;
  if (s0 >= A.n) return;
  const typename AV4<T>::type me = A.xs[s < A.n ? s : A.n - 1];
  const T xi[3] = {me.x, me.y, me.z};
  T acc[3] = {(T)0, (T)0, (T)0};
  int m = 0;
  int* const list = A.pair_n ? A.pair_list + s : nullptr;
  tile_forces<T>(P, S, A.n, s0, xi, acc, [&](int q) {
    if (list && m < A.cap) list[(long long)m * A.n] = q;
    ++m;
  });
  if (s >= A.n) return;
  if (A.pair_n) {
    A.pair_n[s] = m < A.cap ? m : A.cap;
    if (m > A.cap) atomicOr(&A.ctr->err, kErrNeighborOverflow);
  }
  const int i = AV4<T>::dec(me.w);
  const T xn[3] = {xi[0] + acc[0] * A.dt, xi[1] + acc[1] * A.dt, xi[2] + acc[2] * A.dt};
  typename AV4<T>::type out;
  out.x = xn[0];
  out.y = xn[1];
  out.z = xn[2];
  out.w = (T)0;
  A.xn[i] = out;
  if (A.file) adj_file(A, i, xn);
}

// one backward step at state x_n: lambda_n from lambda_{n+1} over the pairs
// recorded by the forward step, and this step's dL/dtheta terms added to the
// block's running partial sums.  The lanes of an agent take its pairs in turn
// and their sums meet in a fixed tree.
template <typename T>
__global__ void __launch_bounds__(kTile) k_adj_backward(AdjParams<T> A) {
  __shared__ double red[3][kTile / 32];
  pdl_wait();
  const int s = blockIdx.x * kSlots + (int)threadIdx.x / kLanes;
  const int lane = threadIdx.x & 31, u = lane & (kLanes - 1);
  T adj[3] = {(T)0, (T)0, (T)0};
  T th[3] = {(T)0, (T)0, (T)0};  // k, a, rho
  T li[3] = {(T)0, (T)0, (T)0};
  int i = 0;
  if (s < A.n) {
    const typename AV4<T>::type me = A.xs[s];
    i = AV4<T>::dec(me.w);
    const typename AV4<T>::type lm = A.lam[i];
    const T xi[3] = {me.x, me.y, me.z};
    li[0] = lm.x;
    li[1] = lm.y;
    li[2] = lm.z;
    const int m = A.pair_n[s];
    const int* const list = A.pair_list + s;
    int t = u < m ? list[(long long)u * A.n] : s;
    for (int kk = u; kk < m; kk += kLanes) {
      const typename AV4<T>::type o = A.xs[t];
      if (kk + kLanes < m) t = list[(long long)(kk + kLanes) * A.n];
      const typename AV4<T>::type lo = A.lam[AV4<T>::dec(o.w)];
      T r[3];
      const T s2 = adj_diff(xi, o, r);
      const bool mid = A.mid && s2 > (T)1e-12 && mid_root(s2);
      T inv0 = (T)0;
      const T dd = adj_sqrt(mid, s2, &inv0);  // every recorded pair has dd < r_att
      const bool rep = dd < A.rho;
      const T kk_ = rep ? A.k : A.a;
      const T gap = A.rho - dd;
      const T F = kk_ * gap;
      const T inv = adj_div(mid, (T)1, dd, inv0);
      const T sc = F * inv;
      const T c = (-kk_ * dd - F) * inv * inv * inv;
      const T dl[3] = {li[0] - lo.x, li[1] - lo.y, li[2] - lo.z};
      T rdl = (T)0, rli = (T)0;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        rdl += r[d] * dl[d];
        rli += r[d] * li[d];
      }
#pragma unroll
      for (int d = 0; d < 3; ++d) adj[d] += sc * dl[d] + c * rdl * r[d];
      const T w = inv * rli;
      th[0] += rep ? gap * w : (T)0;
      th[1] += rep ? (T)0 : gap * w;
      th[2] += kk_ * w;
    }
  }
#pragma unroll
  for (int o = 1; o < kLanes; o <<= 1)
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      adj[d] += __shfl_xor_sync(kFull, adj[d], o);
      th[d] += __shfl_xor_sync(kFull, th[d], o);
    }
  if (s < A.n && u == 0) {
    typename AV4<T>::type out;
    out.x = li[0] + A.dt * adj[0];
    out.y = li[1] + A.dt * adj[1];
    out.z = li[2] + A.dt * adj[2];
    out.w = (T)0;
    A.lam_out[i] = out;
  }
  // deterministic block sum (fixed tree), added to this block's running sum
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    double g = (double)(A.dt * th[q]);
#pragma unroll
    for (int o = kLanes; o < 32; o <<= 1) g += __shfl_xor_sync(kFull, g, o);
    if (lane == 0) red[q][threadIdx.x >> 5] = g;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double g = 0.0;
#pragma unroll
    for (int w = 0; w < kTile / 32; ++w) g += red[threadIdx.x][w];
    A.gpart[blockIdx.x * 3 + threadIdx.x] += g;
  }
}

// lambda_T = 2 (x_T - x*) / (3N) and per-block partial sums of the loss
template <typename T>
__global__ void __launch_bounds__(kTile) k_adj_loss(const typename AV4<T>::type* x, const T* tgt0,
                                                    const T* tgt1, const T* tgt2,
                                                    typename AV4<T>::type* lam, int n,
                                                    double* lpart) {
  __shared__ double red[kTile];
  const int i = blockIdx.x * kTile + threadIdx.x;
  double l = 0.0;
  if (i < n) {
    const T inv3n = (T)2 / (T)(3.0 * (double)n);
    const typename AV4<T>::type v = x[i];
    const T e[3] = {v.x - tgt0[i], v.y - tgt1[i], v.z - tgt2[i]};
    typename AV4<T>::type o;
    o.x = inv3n * e[0];
    o.y = inv3n * e[1];
    o.z = inv3n * e[2];
    o.w = (T)0;
    lam[i] = o;
#pragma unroll
    for (int d = 0; d < 3; ++d) l += (double)e[d] * (double)e[d];
  }
  red[threadIdx.x] = l;
  __syncthreads();
  for (int o = kTile / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) lpart[blockIdx.x] = red[0];
}

// Device buffers and the captured graph of one run shape.
struct Plan {
  int n = -1, nsteps = -1, K = -1;
  bool backward = false;
  std::vector<void*> bufs;
  cudaGraphExec_t graph = nullptr;
  void* in_x[3] = {};    // x0 (index order)
  void* in_tgt[3] = {};  // target
  void* out_xT[3] = {};  // x_T (inside a state buffer)
  void* out_dx0[3] = {}; // lambda_0
  double* gpart = nullptr;
  double* lpart = nullptr;
  int blocks = 1;        // of one thread an agent (lpart)
  int step_blocks = 1;   // of kLanes threads an agent (gpart)
  void release() {
    if (graph) cudaGraphExecDestroy(graph);
    graph = nullptr;
    for (void* p : bufs) cudaFree(p);
    bufs.clear();
    n = nsteps = K = -1;
  }
};

}  // namespace

struct cbm_adjoint {
  cbm_config cfg{};
  int device = 0;
  cudaStream_t stream = nullptr;
  std::string err;
  std::vector<void*> allocs;
  size_t ts = 8;
  int n_max = 0;
  int nc[3] = {1, 1, 1};
  int n_cells = 1;
  int n_tiles = 1;
  int cap = 64;          // pair-row capacity of the recompute pass
  // grid scratch
  int* cell_count = nullptr;
  unsigned long long* scan_state = nullptr;
  int* agent_cell = nullptr;
  int* agent_rank = nullptr;
  int* cell_tmp = nullptr;
  int* cell_of_slot = nullptr;
  Counters* ctr = nullptr;
  Plan plan[2];          // [0] forward only, [1] forward + backward
};

namespace {

std::string g_adj_error;

int afail(cbm_adjoint* a, int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  if (a) a->err = buf;
  else g_adj_error = buf;
  return code;
}

#define ACUDA(a, call)                                                                    \
  do {                                                                                    \
    cudaError_t e_ = (call);                                                              \
    if (e_ != cudaSuccess)                                                                \
      return afail(a, CBM_ERR_CUDA, "%s failed: %s", #call, cudaGetErrorString(e_));      \
  } while (0)

template <typename T>
AdjParams<T> adj_params(cbm_adjoint* a, int n) {
  AdjParams<T> A;
  memset(&A, 0, sizeof A);
  const cbm_config& k = a->cfg;
  A.n = n;
  for (int d = 0; d < 3; ++d) {
    A.nc[d] = a->nc[d];
    A.lo[d] = (T)k.box_lo[d];
    A.hi[d] = (T)k.box_hi[d];
  }
  A.edge = (T)k.cell_edge;
  A.dt = (T)k.dt;
  A.k = (T)k.k_rep;
  A.a = (T)k.k_att;
  A.rho = (T)k.r_rep;
  A.ratt = (T)k.r_att;
  const double c = std::max(k.r_rep, k.r_att), up = c * c * (1.0 + 1e-5);
  const T t = (T)up;
  A.cut2 = (double)t < up ? std::nextafter(t, (T)INFINITY) : t;
  auto mid = [](double v) { return v == 0.0 || (std::fabs(v) > 1e-12 && std::fabs(v) < 1e12); };
  A.mid = mid(k.k_rep) && mid(k.k_att) && c < 1e5;
  A.cap = a->cap;
  A.ctr = a->ctr;
  A.cell_count = a->cell_count;
  A.agent_cell = a->agent_cell;
  A.agent_rank = a->agent_rank;
  A.cell_tmp = a->cell_tmp;
  A.cell_of_slot = a->cell_of_slot;
  return A;
}

// The grid of A.x (already filed in its cells) into A.xs, and the Euler step
// from there to A.xn.  Every kernel follows a kernel on the stream.
template <typename T>
void enqueue_step(cbm_adjoint* a, const AdjParams<T>& A, int* starts, int blocks) {
  ScanArgs S;
  S.count = a->cell_count;
  S.start = starts;
  S.state = a->scan_state;
  S.n = a->n_cells;
  S.n_tiles = a->n_tiles;
  S.ctr = a->ctr;
  S.due = nullptr;
  launch_serial(a->stream, true, k_scan_cells, dim3(a->n_tiles), dim3(kTile), 0, S);
  launch_serial(a->stream, true, k_adj_scatter<T>, dim3(blocks), dim3(kTile), 0, A);
  launch_serial(a->stream, true, k_adj_place<T>, dim3(blocks), dim3(kTile), 0, A);
  Params<T> P;
  memset(&P, 0, sizeof P);
  P.PA = A.xs;
  P.cell_of_slot = A.cell_of_slot;
  P.cell_start = starts;
  for (int d = 0; d < 3; ++d) {
    P.n_cells_d[d] = A.nc[d];
    P.box_lo[d] = A.lo[d];
    P.box_hi[d] = A.hi[d];
  }
  P.edge = A.edge;
  P.cut2 = A.cut2;
  const double c = std::max(a->cfg.r_rep, a->cfg.r_att);
  P.tile_scale = (T)tile_scale(c, a->cfg.cell_edge);
  P.tile_cut = tile_cut(c, a->cfg.cell_edge);
  P.k_rep = A.k;
  P.r_rep = A.rho;
  P.k_att = A.a;
  P.r_att = A.ratt;
  P.att_form = CBM_ATT_FROM_REP;
  launch_serial(a->stream, true, k_adj_step<T>, dim3((A.n + 31) / 32 + (A.n == 0)), dim3(32), 0, P,
                A);
}

// Buffers of a shape and the enqueue of its device work (captured once).
template <typename T>
int make_plan(cbm_adjoint* a, Plan& P, int n, int nsteps, int K, bool backward) {
  using V4 = typename AV4<T>::type;
  P.release();
  const size_t S = sizeof(T), n1 = (size_t)std::max(n, 1), nb = n1 * S, nv = n1 * sizeof(V4);
  const int blocks = n > 0 ? (n + kTile - 1) / kTile : 1;
  const int step_blocks = n > 0 ? (n + kSlots - 1) / kSlots : 1;
  const int nseg = backward ? std::max((nsteps + K - 1) / K, 1) : 0;
  const size_t Kb = backward ? (size_t)K : 1;  // steps kept at once
  bool ok = true;
  auto get = [&](size_t bytes) -> void* {
    void* p = nullptr;
    if (!ok || cudaMalloc(&p, bytes ? bytes : 16) != cudaSuccess) {
      ok = false;
      return nullptr;
    }
    P.bufs.push_back(p);
    return p;
  };
  T* tgt[3] = {};
  V4* lam[2] = {};
  for (int d = 0; d < 3; ++d) {
    P.in_x[d] = get(nb);
    P.out_xT[d] = get(nb);
    if (backward) {
      tgt[d] = (T*)get(nb);
      P.in_tgt[d] = tgt[d];
      P.out_dx0[d] = get(nb);
    }
  }
  V4* fw[2] = {(V4*)get(nv), (V4*)get(nv)};
  V4* ckpt = backward ? (V4*)get(nv * (size_t)nseg) : nullptr;
  if (backward)
    for (int q = 0; q < 2; ++q) lam[q] = (V4*)get(nv);
  int* starts = (int*)get((size_t)(a->n_cells + 1) * 4);
  V4* xs = (V4*)get(nv * Kb);
  int* pair_n = backward ? (int*)get(n1 * 4 * Kb) : nullptr;
  int* pair_list = backward ? (int*)get(n1 * 4 * (size_t)a->cap * Kb) : nullptr;
  P.gpart = (double*)get((size_t)step_blocks * 3 * 8);
  P.lpart = (double*)get((size_t)blocks * 8);
  if (!ok) {
    P.release();
    return afail(a, CBM_ERR_NOMEM, "adjoint buffers do not fit");
  }
  P.n = n;
  P.nsteps = nsteps;
  P.K = K;
  P.backward = backward;
  P.blocks = blocks;
  P.step_blocks = step_blocks;
  cudaStream_t st = a->stream;
  cudaGraph_t g = nullptr;
  // a step from cur to nxt; kept (slot positions and pairs) in place m of the
  // segment, or, m < 0, its positions in place 0 and no pairs
  auto step = [&](const V4* cur, V4* nxt, int m, bool file) {
    AdjParams<T> A = adj_params<T>(a, n);
    const size_t at = (size_t)(m < 0 ? 0 : m) * n1;
    A.x = cur;
    A.xn = nxt;
    A.xs = xs + at;
    A.cell_start = starts;
    A.pair_n = m < 0 ? nullptr : pair_n + at;
    A.pair_list = m < 0 ? nullptr : pair_list + at * (size_t)a->cap;
    A.file = file;
    enqueue_step<T>(a, A, starts, blocks);
  };
  auto file_state = [&](const V4* x) {
    AdjParams<T> A = adj_params<T>(a, n);
    A.x = x;
    k_adj_file<T><<<blocks, kTile, 0, st>>>(A);
  };
  ACUDA(a, cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
  // forward sweep, keeping a checkpoint at the start of every segment but the
  // last, whose steps are kept as they are made
  k_adj_pack<T><<<blocks, kTile, 0, st>>>((const T*)P.in_x[0], (const T*)P.in_x[1],
                                          (const T*)P.in_x[2], fw[0], n);
  const int last0 = (nseg - 1) * K;  // first step of the last segment
  if (nsteps) file_state(fw[0]);
  for (int s = 0; s < nsteps; ++s) {
    const V4* cur = fw[s % 2];
    const bool kept = backward && s >= last0;
    step(cur, fw[(s + 1) % 2], kept ? s - last0 : -1, s + 1 < nsteps);
    if (backward && !kept && s % K == 0)
      k_adj_keep<T><<<blocks, kTile, 0, st>>>(cur, ckpt + (size_t)(s / K) * n1, n);
  }
  V4* xT = fw[nsteps % 2];
  k_adj_unpack<T><<<blocks, kTile, 0, st>>>(xT, (T*)P.out_xT[0], (T*)P.out_xT[1], (T*)P.out_xT[2], n);
  if (backward) {
    k_adj_loss<T><<<blocks, kTile, 0, st>>>(xT, tgt[0], tgt[1], tgt[2], lam[0], n, P.lpart);
    cudaMemsetAsync(P.gpart, 0, (size_t)step_blocks * 3 * 8, st);
    int li = 0;  // lam[li] holds lambda_{n+1}
    for (int sg = nseg - 1; sg >= 0; --sg) {
      const int n0 = sg * K, len = std::min(n0 + K, nsteps) - n0;
      if (sg != nseg - 1) {  // recompute the segment, keeping its steps
        cudaMemcpyAsync(fw[0], ckpt + (size_t)sg * n1, nv, cudaMemcpyDeviceToDevice, st);
        file_state(fw[0]);
        for (int m = 0; m < len; ++m) step(fw[m % 2], fw[(m + 1) % 2], m, m + 1 < len);
      }
      for (int m = len - 1; m >= 0; --m) {
        AdjParams<T> A = adj_params<T>(a, n);
        const size_t at = (size_t)m * n1;
        A.xs = xs + at;
        A.lam = lam[li];
        A.lam_out = lam[li ^ 1];
        A.pair_n = pair_n + at;
        A.pair_list = pair_list + at * (size_t)a->cap;
        A.gpart = P.gpart;
        // (the first after the memset is a plain launch)
        launch_serial(st, sg != nseg - 1 || m != len - 1, k_adj_backward<T>, dim3(step_blocks),
                      dim3(kTile), 0, A);
        li ^= 1;
      }
    }
    k_adj_unpack<T><<<blocks, kTile, 0, st>>>(lam[li], (T*)P.out_dx0[0], (T*)P.out_dx0[1],
                                              (T*)P.out_dx0[2], n);
  }
  cudaError_t e = cudaStreamEndCapture(st, &g);
  if (e != cudaSuccess) {
    P.release();
    return afail(a, CBM_ERR_CUDA, "adjoint graph capture failed: %s", cudaGetErrorString(e));
  }
  e = cudaGraphInstantiate(&P.graph, g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) {
    P.graph = nullptr;
    P.release();
    return afail(a, CBM_ERR_CUDA, "adjoint graph instantiate failed: %s", cudaGetErrorString(e));
  }
  return CBM_OK;
}

template <typename T>
int run(cbm_adjoint* a, const void* const* x0h, int n, int nsteps, int K, const void* const* tgth,
        double* loss, double* dtheta, void* const* dx0h, void* const* xTh, bool backward) {
  const size_t nb = (size_t)n * sizeof(T);
  if (backward && K > nsteps) K = std::max(nsteps, 1);  // one segment either way
  Plan& P = a->plan[backward ? 1 : 0];
  if (P.n != n || P.nsteps != nsteps || (backward && P.K != K) || !P.graph) {
    int rc = make_plan<T>(a, P, n, nsteps, backward ? K : 1, backward);
    if (rc) return rc;
  }
  cudaStream_t st = a->stream;
  for (int d = 0; d < 3; ++d) {
    if (nb) ACUDA(a, cudaMemcpyAsync(P.in_x[d], x0h[d], nb, cudaMemcpyHostToDevice, st));
    if (backward && nb) ACUDA(a, cudaMemcpyAsync(P.in_tgt[d], tgth[d], nb, cudaMemcpyHostToDevice, st));
  }
  ACUDA(a, cudaGraphLaunch(P.graph, st));
  if (xTh)
    for (int d = 0; d < 3; ++d)
      if (xTh[d] && nb) ACUDA(a, cudaMemcpyAsync(xTh[d], P.out_xT[d], nb, cudaMemcpyDeviceToHost, st));
  std::vector<double> gp, lp;
  if (backward) {
    gp.resize((size_t)P.step_blocks * 3);
    lp.resize((size_t)P.blocks);
    ACUDA(a, cudaMemcpyAsync(gp.data(), P.gpart, gp.size() * 8, cudaMemcpyDeviceToHost, st));
    ACUDA(a, cudaMemcpyAsync(lp.data(), P.lpart, lp.size() * 8, cudaMemcpyDeviceToHost, st));
    if (dx0h)
      for (int d = 0; d < 3; ++d)
        if (dx0h[d] && nb) ACUDA(a, cudaMemcpyAsync(dx0h[d], P.out_dx0[d], nb, cudaMemcpyDeviceToHost, st));
  }
  Counters hc;
  ACUDA(a, cudaMemcpyAsync(&hc, a->ctr, sizeof hc, cudaMemcpyDeviceToHost, st));
  ACUDA(a, cudaStreamSynchronize(st));
  if (hc.err) {
    int zero = 0;
    ACUDA(a, cudaMemcpy(&a->ctr->err, &zero, sizeof zero, cudaMemcpyHostToDevice));
    if (hc.err & kErrTimeout) return afail(a, CBM_ERR_TIMEOUT, "a bounded device-side wait gave up");
    if (hc.err & kErrNeighborOverflow)
      return afail(a, CBM_ERR_NEIGHBOR_OVERFLOW,
                   "an agent had more than %d interacting partners in one step", a->cap);
  }
  if (backward) {
    double l = 0.0, g[3] = {0.0, 0.0, 0.0};
    for (int b = 0; b < P.blocks; ++b) l += lp[(size_t)b];  // fixed order: deterministic
    for (int b = 0; b < P.step_blocks; ++b)
      for (int m = 0; m < 3; ++m) g[m] += gp[(size_t)b * 3 + m];
    if (loss) *loss = n > 0 ? l / (3.0 * (double)n) : 0.0;
    if (dtheta)
      for (int m = 0; m < 3; ++m) dtheta[m] = g[m];
  }
  return CBM_OK;
}

}  // namespace

extern "C" {

const char* cbm_adjoint_last_error(const cbm_adjoint* a) {
  return a ? a->err.c_str() : g_adj_error.c_str();
}

int cbm_adjoint_create(cbm_adjoint** out, const cbm_config* cfg) {
  if (!out || !cfg) return afail(nullptr, CBM_ERR_ARG, "null argument");
  *out = nullptr;
  const cbm_config& k = *cfg;
  if (k.dims != 3 || k.integrator != CBM_INT_EULER || k.force_mode != CBM_FORCE_DIRECT ||
      k.att_form != CBM_ATT_FROM_REP || k.neighbors != CBM_NEIGH_CELL_LINKED ||
      k.walls != CBM_WALLS_NONE || k.fate != CBM_FATE_NONE || k.medium || k.growth ||
      k.drift_linear != 0)
    return afail(nullptr, CBM_ERR_ARG,
                 "the adjoint covers the 3D soft-sphere Euler ODE with CellLinked neighbors "
                 "(no walls, fate, growth, medium or drift)");
  if (!(k.dt > 0) || !(k.cell_edge >= std::max(k.r_rep, k.r_att)) || !(k.r_att >= k.r_rep))
    return afail(nullptr, CBM_ERR_ARG, "need dt > 0, r_att >= r_rep and cell_edge >= r_att");
  if (k.n_max < 0 || k.n_max >= (1ll << 28)) return afail(nullptr, CBM_ERR_ARG, "n_max out of range");
  cbm_adjoint* a = new cbm_adjoint;
  a->cfg = k;
  a->ts = k.precision == CBM_F64 ? 8 : 4;
  a->n_max = (int)k.n_max;
  cudaGetDevice(&a->device);
  if (cudaStreamCreateWithFlags(&a->stream, cudaStreamNonBlocking) != cudaSuccess) {
    delete a;
    return afail(nullptr, CBM_ERR_CUDA, "cudaStreamCreate failed (is a CUDA device present?)");
  }
  long long nc = 1;
  for (int d = 0; d < 3; ++d) {
    a->nc[d] = (int)std::ceil((k.box_hi[d] - k.box_lo[d]) / k.cell_edge + 2.0);  // neighbors.jl:605
    nc *= a->nc[d];
  }
  if (nc >= (1ll << 28)) {
    cudaStreamDestroy(a->stream);
    delete a;
    return afail(nullptr, CBM_ERR_ARG, "cell grid too large");
  }
  a->n_cells = (int)nc;
  a->n_tiles = (a->n_cells + kScanTile - 1) / kScanTile;
  a->cap = std::max(k.n_max_neighbors, 64);
  if (a->ts == 8)
    cudaFuncSetAttribute(k_adj_step<double>, cudaFuncAttributePreferredSharedMemoryCarveout, 72);
  else
    cudaFuncSetAttribute(k_adj_step<float>, cudaFuncAttributePreferredSharedMemoryCarveout, 72);
  const size_t n = (size_t)std::max(a->n_max, 1);
  bool ok = true;
  auto get = [&](size_t bytes) -> void* {
    void* p = nullptr;
    if (!ok || cudaMalloc(&p, bytes ? bytes : 16) != cudaSuccess) {
      ok = false;
      return nullptr;
    }
    a->allocs.push_back(p);
    return p;
  };
  a->cell_count = (int*)get((size_t)a->n_cells * 4);
  a->scan_state = (unsigned long long*)get((size_t)a->n_tiles * 8);
  a->agent_cell = (int*)get(n * 4);
  a->agent_rank = (int*)get(n * 4);
  a->cell_tmp = (int*)get(n * 4);
  a->cell_of_slot = (int*)get(n * 4);
  a->ctr = (Counters*)get(sizeof(Counters));
  if (!ok) {
    for (void* p : a->allocs) cudaFree(p);
    cudaStreamDestroy(a->stream);
    delete a;
    return afail(nullptr, CBM_ERR_NOMEM, "device allocation failed");
  }
  cudaMemsetAsync(a->cell_count, 0, (size_t)a->n_cells * 4, a->stream);
  cudaMemsetAsync(a->scan_state, 0, (size_t)a->n_tiles * 8, a->stream);
  cudaMemsetAsync(a->ctr, 0, sizeof(Counters), a->stream);
  cudaStreamSynchronize(a->stream);
  *out = a;
  return CBM_OK;
}

void cbm_adjoint_destroy(cbm_adjoint* a) {
  if (!a) return;
  cudaSetDevice(a->device);
  cudaStreamSynchronize(a->stream);
  for (Plan& P : a->plan) P.release();
  for (void* p : a->allocs) cudaFree(p);
  cudaStreamDestroy(a->stream);
  delete a;
}

int cbm_adjoint_run(cbm_adjoint* a, int64_t n, const void* const* x0, int32_t nsteps,
                    int32_t checkpoint_every, const void* const* target, double* loss,
                    double* dtheta, void* const* dx0, void* const* xT) {
  if (!a || !x0 || !target || nsteps < 0 || checkpoint_every < 1) return afail(a, CBM_ERR_ARG, "bad argument");
  if (n < 0 || n > a->n_max) return afail(a, CBM_ERR_ARG, "n exceeds n_max");
  cudaSetDevice(a->device);
  if (a->ts == 8)
    return run<double>(a, x0, (int)n, nsteps, checkpoint_every, target, loss, dtheta, dx0, xT, true);
  return run<float>(a, x0, (int)n, nsteps, checkpoint_every, target, loss, dtheta, dx0, xT, true);
}

int cbm_adjoint_forward(cbm_adjoint* a, int64_t n, const void* const* x0, int32_t nsteps,
                        void* const* xT) {
  if (!a || !x0 || nsteps < 0) return afail(a, CBM_ERR_ARG, "bad argument");
  if (n < 0 || n > a->n_max) return afail(a, CBM_ERR_ARG, "n exceeds n_max");
  cudaSetDevice(a->device);
  if (a->ts == 8)
    return run<double>(a, x0, (int)n, nsteps, 1, nullptr, nullptr, nullptr, nullptr, xT, false);
  return run<float>(a, x0, (int)n, nsteps, 1, nullptr, nullptr, nullptr, nullptr, xT, false);
}

void* cbm_adjoint_stream(cbm_adjoint* a) { return a ? (void*)a->stream : nullptr; }

}  // extern "C"
