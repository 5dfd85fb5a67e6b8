// cbm_small.cuh — small CellLinked communities stepped by one launch.
//
// A community of a few thousand agents (the 2D aggregation of 4096 agents)
// costs far less than the launches of its step graph: the graph's seven
// kernels each wait for the previous one to drain.  Here one launch of a
// single thread-block cluster (up to 16 blocks of 1024 threads, scheduled
// together on one GPC) runs all the steps of a cbm_step call.  Its blocks
// meet at three hardware cluster barriers a step (barrier.cluster with
// release / acquire), between the phases:
//
//   DE     agentStepDE! of every slot over the grid of the committed
//          positions (the rule's wall reflection computed on the fly), four
//          lanes an agent, the same sums in the same order as k_agent_de,
//          into the working set B; then the histogram of the new cells
//   scan   update!'s counters; every block scans the cell counts
//          into shared memory (the cell grid of these communities fits one
//          block), block 0 stores the offsets, and agent indices are
//          scattered by (cell, arrival)
//   place  the stable placement B -> A by (cell, agent index) of
//          k_sort_place, and the counts are cleared for the next step
//
// The state after the launch is the one the step graphs leave.  Every block
// takes every barrier (the loops are uniform), so no wait depends on a
// condition that could fail to arrive.
#pragma once
#include "cbm_kernels.cuh"

namespace cbm {

// Threads a block: four lanes an agent over the sixteen blocks, so that a
// community of fewer than 4096 agents has fewer warps a scheduler instead of
// fewer blocks (700 agents: 19.2 us a step as three blocks of 1024 threads,
// 15.7 as eleven of 256).
constexpr int kSmallMaxThreads = 1024, kSmallMinThreads = 256;
constexpr int kSmallMaxBlocks = 16;     // blocks of the cluster (16 needs the non-portable size)
// Communities stepped by one launch (fate-free CellLinked).  The step graph
// takes much the same time whatever their size (27 us in 2D, 44 in 3D in
// Float64; 24 and 38 in Float32), the cluster's sixteen SMs take theirs in
// proportion once their lanes are all in use: Float64 19 and 37 us at 4096
// agents, 28 and 53 at 5500; Float32 20 and 36 at 5500, 28 and 53 at 9000.
template <typename T>
constexpr int kSmallMaxAgents = sizeof(T) == 8 ? 4096 : 6144;
constexpr int kSmallMaxCells = 8192;    // cell grids a block scans in shared memory

// Barrier of the cluster's blocks: every thread arrives with release and
// waits with acquire, so the global writes before it are visible after it.
__device__ __forceinline__ void cluster_barrier() {
  asm volatile(
      "barrier.cluster.arrive.release;\n\t"
      "barrier.cluster.wait.acquire;" ::: "memory");
}

// Exclusive scan of counts[0, n) by one block into out[0, n]; out[n] = total.
__device__ __forceinline__ void block_scan_counts(const int* counts, int n, int* out,
                                                  int* warp_sums) {
  const int nth = (int)blockDim.x;
  const int per = (n + nth - 1) / nth;
  const int c0 = min(n, (int)threadIdx.x * per), c1 = min(n, c0 + per);
  int local = 0;
  for (int c = c0; c < c1; ++c) {
    const int v = counts[c];
    out[c] = v;
    local += v;
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int x = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(kFull, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[w] = x;
  __syncthreads();
  if (w == 0) {
    int v = lane < nth / 32 ? warp_sums[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(kFull, v, o);
      if (lane >= o) v += y;
    }
    if (lane < nth / 32) warp_sums[lane] = v;
  }
  __syncthreads();
  int run = (w > 0 ? warp_sums[w - 1] : 0) + x - local;
  for (int c = c0; c < c1; ++c) {
    const int v = out[c];
    out[c] = run;
    run += v;
  }
  if ((int)threadIdx.x == nth - 1) out[n] = warp_sums[nth / 32 - 1];
  __syncthreads();
}

// agentStepDE! of slot s for CellLinked, by the kSmallLanes lanes of a group
// (lane gl of the group takes candidates gl, gl + kSmallLanes, ... of the
// three rows of cells of a plane, one sequence): the candidates of the 3^D
// cells in the reference's order, the pair terms of each chunk added in
// candidate order through the group's shuffles, so the sums are those of
// k_agent_de (skipping cells with no partner, as its pruning does, changes no
// sum, nor does adding the zero of a candidate beyond the cutoff).  A chunk
// is one serial chain of position load, root, quotient and ordered sums: the
// next chunk's positions are loaded before it, and root and quotient take the
// branch-free forms.  With reflecting walls the rule's reflected positions
// are computed from the committed ones, here for xi and every candidate.
// `start`: the grid's offsets, in shared memory.  The group's first lane
// integrates.
constexpr int kSmallLanes = 4;

template <typename T, int D>
__device__ __forceinline__ void small_de(const Params<T>& P, const PairLine<T>& line,
                                         const int* start, int s, T* x_new) {
  constexpr int L = kSmallLanes;
  const int lane = threadIdx.x & 31, gl = lane & (L - 1);
  const unsigned gmask = ((1u << L) - 1u) << (lane & ~(L - 1));
  const bool reflect = P.walls == CBM_WALLS_REFLECT;
  auto pos = [&](int q, T* x) {
    to3<T>(P.PA[q], x);
    if (reflect) {
#pragma unroll
      for (int d = 0; d < D; ++d) {
        if (x[d] < P.box_lo[d]) x[d] = (T)2 * P.box_lo[d] - x[d];
        else if (x[d] > P.box_hi[d]) x[d] = (T)2 * P.box_hi[d] - x[d];
      }
    }
  };
  T xi[3] = {(T)0, (T)0, (T)0};
  pos(s, xi);
  T acc[3] = {(T)0, (T)0, (T)0};
  int q3[3] = {0, 0, 0};
  cell_coords<D>(P.n_cells_d, cell_of_pos<T, D>(P, xi), q3);
  const int nx = P.n_cells_d[0];
  const int x0 = q3[0] > 0 ? q3[0] - 1 : 0, x1 = q3[0] < nx - 1 ? q3[0] + 1 : nx - 1;
  constexpr int ny_rows = D > 1 ? 3 : 1, nz_rows = D > 2 ? 3 : 1;
  for (int dz = 0; dz < nz_rows; ++dz) {
    const int pz = D > 2 ? q3[2] + dz - 1 : 0;
    if (D > 2 && (pz < 0 || pz >= P.n_cells_d[2])) continue;
    // candidate k of the plane: slot off[r] + k of the row r it falls in
    int off[3] = {0, 0, 0}, end[3] = {0, 0, 0}, total = 0;
#pragma unroll
    for (int r = 0; r < ny_rows; ++r) {
      const int py = D > 1 ? q3[1] + r - 1 : 0;
      if (D == 1 || (py >= 0 && py < P.n_cells_d[1])) {
        const int row = nx * (py + P.n_cells_d[1] * pz);
        const int s0 = start[row + x0];
        off[r] = s0 - total;
        total += start[row + x1 + 1] - s0;
      }
      end[r] = total;
    }
    auto slot = [&](int k) {
      return k + (D == 1 || k < end[0] ? off[0] : (k < end[1] ? off[1] : off[2]));
    };
    int qn = gl < total ? slot(gl) : s;
    T xn[3] = {(T)0, (T)0, (T)0};
    pos(qn, xn);
    for (int base = 0; base < total; base += L) {
      const int q = qn;
      const T xj[3] = {xn[0], xn[1], xn[2]};
      if (base + L < total) {
        qn = base + L + gl < total ? slot(base + L + gl) : s;
        pos(qn, xn);
      }
      T e[3];
      const T s2 = pair_diff<T, D>(xi, xj, e);
      T sc = (T)0;
      if (q != s) {
        T inv = (T)0;
        const bool mid = line.mid && s2 > (T)1e-12 && s2 < (T)1e12 && mid_root(s2);
        const T d = mid ? sqrt_mid(s2, &inv) : sqrt(s2);
        const bool rep = d < -line.nrrep;
        const T F = (rep ? line.krep : line.katt) * ((rep ? line.rrep : line.abase) - d);
        const T f = mid ? div_mid(F, d, inv) : F / d;
        sc = d < -line.nreach ? f : (T)0;
      }
      T t[3];
#pragma unroll
      for (int d = 0; d < D; ++d) t[d] = sc != (T)0 ? sc * e[d] : (T)0;
      // the chunk's terms, added in candidate order by every lane of the group
#pragma unroll
      for (int u = 0; u < L; ++u)
#pragma unroll
        for (int d = 0; d < D; ++d) acc[d] = acc[d] + __shfl_sync(gmask, t[d], u, L);
    }
  }
  if (gl == 0) finish_agent<T, D>(P, s, xi, acc, x_new);
}

// nsteps steps; P0 has the parity of the first step, P1 the other one.  The
// counts of the histogram are complete after the first barrier.  The
// counters' commit is made by the cluster's last thread in the placement
// phase (no thread reads those counters before the next step) so that it
// stays off the scan's path.
template <typename T, int D>
__global__ void __launch_bounds__(kSmallMaxThreads) k_small_steps(Params<T> P0, Params<T> P1,
                                                               int nsteps, int n_cells) {
  extern __shared__ int s_start[];  // n_cells + 1 offsets of the grid being built
  __shared__ int warp_sums[kSmallMaxThreads / 32];
  const int bth = (int)blockDim.x;
  const int tid = (int)blockIdx.x * bth + (int)threadIdx.x;
  const int nth = (int)gridDim.x * bth;
  const PairLine<T> line = make_pair_line<T>(P0.cut2, P0.k_rep, P0.r_rep, P0.k_att, P0.r_att,
                                             P0.att_form == CBM_ATT_FROM_REP);
  // every block keeps the offsets of the grid in use
  for (int c = threadIdx.x; c <= n_cells; c += bth) s_start[c] = P0.cell_start[c];
  __syncthreads();
  for (int t = 0; t < nsteps; ++t) {
    const Params<T>& P = (t & 1) ? P1 : P0;
    Counters* C = P.ctr;
    const int p = P.parity;
    const int N = (int)C->N[p];
    // DE, kSmallLanes lanes an agent; the histogram of the new cells follows
    // in the same phase (the agent's own written position is all it reads).
    // Slots are dealt to the blocks in turn (slot s to block s mod blocks),
    // so every block holds agents from all over the community and the dense
    // clumps do not all fall to the same block.
    const int groups = bth / kSmallLanes;
    for (int s = (int)(threadIdx.x / kSmallLanes) * (int)gridDim.x + (int)blockIdx.x; s < N;
         s += groups * (int)gridDim.x) {
      T x[3];
      small_de<T, D>(P, line, s_start, s, x);
      if ((threadIdx.x & (kSmallLanes - 1)) == 0) {  // k_sort_hist
        const int c = cell_of_pos<T, D>(P, x);
        P.s_cell[s] = c;
        P.s_rank[s] = atomicAdd(P.cell_count + c, 1);
      }
    }
    cluster_barrier();
    block_scan_counts(P.cell_count, n_cells, s_start, warp_sums);
    if (blockIdx.x == 0)
      for (int c = threadIdx.x; c <= n_cells; c += bth) P.cell_start[c] = s_start[c];
    for (int s = tid; s < N; s += nth) P.s_key[s_start[P.s_cell[s]] + P.s_rank[s]] = P.IB[s];
    cluster_barrier();
    for (int s = tid; s < N; s += nth) {  // stable placement by agent index (k_sort_place)
      const int c = P.s_cell[s];
      const int key = P.IB[s];
      const typename V4T<T>::type x = P.PB[s];
      const T v = P.VB[s];
      const int s0 = s_start[c], s1 = s_start[c + 1];
      int r = 0;
      for (int q = s0; q < s1; q += 4) {  // four keys in flight
        int k4[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) k4[u] = q + u < s1 ? P.s_key[q + u] : key;
#pragma unroll
        for (int u = 0; u < 4; ++u) r += k4[u] < key;
      }
      const int ns = s0 + r;
      P.PA[ns] = x;
      P.VA[ns] = v;
      P.IA[ns] = key;
      P.inv[key] = ns;
      P.cell_of_slot[ns] = c;
    }
    for (int c = tid; c < n_cells; c += nth) P.cell_count[c] = 0;
    if (tid == nth - 1) {  // update!'s counters, as commit_counters (no births or deaths here)
      C->slots = C->N[p];
      C->N[p ^ 1] = C->N[p];
      C->n_add = 0;
      C->n_remove = 0;
      C->t[p ^ 1] = C->t[p] + P.dt_time;
      C->step[p ^ 1] = C->step[p] + 1;
      C->flag[p ^ 1] = 0;
      C->resort = 1;
      C->events = 0;
      C->list_written = 0;
      C->list_valid = 0;  // the grid was rebuilt (computeNeighbors!)
    }
    cluster_barrier();
  }
}

}  // namespace cbm
