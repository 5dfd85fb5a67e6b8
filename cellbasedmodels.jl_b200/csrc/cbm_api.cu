// cbm_api.cu — host side of the C ABI declared in include/cbm_b200.h.
//
// A context owns every device buffer of one Community (capacity n_max) and
// one CUDA stream.  Its committed agent state lives in cell-sorted slots (set
// A) and each step writes set B (see cbm_kernels.cuh); a full step of each
// counter parity is captured once as a CUDA graph and replayed.
#include <cuda_runtime.h>

#include <cmath>
#include <cstddef>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/cbm_b200.h"
#include "cbm_kernels.cuh"
#include "cbm_small.cuh"
#include "cbm_stencil_vec.cuh"
#include "cbm_tile.cuh"
#include <utility>

using namespace cbm;

// Steps of one chained step graph, replayed by cbm_step calls of at least
// this many steps when there is a medium: inside the chain the field's
// kernels and the agents' kernels run as two pipelines that wait for each
// other only where they share a buffer.  Even, so that a chain leaves the
// parity as it found it.
constexpr int kChainSteps = 8;
static_assert(kChainSteps % 2 == 0, "a chain must keep the parity");

// The exchange in agent order takes lists (k_medium_links, k_medium_apply)
// when the field has at least this many nodes per (agent, stencil node), else
// the gather over the field's patches (k_secrete_rows).
constexpr unsigned long long kListNodes = 4;

struct cbm_ctx {
  cbm_config cfg{};
  int device = 0;
  cudaStream_t stream = nullptr;
  // with a medium: the agents' pipeline of a step, forked from and joined to
  // `stream`, which keeps the field's, and the events between the two
  cudaStream_t side = nullptr;
  cudaEvent_t fork_ev = nullptr, join_ev = nullptr, links_ev = nullptr, field_ev = nullptr,
              de_ev = nullptr, update_ev = nullptr;
  size_t tsize = 4;
  std::string err;
  std::vector<void*> allocs;

  // slot-ordered state
  void* PA = nullptr;
  void* PB = nullptr;
  void* VA = nullptr;
  void* VB = nullptr;
  void* FA = nullptr;
  void* FB = nullptr;
  int* IA = nullptr;
  int* IB = nullptr;
  void* U = nullptr;
  void* POLD = nullptr;
  int* inv = nullptr;
  int* cell_of_slot = nullptr;
  // index-ordered constants and staging
  void* G = nullptr;
  long long* ID = nullptr;
  long long* PAR = nullptr;
  void* hx[3] = {};
  void* hv = nullptr;
  void* hf[3] = {};
  // fate
  unsigned char* fate = nullptr;
  int* holes = nullptr;
  unsigned long long* fate_state = nullptr;  // per tile of the fused rule / births kernel
  // sort and grid
  int* s_cell = nullptr;
  int* s_rank = nullptr;
  int* s_key = nullptr;
  int* cell_count = nullptr;
  int* cell_start = nullptr;
  unsigned long long* scan_state = nullptr;
  // Verlet
  int* nbr_n = nullptr;
  int* nbr_list = nullptr;
  // medium
  void* c[2] = {};
  void* grad[2][3] = {};
  int* gather_box = nullptr;  // cell-box tables of the exchange's gather (k_gather_box)
  // exchange by lists: buckets' first entries, entries, Float64 weights, and
  // room to sort the entries of crowded nodes
  unsigned* link_head = nullptr;
  unsigned link_buckets = 0;
  uint4* link = nullptr;
  void* link_w = nullptr;
  unsigned long long* link_sort = nullptr;
  Counters* ctr = nullptr;
  Counters* h_ctr = nullptr;   // pinned staging of the counters an upload writes
  int* scratch_int = nullptr;  // n_max ints for inspection calls
  void* ext_noise = nullptr;   // EM increments of cbm_step_noise (n_max * dims reals, lazy)
  bool ext_noise_on = false;   // the step being enqueued reads ext_noise

  int n_blocks = 0;
  int n_sm = 148;             // multiprocessors of the device (grid of the compaction)
  int de_blocks = 1;          // persistent grid of the force kernel
  int split = -1;             // preferred percentage of shared memory of the step's kernels
  int tile_blocks = 0;        // resident blocks of k_agent_de_tile (0: not used)
  bool sparse = false;        // the walks that the tiles could take are made by threads
  void* pair_list = nullptr;  // partner lists of the walks by threads
  void* pos32 = nullptr;      // Float64 3D cell walks: positions rounded to Float32
  void* pos_rows = nullptr;   // Float32 3D cell walks: positions as rows x | y | z
  int rows_stride = 0;
  void* stage[3] = {nullptr, nullptr, nullptr};  // Heun / RK4: h, running sum, derivative
  int n_cells = 1;
  int n_cells_d[3] = {1, 1, 1};
  int n_scan_tiles = 1;
  int n_nodes = 0;
  bool grid_exposed = false;  // CellLinked / CLVD: the reference has a cell grid
  bool has_list = false;      // CLVD / VerletDisplacement

  // host-side bookkeeping
  bool loaded = false;
  int parity = 0;
  bool rule_done = false, de_done = false, mrule_done = false, mde_done = false;
  cudaGraphExec_t graph[2] = {nullptr, nullptr};   // step graphs of each parity
  cudaGraphExec_t tgraph[2] = {nullptr, nullptr};  // the same with kernel timing events
  cudaGraphExec_t chain[2] = {nullptr, nullptr};   // kChainSteps steps from each parity
  // small fate-free communities: all steps of a call in one cluster launch
  long long n_loaded = 0;         // N of the last upload (fixed without births and deaths)

  // per-kernel event timing: of eager steps (cbm_profile_step, `marks`) and,
  // when graph timing is on, inside the step graph of each parity
  // (`gmarks[p]`, re-recorded by every replay)
  bool prof = false;
  struct Mark {
    const char* name;
    cudaEvent_t ev[2];
  };
  std::vector<Mark> marks;
  size_t mark_used = 0;
  bool graph_timing = false;
  std::vector<Mark> gmarks[2];
  size_t gmark_used[2] = {0, 0};
  std::vector<Mark>* prof_set = nullptr;  // the set being recorded
  size_t* prof_used = nullptr;
};

extern "C" int cbm_sync(cbm_ctx* c);

namespace {

std::string g_create_error;

int fail(cbm_ctx* ctx, int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  if (ctx) ctx->err = buf;
  else g_create_error = buf;
  return code;
}

#define CUDA_TRY(ctx, call)                                                                \
  do {                                                                                     \
    cudaError_t e_ = (call);                                                               \
    if (e_ != cudaSuccess)                                                                 \
      return fail(ctx, CBM_ERR_CUDA, "%s failed: %s", #call, cudaGetErrorString(e_));      \
  } while (0)

int grid_blocks(long long n) { return n > 0 ? (int)((n + kTile - 1) / kTile) : 1; }

// device address of the counter block's re-sort flag
const int* resort_flag(const cbm_ctx* c) {
  return (const int*)((const char*)c->ctr + offsetof(Counters, resort));
}

// Brackets one kernel launch with events when profiling an eager step.
struct Prof {
  cbm_ctx* c;
  cbm_ctx::Mark* m = nullptr;
  Prof(cbm_ctx* ctx, const char* name) : c(ctx) {
    if (!c->prof) return;
    std::vector<cbm_ctx::Mark>& set = c->prof_set ? *c->prof_set : c->marks;
    size_t& used = c->prof_used ? *c->prof_used : c->mark_used;
    if (used == set.size()) {
      cbm_ctx::Mark mk{name, {nullptr, nullptr}};
      cudaEventCreate(&mk.ev[0]);
      cudaEventCreate(&mk.ev[1]);
      set.push_back(mk);
    }
    m = &set[used++];
    m->name = name;
    record(m->ev[0]);
  }
  ~Prof() {
    if (m) record(m->ev[1]);
  }
  // inside a stream capture an event record becomes a graph node only with
  // the external flag (a plain record there just orders the capture)
  void record(cudaEvent_t e) {
    if (c->prof_set) cudaEventRecordWithFlags(e, c->stream, cudaEventRecordExternal);
    else cudaEventRecord(e, c->stream);
  }
};
#define PROF(name) Prof prof_scope_(c, name)

// Launch on the context's stream with programmatic stream serialization,
// where the kernel before it on the stream is a kernel (no event between):
// the launch follows that kernel's completion without the full gap between
// launches, and the kernel's pdl_wait() orders its memory accesses after
// it.  A plain launch while kernels are timed (the event records sit
// between).
//
// Beside a 3D medium every kernel asks for the same split of an SM between
// shared memory and L1: the two pipelines run at once, and an SM takes no
// block of a kernel with another split until it is idle.  Left to themselves
// the vector stencils prefer L1 and the force kernels and the scan shared
// memory, and each waited for the other's blocks to leave.  The tiled walk's
// split suits them; beside a walk by threads it is what three of its blocks
// need (164 KB; 3e5 agents on 160^3 nodes, Float64, 745 us a step, with the
// tiles' 132 KB and two blocks 776).  Us a step before / so / with stencils
// that staged planes in shared memory, which had no such conflict:
//   no neighbors, uptake and chemotaxis by atomics, Float32
//     1e4 agents, 100^3 nodes 45 / 26 / 32;  4e4, 160^3 77 / 57 / 63
//   CellLinked, the same exchange in order, Float64
//     4479 agents, 72^3 44 / 36 / 38;  10616, 96^3 51 / 40 / 44
//   CellLinked, Float32, 2e5 agents, 256^3 180 / 182 / 246
constexpr int kThreadCarveout = 72;
template <typename... KP, typename... A>
void launch_pdl(cbm_ctx* c, bool pdl, void (*kern)(KP...), dim3 grid, dim3 block, size_t smem,
                A&&... args) {
  launch_split(c->stream, c->split, pdl && !c->prof, kern, grid, block, smem,
               std::forward<A>(args)...);
}
template <typename... KP, typename... A>
void launch(cbm_ctx* c, void (*kern)(KP...), unsigned grid, unsigned block, A&&... args) {
  launch_pdl(c, false, kern, dim3(grid), dim3(block), 0, std::forward<A>(args)...);
}

// r^2 (1 + 1e-5) rounded up to T: a squared distance at or above it has a
// correctly rounded sqrt >= (T)r, so the exact `d < r` test can be skipped
template <typename T>
T bound2(double r) {
  if (!(r > 0)) return (T)0;
  double v = r * r * (1.0 + 1e-5);
  T t = (T)v;
  return (double)t < v ? std::nextafter(t, (T)INFINITY) : t;
}

// r^2 (1 - 1e-5) rounded down to T: a squared distance below it has a
// correctly rounded sqrt < (T)r
template <typename T>
T bound2_lo(double r) {
  if (!(r > 0)) return (T)0;
  double v = r * r * (1.0 - 1e-5);
  T t = (T)v;
  return (double)t > v ? std::nextafter(t, (T)0) : t;
}

// 1 / v when v > 0 is a power of two whose reciprocal is representable
// (exactly), else 0.
template <typename T>
T exact_reciprocal(T v) {
  if (!(v > (T)0) || !std::isfinite(v)) return (T)0;
  int e = 0;
  if (std::frexp(v, &e) != (T)0.5) return (T)0;
  const T r = std::ldexp((T)1, 1 - e);
  return (r > (T)0 && std::isfinite(r) && r * v == (T)1) ? r : (T)0;
}

double cutoff(const cbm_config& k) { return k.r_rep > k.r_att ? k.r_rep : k.r_att; }

template <typename T>
Params<T> params(const cbm_ctx* c, int parity) {
  using V4 = typename V4T<T>::type;
  Params<T> P;
  memset(&P, 0, sizeof P);
  const cbm_config& k = c->cfg;
  const int p = parity, q = parity ^ 1;
  P.PA = (V4*)c->PA;
  P.PB = (V4*)c->PB;
  P.VA = (T*)c->VA;
  P.VB = (T*)c->VB;
  P.FA = (V4*)c->FA;
  P.FB = (V4*)c->FB;
  P.IA = c->IA;
  P.IB = c->IB;
  P.U = (V4*)c->U;
  P.stage_h = (V4*)c->stage[0];
  P.stage_s = (V4*)c->stage[1];
  P.stage_k = (V4*)c->stage[2];
  P.POLD = (V4*)c->POLD;
  P.inv = c->inv;
  P.cell_of_slot = c->cell_of_slot;
  P.G = (T*)c->G;
  P.ID = c->ID;
  P.PAR = c->PAR;
  for (int d = 0; d < 3; ++d) {
    P.hx[d] = (T*)c->hx[d];
    P.hf[d] = (T*)c->hf[d];
    P.grad_cur[d] = (T*)c->grad[p][d];
    P.grad_nxt[d] = (T*)c->grad[q][d];
  }
  P.hv = (T*)c->hv;
  P.fate = c->fate;
  P.holes = c->holes;
  P.fate_state = c->fate_state;
  P.noise = c->ext_noise_on ? (const T*)c->ext_noise : nullptr;
  P.s_cell = c->s_cell;
  P.s_rank = c->s_rank;
  P.s_key = c->s_key;
  P.cell_count = c->cell_count;
  P.cell_start = c->cell_start;
  P.gather_box = c->gather_box;
  P.link_head = c->link_head;
  P.link_mask = c->link_buckets ? c->link_buckets - 1u : 0u;
  P.link_shift = 35;
  for (unsigned b = c->link_buckets; b > 1; b >>= 1) --P.link_shift;
  P.link = c->link;
  P.link_w = (T*)c->link_w;
  P.link_sort = c->link_sort;
  P.scan_state = c->scan_state;
  P.nbr_n = c->nbr_n;
  P.nbr_list = c->nbr_list;
  P.tiled = c->tile_blocks > 0 && !c->sparse;
  P.pair_list = P.tiled ? nullptr : (int4*)c->pair_list;
  P.pair_cap4 = kPairCap4;
  P.PA32 = P.tiled ? nullptr : (float4*)c->pos32;
  P.PS = P.tiled ? nullptr : (float*)c->pos_rows;
  P.ps_stride = c->rows_stride;
  P.c_cur = (T*)c->c[p];
  P.c_nxt = (T*)c->c[q];
  P.ctr = c->ctr;
  P.n_max = (int)k.n_max;
  P.n_blocks = c->n_blocks;
  P.n_cells = c->n_cells;
  for (int d = 0; d < 3; ++d) {
    P.n_cells_d[d] = c->n_cells_d[d];
    P.n_medium[d] = d < k.dims && k.medium ? k.n_medium[d] : 1;
    P.box_lo[d] = (T)k.box_lo[d];
    P.box_hi[d] = (T)k.box_hi[d];
    // dx = (hi - lo) / NMedium in Float64 (communityStructure.jl:274)
    P.dx_m[d] = d < k.dims && k.medium ? (T)((k.box_hi[d] - k.box_lo[d]) / (double)k.n_medium[d])
                                       : (T)1;
  }
  P.exact_scale = k.medium ? 1 : 0;
  for (int d = 0; d < 3; ++d) {
    P.inv_dx[d] = P.inv_dx2[d] = P.inv_2dx[d] = (T)0;
    if (d < k.dims && k.medium) {
      P.inv_dx[d] = exact_reciprocal<T>(P.dx_m[d]);
      P.inv_dx2[d] = exact_reciprocal<T>(P.dx_m[d] * P.dx_m[d]);
      P.inv_2dx[d] = exact_reciprocal<T>((T)2 * P.dx_m[d]);
      if (P.inv_dx2[d] == (T)0 || P.inv_2dx[d] == (T)0) P.exact_scale = 0;
    }
  }
  P.n_scan_tiles = c->n_scan_tiles;
  P.n_nodes = c->n_nodes;
  P.max_nbrs = k.n_max_neighbors;
  P.parity = parity;
  P.neighbors = k.neighbors;
  P.integrator = k.integrator;
  P.force_mode = k.force_mode;
  P.att_form = k.att_form;
  P.walls = k.walls;
  P.fate_rule = k.fate;
  P.growth = k.growth;
  P.medium = k.medium;
  P.medium_sampling = k.medium_sampling;
  P.dt = (T)k.dt;
  P.dt_time = k.dt;
  P.sqrt_dt = std::sqrt((T)k.dt);
  P.sigma = (T)k.sigma;
  P.edge = (T)(k.neighbors == CBM_NEIGH_VERLET_DISPLACEMENT ? k.skin : k.cell_edge);
  P.skin = (T)k.skin;
  P.rebuild_thr = k.rebuild_threshold > 0 ? (T)k.rebuild_threshold : (T)k.skin / (T)2;
  P.k_rep = (T)k.k_rep;
  P.r_rep = (T)k.r_rep;
  P.k_att = (T)k.k_att;
  P.r_att = (T)k.r_att;
  P.cut2 = bound2<T>(k.r_rep > k.r_att ? k.r_rep : k.r_att);
  P.skin2 = bound2<T>(k.skin);
  P.skin2_lo = bound2_lo<T>(k.skin);
  P.tile_scale = (T)tile_scale(cutoff(k), k.cell_edge);
  P.tile_cut = tile_cut(cutoff(k), k.cell_edge);
  P.force_in_list = (T)(k.r_rep > k.r_att ? k.r_rep : k.r_att) <= (T)k.skin ? 1 : 0;
  P.cut_reach = (T)((k.r_rep > k.r_att ? k.r_rep : k.r_att) * (1.0 + 1e-4));
  P.skin_reach = (T)(k.skin * (1.0 + 1e-4));
  P.wall_force = (T)k.wall_force;
  P.wall_range = (T)k.wall_range;
  P.drift_linear = (T)k.drift_linear;
  P.v_div = (T)k.v_div;
  P.div_sep = (T)k.div_sep;
  P.p_death = (T)k.p_death;
  P.diff_D = (T)k.diff_D;
  P.decay = (T)k.decay;
  P.secretion_amt = (T)k.secretion * (T)k.dt;
  P.uptake_amt = (T)k.uptake * (T)k.dt;
  P.chemotaxis = (T)k.chemotaxis;
  P.seed = k.seed;
  P.community = k.community;
  return P;
}

// agents add to the medium (secretion) or take from it (uptake)
bool exchanges(const cbm_config& k) { return k.medium && (k.secretion != 0 || k.uptake != 0); }
bool orders_exchange(const cbm_config& k) {
  return exchanges(k) && k.medium_sampling == CBM_MEDIUM_BILINEAR &&
         k.neighbors == CBM_NEIGH_CELL_LINKED;
}
// the exchange in agent order by lists: an entry per agent and stencil node
unsigned long long list_entries(const cbm_config& k) {
  return (unsigned long long)(k.n_max > 0 ? k.n_max : 1) << k.dims;
}
bool exchange_by_lists(const cbm_config& k) {
  if (!orders_exchange(k)) return false;
  unsigned long long nodes = 1;
  for (int d = 0; d < k.dims; ++d) nodes *= (unsigned long long)k.n_medium[d];
  return list_entries(k) * kListNodes <= nodes;
}
bool rule_needed(const cbm_config& k) {
  return k.walls == CBM_WALLS_REFLECT || (exchanges(k) && !orders_exchange(k)) ||
         k.fate != CBM_FATE_NONE;
}
// the atomic rule path reads the committed field from a snapshot
bool needs_snapshot(const cbm_config& k) { return k.uptake != 0 && exchanges(k) && !orders_exchange(k); }

// The 3D cell walks that k_agent_de_tile takes: of the committed positions
// (no wall reflection and no stage positions, whose agents may lie outside
// the cells they are filed in), with CellLinked, or with CLVD in the steps
// with births or deaths, where the tile's filter serves (tile_scale).
bool walk_by_tile(const cbm_config& k) {
  return k.dims == 3 && k.walls != CBM_WALLS_REFLECT &&
         (k.integrator == CBM_INT_EULER || k.integrator == CBM_INT_EM) &&
         tile_scale(cutoff(k), k.cell_edge) != 0.0 &&
         (k.neighbors == CBM_NEIGH_CELL_LINKED ||
          (k.neighbors == CBM_NEIGH_CLVD && k.fate != CBM_FATE_NONE));
}
// the 3D force-only walks left to k_agent_de, one thread an agent
bool walk_by_thread(const cbm_config& k) {
  return k.dims == 3 && !walk_by_tile(k) &&
         (k.neighbors == CBM_NEIGH_CELL_LINKED ||
          (k.neighbors == CBM_NEIGH_CLVD && k.fate != CBM_FATE_NONE));
}

// Sparse communities of many agents are walked by threads: their tiles find
// too few partners to share, and each lane's own candidates then wait on
// gathers with thirteen warps an SM, in Float64 on 32-byte positions that
// saturate L1 (82 %).  The walk by threads has full occupancy and, in Float64,
// the filter's Float32 copy.  The measure is the mean number of agents in an
// agent's cell, itself included.  Step in us, by tiles / by threads, cells of
// 1.1 cutoffs:
//   Float64, 1e6 agents     2.4 a cell 465 / 314   6.4: 506 / 412   8.2: 526 / 469   10: 564 / 574
//            1e5            1.2: 50 / 45   3.2: 91 / 55   8.2: 92 / 73   10: 94 / 85   15: 114 / 110
//            5e4            1.2: 33 / 40   3.2: 55 / 49   8.2: 65 / 62   10: 62 / 69
//   Float32, 1e6            1.7: 201 / 230   3.2: 291 / 275   4.6: 364 / 295   8.2: 361 / 358   10: 385 / 435
//            1e5            1.7: 42 / 46   3.2: 58 / 54   4.6: 63 / 55   8.2: 69 / 64   12: 78 / 77
//            5e4            3.2: 40 / 48   4.6: 46 / 50
constexpr long long kSparseFrom = 65536;
bool may_be_sparse(const cbm_config& k) { return walk_by_tile(k) && k.n_max >= kSparseFrom; }
// `now`: a margin keeps a community at the line where it is.
bool is_sparse(const cbm_config& k, double per_cell, long long n, bool now) {
  const double lo = k.precision == CBM_F64 ? 0.0 : 2.5, hi = k.precision == CBM_F64 ? 9.5 : 8.2;
  const double m = now ? 1.1 : 1.0;
  return n >= kSparseFrom && per_cell * m > lo && per_cell < hi * m;
}

// blocks of the 2D shared-memory stencils (one tile per block)
dim3 stencil_grid(const cbm_ctx* c) {
  const int nx = c->cfg.n_medium[0] > 0 ? c->cfg.n_medium[0] : 1;
  const int ny = c->cfg.n_medium[1] > 0 ? c->cfg.n_medium[1] : 1;
  return dim3((unsigned)((nx + kStX - 1) / kStX), (unsigned)((ny + kStTileY - 1) / kStTileY));
}

// z planes per block of the tiled 3D stencils: about twelve blocks for every
// SM (each block works through its planes one after another, so more and
// shorter runs keep more planes in flight), and runs of at least 8 planes
// (each run also reads the two planes that close it)
int stencil_z_run(const cbm_ctx* c) {
  const dim3 g = stencil_grid(c);
  const long long xy = (long long)g.x * g.y;
  const int nz = c->cfg.n_medium[2] > 0 ? c->cfg.n_medium[2] : 1;
  const long long want = 12LL * (c->n_sm > 0 ? c->n_sm : 148);
  long long runs = (want + xy - 1) / xy;
  if (runs < 1) runs = 1;
  long long z_run = (nz + runs - 1) / runs;
  if (z_run < 8) z_run = 8;
  return (int)z_run;
}
// The vector stencils: rows of whole 16-byte vectors.
bool vec_medium(const cbm_ctx* c) {
  return ((size_t)c->cfg.n_medium[0] * c->tsize) % 16 == 0;
}
int vec_blocks(const cbm_ctx* c) {
  return grid_blocks((long long)c->cfg.n_medium[0] * (long long)c->tsize / 16 * c->cfg.n_medium[1]);
}
// planes a run: about sixteen blocks of 256 for every SM (two to three waves;
// eight an SM measured 36 and 61 us for the two at 256^3 Float32, sixteen 34
// and 49), and runs of at least 4 planes
int vec_z_run(const cbm_ctx* c) {
  const int nz = c->cfg.n_medium[2] > 0 ? c->cfg.n_medium[2] : 1;
  const int xy = vec_blocks(c);
  const long long want = 16LL * (c->n_sm > 0 ? c->n_sm : 148);
  const long long runs = (want + xy - 1) / xy;
  const int z_run = (int)((nz + runs - 1) / runs);
  return z_run < 4 ? 4 : z_run;
}
dim3 vec_grid(const cbm_ctx* c) {
  const int nz = c->cfg.n_medium[2] > 0 ? c->cfg.n_medium[2] : 1, zr = vec_z_run(c);
  return dim3((unsigned)vec_blocks(c), (unsigned)((nz + zr - 1) / zr));
}
dim3 stencil_grid_3d(const cbm_ctx* c) {
  dim3 g = stencil_grid(c);
  const int nz = c->cfg.n_medium[2] > 0 ? c->cfg.n_medium[2] : 1;
  const int zr = stencil_z_run(c);
  g.z = (unsigned)((nz + zr - 1) / zr);
  return g;
}

// ---- stage launches (enqueue only) -----------------------------------------
template <typename T, int D>
void enqueue_medium_rule(cbm_ctx* c, const Params<T>& P) {
  if (c->cfg.medium && c->cfg.chemotaxis != 0) {
    PROF("k_medium_grad");
    if (D == 2)
      k_medium_grad_2d<T><<<stencil_grid(c), dim3(kStX, kStY), 0, c->stream>>>(P);
    else if (D == 3)
      if (vec_medium(c))
        launch_pdl(c, false, k_medium_grad_3d_vec<T>, vec_grid(c), dim3(kTile), 0, P, vec_z_run(c));
      else
        k_medium_grad_3d<T><<<stencil_grid_3d(c), dim3(kStX, kStY), 0, c->stream>>>(P, stencil_z_run(c));
    else
      k_medium_grad<T, D><<<grid_blocks(c->n_nodes), kTile, 0, c->stream>>>(P);
  }
}

// the heads and the count that follows them, to a length that clears by
// whole vectors
size_t link_head_bytes(const cbm_ctx* c) { return ((size_t)c->link_buckets + 64) * 4; }

template <typename T, int D>
void enqueue_links(cbm_ctx* c, const Params<T>& P) {
  cudaMemsetAsync(c->link_head, 0xff, link_head_bytes(c), c->stream);
  PROF("k_medium_links");
  launch(c, k_medium_links<T, D>, grid_blocks(c->cfg.n_max << D), kTile, P);
}
template <typename T, int D>
void enqueue_apply(cbm_ctx* c, const Params<T>& P) {
  PROF("k_medium_apply");
  launch(c, k_medium_apply<T, D>, grid_blocks(c->cfg.n_max << D), kTile, P);
}
template <typename T, int D>
void enqueue_gather(cbm_ctx* c, const Params<T>& P) {
  PROF("k_secrete_rows");
  const int nm[3] = {c->cfg.n_medium[0], D > 1 ? c->cfg.n_medium[1] : 1,
                     D > 2 ? c->cfg.n_medium[2] : 1};
  const int py = (nm[1] + GatherPatch<D>::kY - 1) / GatherPatch<D>::kY;
  constexpr int W = GatherPatch<D>::kWarps;
  const dim3 grid((unsigned)((nm[0] + 31) / 32), (unsigned)((py + W - 1) / W),
                  (unsigned)((nm[2] + GatherPatch<D>::kZ - 1) / GatherPatch<D>::kZ));
  launch_pdl(c, false, k_secrete_rows<T, D>, grid, dim3(W * 32), 0, P);
}
// walls, births and deaths, and the exchange that atomics add
template <typename T, int D>
void enqueue_rule(cbm_ctx* c, const Params<T>& P) {
  const cbm_config& k = c->cfg;
  if (needs_snapshot(k)) {
    PROF("k_medium_snapshot");
    launch(c, k_medium_snapshot<T>, grid_blocks(c->n_nodes), kTile, P);
  }
  if (!rule_needed(k)) return;
  if (k.fate != CBM_FATE_NONE) {
    PROF("k_agent_fate");
    launch(c, k_agent_fate<T, D>, fate_tiles(c->cfg.n_max), kTile, P);
  } else {
    PROF("k_agent_rule");
    launch(c, k_agent_rule<T, D>, c->n_blocks, kTile, P);
  }
}
template <typename T, int D>
void enqueue_agent_rule(cbm_ctx* c, const Params<T>& P) {
  if (c->link_buckets) {
    enqueue_links<T, D>(c, P);
    enqueue_apply<T, D>(c, P);
  } else if (orders_exchange(c->cfg)) {
    enqueue_gather<T, D>(c, P);
  }
  enqueue_rule<T, D>(c, P);
}

template <typename T, int D>
void enqueue_agent_de(cbm_ctx* c, const Params<T>& P) {
  const unsigned grid = kPartnerLists<D> ? c->de_blocks : c->n_blocks;
  const int integ = c->cfg.integrator;
  if (P.PA32) {
    PROF("k_pos32");
    launch(c, k_pos32<T>, c->n_blocks, kTile, P);
  }
  if (P.PS) {
    PROF("k_pos_rows");
    launch(c, k_pos_rows<T>, c->n_blocks, kTile, P);
  }
  if (integ != CBM_INT_HEUN && integ != CBM_INT_RK4 && integ != CBM_INT_EULER_HEUN) {
    if constexpr (D == 3) {
      if (P.tiled) {
        PROF("k_agent_de_tile");
        k_agent_de_tile<T><<<c->tile_blocks, 32, 0, c->stream>>>(P);
      }
      if (P.tiled && c->cfg.neighbors == CBM_NEIGH_CELL_LINKED) return;
    }
    PROF("k_agent_de");
    launch_pdl(c, P.tiled != 0, k_agent_de<T, D>, dim3(grid), dim3(kTile), 0, P);
    return;
  }
  // multi-stage: f at u, then at each stage's positions (own cell from the
  // position, no face pruning), each followed by its combination
  auto stage = [&](bool at_h, int op) {
    Params<T> Q = P;
    Q.KOUT = Q.stage_k;
    if (at_h) {
      Q.XS = Q.stage_h;
      Q.no_prune = 1;
    }
    {
      PROF("k_agent_de");
      launch(c, k_agent_de<T, D>, grid, kTile, Q);
    }
    PROF("k_stage_combine");
    launch(c, k_stage_combine<T, D>, c->n_blocks, kTile, P, op);
  };
  if (integ == CBM_INT_HEUN) {
    stage(false, kHeunStage);
    stage(true, kHeunFinal);
  } else if (integ == CBM_INT_EULER_HEUN) {
    stage(false, kEhStage);
    stage(true, kEhFinal);
  } else {
    stage(false, kRk1);
    stage(true, kRk2);
    stage(true, kRk3);
    stage(true, kRkFinal);
  }
}

template <typename T, int D>
void enqueue_medium_de(cbm_ctx* c, const Params<T>& P) {
  if (c->cfg.medium) {
    PROF("k_medium_de");
    if (D == 2)
      k_medium_de_2d<T><<<stencil_grid(c), dim3(kStX, kStY), 0, c->stream>>>(P);
    else if (D == 3)
      if (vec_medium(c))
        launch_pdl(c, false, k_medium_de_3d_vec<T>, vec_grid(c), dim3(kTile), 0, P, vec_z_run(c));
      else
        k_medium_de_3d<T><<<stencil_grid_3d(c), dim3(kStX, kStY), 0, c->stream>>>(P, stencil_z_run(c));
    else
      k_medium_de<T, D><<<grid_blocks(c->n_nodes), kTile, 0, c->stream>>>(P);
  }
}

// In a step whose agents are neither born nor die and whose grid is rebuilt
// every time, the force kernel files each agent in its new cell: the re-sort
// then begins with the scan, which commits the counters.
bool hist_in_de(const cbm_config& k) {
  static_assert(kHistInDE<2> && !kHistInDE<3>, "as below");
  return k.dims < 3 && k.neighbors == CBM_NEIGH_CELL_LINKED && k.fate == CBM_FATE_NONE &&
         (k.integrator == CBM_INT_EULER || k.integrator == CBM_INT_EM);
}

// update!: compaction, then B -> A (copy, or re-sort = grid rebuild) with the
// commit of the counters.  The kernels follow one another on the stream;
// `after_kernel`: so does the first of them.
template <typename T, int D>
void enqueue_update(cbm_ctx* c, const Params<T>& P, bool after_kernel = false) {
  if (c->cfg.fate != CBM_FATE_NONE) {
    PROF("k_compact");
    launch(c, k_compact<T, D>, c->n_sm, kCompactThreads, P);
    after_kernel = true;
  }
  ScanArgs A{c->cell_count, c->cell_start, c->scan_state, c->n_cells, c->n_scan_tiles, c->ctr,
             resort_flag(c)};
  A.crowd = may_be_sparse(c->cfg);
  if (P.hist_in_de) {
    A.due = nullptr;
    A.commit = 1;
    A.parity = P.parity;
    A.dt = P.dt_time;
  } else {
    PROF("k_sort_hist");
    launch_pdl(c, after_kernel, k_sort_hist<T, D>, dim3(c->n_blocks), dim3(kTile), 0, P, 1);
    after_kernel = true;
  }
  {
    PROF("k_scan_cells");
    launch_pdl(c, after_kernel, k_scan_cells, dim3(c->n_scan_tiles), dim3(kTile), 0, A);
  }
  {
    PROF("k_sort_scatter");
    launch_pdl(c, true, k_sort_scatter<T>, dim3(c->n_blocks), dim3(kTile), 0, P);
  }
  PROF("k_sort_place");
  launch_pdl(c, true, k_sort_place<T, D>, dim3(c->n_blocks), dim3(kTile), 0, P);
}

// computeNeighbors! after update!: the grid was rebuilt by the re-sort; a
// VerletDisplacement list is rebuilt eagerly (ascending agent order), a CLVD
// list is walked from the grid by the next DE stage.  Q has the parity of the
// step that starts.
template <typename T, int D>
void enqueue_neighbors(cbm_ctx* c, const Params<T>& Q) {
  if (c->cfg.neighbors == CBM_NEIGH_VERLET_DISPLACEMENT) {
    PROF("k_verlet_list");
    launch(c, k_verlet_list<T, D>, c->n_blocks, kTile, Q, 1);
  }
}

int kernels_per_step(const cbm_ctx* c) {
  const cbm_config& k = c->cfg;
  int n = 0;
  if (k.medium && k.chemotaxis != 0) n += 1;
  if (needs_snapshot(k)) n += 1;
  if (orders_exchange(k)) n += c->link_buckets ? 2 : 1;  // the lists and their sums, or the gather
  if (rule_needed(k)) n += 1;           // rule (with births and deaths when fate is on)
  if (k.fate != CBM_FATE_NONE) n += 1;  // compaction
  n += 1;                               // agent DE
  const bool tiled = c->tile_blocks && !c->sparse;
  if (tiled && k.neighbors == CBM_NEIGH_CLVD) n += 1;  // its steps on the list
  if (c->pos32 && !tiled) n += 1;       // its Float32 positions (Float64 walks by threads)
  if (c->pos_rows && !tiled) n += 1;    // its position rows (Float32 walks by threads)
  if (k.medium) n += 1;
  n += hist_in_de(k) ? 3 : 4;           // sort hist, scan, scatter, place
  if (k.neighbors == CBM_NEIGH_VERLET_DISPLACEMENT) n += 1;
  return n;
}

// One step from parity `parity`; `first` and `last` of the steps enqueued
// together.  With a medium they form two pipelines.  The field's, on `stream`:
// gradient G, exchange A, FTCS F; the agents', on `side`: lists L of the
// exchange, rule, force kernel D, update and neighbors U.  They wait for each
// other where they share a buffer:
//   A by lists needs L, and the next L (which writes the lists again) needs A;
//   A by the gather, or as a rule that adds with atomics, reads the agents: it
//   needs the U before it and the U after needs it; the rule is also needed by
//   D, which reads the reflected positions;
//   D reads the gradient of the step before, the next G writes that buffer.
// U and F, which share nothing, overlap, and in a chain the two pipelines run
// ahead of each other.  Per-kernel timing keeps the series order.  A failed
// event call is seen like a failed launch (by the capture, or by
// cudaGetLastError after an eager step).
template <typename T, int D>
void enqueue_full_step(cbm_ctx* c, int parity, bool first = true, bool last = true) {
  Params<T> P = params<T>(c, parity);
  const cbm_config& k = c->cfg;
  P.hist_in_de = hist_in_de(k) ? 1 : 0;
  if (!c->side || c->prof) {
    enqueue_medium_rule<T, D>(c, P);
    enqueue_agent_rule<T, D>(c, P);
    enqueue_agent_de<T, D>(c, P);
    enqueue_medium_de<T, D>(c, P);
    enqueue_update<T, D>(c, P, true);
    enqueue_neighbors<T, D>(c, params<T>(c, parity ^ 1));
    return;
  }
  cudaStream_t field = c->stream, agents = c->side;
  const bool lists = c->link_buckets != 0;
  const bool gather = orders_exchange(k) && !lists;
  const bool atomics = exchanges(k) && !orders_exchange(k);
  const bool grad = k.chemotaxis != 0;
  if (first) {
    cudaEventRecord(c->fork_ev, field);
    cudaStreamWaitEvent(agents, c->fork_ev, 0);
  }
  c->stream = agents;
  // the last step's A (the lists) and G (the gradient D reads)
  if (!first && (lists || grad)) cudaStreamWaitEvent(agents, c->field_ev, 0);
  if (lists) {
    enqueue_links<T, D>(c, P);
    cudaEventRecord(c->links_ev, agents);
  }
  c->stream = field;
  if (grad) {
    if (!first) cudaStreamWaitEvent(field, c->de_ev, 0);
    enqueue_medium_rule<T, D>(c, P);
  }
  if (lists) {
    cudaStreamWaitEvent(field, c->links_ev, 0);
    enqueue_apply<T, D>(c, P);
  }
  if ((gather || atomics) && !first) cudaStreamWaitEvent(field, c->update_ev, 0);
  if (gather) enqueue_gather<T, D>(c, P);
  if (atomics) enqueue_rule<T, D>(c, P);
  cudaEventRecord(c->field_ev, field);
  enqueue_medium_de<T, D>(c, P);
  c->stream = agents;
  if (atomics) cudaStreamWaitEvent(agents, c->field_ev, 0);
  if (!atomics) enqueue_rule<T, D>(c, P);
  enqueue_agent_de<T, D>(c, P);
  cudaEventRecord(c->de_ev, agents);
  if (gather) cudaStreamWaitEvent(agents, c->field_ev, 0);
  enqueue_update<T, D>(c, P);
  enqueue_neighbors<T, D>(c, params<T>(c, parity ^ 1));
  cudaEventRecord(c->update_ev, agents);
  c->stream = field;
  if (last) {
    cudaEventRecord(c->join_ev, agents);
    cudaStreamWaitEvent(field, c->join_ev, 0);
  }
}

// dispatch on (precision, dims)
template <template <typename, int> class Fn, typename... A>
void dispatch(cbm_ctx* c, A... a) {
  if (c->cfg.precision == CBM_F64) {
    switch (c->cfg.dims) {
      case 1: Fn<double, 1>::run(c, a...); break;
      case 2: Fn<double, 2>::run(c, a...); break;
      default: Fn<double, 3>::run(c, a...); break;
    }
  } else {
    switch (c->cfg.dims) {
      case 1: Fn<float, 1>::run(c, a...); break;
      case 2: Fn<float, 2>::run(c, a...); break;
      default: Fn<float, 3>::run(c, a...); break;
    }
  }
}

// resident blocks of the force kernel per multiprocessor
template <typename T, int D>
struct DEOccupancy {
  static void run(cbm_ctx*, int* bps) {
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(bps, k_agent_de<T, D>, kTile, 0) !=
            cudaSuccess ||
        *bps < 1)
      *bps = 1;
  }
};

// resident one-warp blocks of the tiled force walk per multiprocessor
template <typename T, int D>
struct TileOccupancy {
  static void run(cbm_ctx*, int* bps) {
    cudaFuncSetAttribute(k_agent_de_tile<T>, cudaFuncAttributePreferredSharedMemoryCarveout,
                         kTileCarveout);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(bps, k_agent_de_tile<T>, 32, 0) !=
            cudaSuccess ||
        *bps < 1)
      *bps = 1;
  }
};

template <typename T, int D>
struct FullStep {
  static void run(cbm_ctx* c, int parity) { enqueue_full_step<T, D>(c, parity); }
};
// kChainSteps steps from parity p
template <typename T, int D>
struct ChainSteps {
  static void run(cbm_ctx* c, int parity) {
    for (int i = 0; i < kChainSteps; ++i)
      enqueue_full_step<T, D>(c, parity ^ (i & 1), i == 0, i + 1 == kChainSteps);
  }
};
template <typename T, int D>
struct StageRule {
  static void run(cbm_ctx* c) {
    Params<T> P = params<T>(c, c->parity);
    if (!c->mrule_done) enqueue_medium_rule<T, D>(c, P);
    enqueue_agent_rule<T, D>(c, P);
  }
};
template <typename T, int D>
struct StageDE {
  static void run(cbm_ctx* c) { enqueue_agent_de<T, D>(c, params<T>(c, c->parity)); }
};
template <typename T, int D>
struct StageMediumRule {
  static void run(cbm_ctx* c) { enqueue_medium_rule<T, D>(c, params<T>(c, c->parity)); }
};
template <typename T, int D>
struct StageMediumDE {
  static void run(cbm_ctx* c) { enqueue_medium_de<T, D>(c, params<T>(c, c->parity)); }
};
template <typename T, int D>
struct StageUpdate {
  static void run(cbm_ctx* c, int copy_agents, int use_u, int copy_c, int copy_grad) {
    Params<T> P = params<T>(c, c->parity);
    if (copy_agents) k_copy_ab<T, D><<<c->n_blocks, kTile, 0, c->stream>>>(P, use_u);
    if (c->cfg.medium && (copy_c || copy_grad))
      k_copy_medium<T, D><<<grid_blocks(c->n_nodes), kTile, 0, c->stream>>>(P, copy_c ? 0 : 1);
    enqueue_update<T, D>(c, P);
  }
};
template <typename T, int D>
struct StageNeighbors {
  static void run(cbm_ctx* c) { enqueue_neighbors<T, D>(c, params<T>(c, c->parity)); }
};
template <typename T, int D>
struct BuildList {  // the list of the current slots, on request
  static void run(cbm_ctx* c) {
    k_verlet_list<T, D><<<c->n_blocks, kTile, 0, c->stream>>>(params<T>(c, c->parity), 0);
  }
};
template <typename T, int D>
struct CountNeighbors {
  static void run(cbm_ctx* c, double radius, int* out) {
    k_count_neighbors<T, D><<<c->n_blocks, kTile, 0, c->stream>>>(params<T>(c, c->parity),
                                                                  (T)radius, out);
  }
};
template <typename T, int D>
struct Pack {
  static void run(cbm_ctx* c, int N) {
    k_pack_upload<T, D><<<grid_blocks(N), kTile, 0, c->stream>>>(params<T>(c, c->parity), N);
  }
};
template <typename T, int D>
struct Gather {
  static void run(cbm_ctx* c, int N, int which) {
    k_gather_download<T, D><<<grid_blocks(N), kTile, 0, c->stream>>>(params<T>(c, c->parity), N,
                                                                      which);
  }
};
template <typename T, int D>
struct FirstSort {  // the re-sort half of update!, for loadToPlatform!
  static void run(cbm_ctx* c) {
    Params<T> P = params<T>(c, c->parity);
    k_sort_hist<T, D><<<c->n_blocks, kTile, 0, c->stream>>>(P, 0);
    ScanArgs A{c->cell_count, c->cell_start, c->scan_state, c->n_cells, c->n_scan_tiles, c->ctr,
               resort_flag(c)};
    A.crowd = may_be_sparse(c->cfg);
    k_scan_cells<<<c->n_scan_tiles, kTile, 0, c->stream>>>(A);
    k_sort_scatter<T><<<c->n_blocks, kTile, 0, c->stream>>>(P);
    k_sort_place<T, D><<<c->n_blocks, kTile, 0, c->stream>>>(P);
    if (c->cfg.neighbors == CBM_NEIGH_VERLET_DISPLACEMENT)
      k_verlet_list<T, D><<<c->n_blocks, kTile, 0, c->stream>>>(P, 0);
  }
};

int check_launch(cbm_ctx* c) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(c, CBM_ERR_CUDA, "kernel launch failed: %s", cudaGetErrorString(e));
  return CBM_OK;
}

void* dalloc(cbm_ctx* c, size_t bytes, bool* ok) {
  if (!*ok) return nullptr;
  if (bytes == 0) bytes = 16;
  void* p = nullptr;
  if (cudaMalloc(&p, bytes) != cudaSuccess) {
    *ok = false;
    return nullptr;
  }
  c->allocs.push_back(p);
  return p;
}

// the nodes of a step with lists keep the priorities of the streams they were
// captured on
unsigned instantiate_flags(const cbm_ctx* c) {
  return c->link_buckets ? cudaGraphInstantiateFlagUseNodePriority : 0;
}

void drop_graphs(cbm_ctx* c) {
  for (int q = 0; q < 2; ++q)
    for (cudaGraphExec_t* g : {&c->graph[q], &c->tgraph[q], &c->chain[q]}) {
      if (*g) cudaGraphExecDestroy(*g);
      *g = nullptr;
    }
}

void free_all(cbm_ctx* c) {
  for (auto& m : c->marks) {
    cudaEventDestroy(m.ev[0]);
    cudaEventDestroy(m.ev[1]);
  }
  c->marks.clear();
  drop_graphs(c);
  for (int q = 0; q < 2; ++q) {
    for (auto& m : c->gmarks[q]) {
      cudaEventDestroy(m.ev[0]);
      cudaEventDestroy(m.ev[1]);
    }
    c->gmarks[q].clear();
  }
  for (void* p : c->allocs) cudaFree(p);
  if (c->h_ctr) cudaFreeHost(c->h_ctr);
  c->h_ctr = nullptr;
  c->allocs.clear();
  if (c->side) cudaStreamDestroy(c->side);
  c->side = nullptr;
  for (cudaEvent_t* e :
       {&c->fork_ev, &c->join_ev, &c->links_ev, &c->field_ev, &c->de_ev, &c->update_ev}) {
    if (*e) cudaEventDestroy(*e);
    *e = nullptr;
  }
  if (c->stream) cudaStreamDestroy(c->stream);
  c->stream = nullptr;
}

int flags_to_status(int err) {
  if (err & kErrAgentOverflow) return CBM_ERR_AGENT_OVERFLOW;
  if (err & kErrNeighborOverflow) return CBM_ERR_NEIGHBOR_OVERFLOW;
  if (err & kErrTimeout) return CBM_ERR_TIMEOUT;
  return CBM_OK;
}

// The counters after all that is enqueued: one copy to page-locked memory and
// one wait.  With them comes the choice of the walk for the steps to come (the
// sums are the same bits either way); steps being timed keep theirs.
int read_counters(cbm_ctx* c, Counters* h) {
  CUDA_TRY(c, cudaMemcpyAsync(c->h_ctr, c->ctr, sizeof(Counters), cudaMemcpyDeviceToHost, c->stream));
  CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  *h = *c->h_ctr;
  const long long n = h->N[c->parity];
  if (c->tile_blocks && c->pair_list && n > 0 && !c->graph_timing) {
    const bool sparse = is_sparse(c->cfg, (double)h->crowd / (double)n, n, c->sparse);
    if (sparse != c->sparse) drop_graphs(c);
    c->sparse = sparse;
  }
  return CBM_OK;
}

void reset_stage_flags(cbm_ctx* c) {
  c->rule_done = c->de_done = c->mrule_done = c->mde_done = false;
}

// CLVD builds its list lazily; inspection calls build it when missing
int ensure_list(cbm_ctx* c) {
  Counters hc;
  int rc = read_counters(c, &hc);
  if (rc) return rc;
  if (!hc.list_valid) {
    dispatch<BuildList>(c);
    rc = check_launch(c);
    if (rc) return rc;
    return cbm_sync(c);  // reports a row that exceeded n_max_neighbors
  }
  return CBM_OK;
}

}  // namespace

// ============================================================================
// C ABI
// ============================================================================
extern "C" {

const char* cbm_version(void) { return "cbm_b200 0.2.0 (sm_100a)"; }

const char* cbm_last_error(const cbm_ctx* ctx) {
  return ctx ? ctx->err.c_str() : g_create_error.c_str();
}

int cbm_create(cbm_ctx** out, const cbm_config* cfg) {
  if (!out || !cfg) return fail(nullptr, CBM_ERR_ARG, "null argument");
  *out = nullptr;
  const cbm_config& k = *cfg;
  if (k.dims < 1 || k.dims > 3) return fail(nullptr, CBM_ERR_ARG, "dims must be 1, 2 or 3");
  if (k.precision != CBM_F32 && k.precision != CBM_F64)
    return fail(nullptr, CBM_ERR_ARG, "precision must be CBM_F32 or CBM_F64");
  if (k.n_max < 0 || k.n_max >= (1ll << 30))
    return fail(nullptr, CBM_ERR_ARG, "n_max must be in [0, 2^30)");
  // the births/deaths scan packs two prefix counts of up to 2 n_max into 29 bits each
  if (k.fate != CBM_FATE_NONE && k.n_max >= (1ll << 28))
    return fail(nullptr, CBM_ERR_ARG, "with births and deaths n_max must be below 2^28");
  if (!(k.dt > 0)) return fail(nullptr, CBM_ERR_ARG, "dt must be positive");
  if (k.neighbors < CBM_NEIGH_NONE || k.neighbors > CBM_NEIGH_CLVD)
    return fail(nullptr, CBM_ERR_ARG, "unknown neighbor algorithm %d", k.neighbors);
  if (k.integrator < CBM_INT_EULER || k.integrator > CBM_INT_EULER_HEUN)
    return fail(nullptr, CBM_ERR_ARG, "unknown integrator %d", k.integrator);
  const bool multistage = k.integrator == CBM_INT_HEUN || k.integrator == CBM_INT_RK4 ||
                          k.integrator == CBM_INT_EULER_HEUN;
  if (multistage) {
    if (k.integrator != CBM_INT_EULER_HEUN && k.sigma != 0)
      return fail(nullptr, CBM_ERR_ARG, "Heun and RungeKutta4 integrate ODEs: sigma must be 0");
    if (k.force_mode == CBM_FORCE_LAGGED)
      return fail(nullptr, CBM_ERR_ARG, "multi-stage integrators need force_mode = CBM_FORCE_DIRECT");
    if (k.neighbors == CBM_NEIGH_CLVD)
      return fail(nullptr, CBM_ERR_ARG,
                  "multi-stage integrators need neighbors NONE, FULL, CELL_LINKED or "
                  "VERLET_DISPLACEMENT");
  }
  for (int d = 0; d < k.dims; ++d)
    if (!(k.box_hi[d] > k.box_lo[d])) return fail(nullptr, CBM_ERR_ARG, "empty simBox on axis %d", d);
  const bool cells = k.neighbors == CBM_NEIGH_CELL_LINKED || k.neighbors == CBM_NEIGH_CLVD;
  const bool list = k.neighbors == CBM_NEIGH_CLVD || k.neighbors == CBM_NEIGH_VERLET_DISPLACEMENT;
  if (cells && !(k.cell_edge > 0)) return fail(nullptr, CBM_ERR_ARG, "cell_edge must be positive");
  if (list && !(k.skin > 0)) return fail(nullptr, CBM_ERR_ARG, "skin must be positive");
  if (k.neighbors == CBM_NEIGH_CLVD && k.cell_edge < k.skin)
    return fail(nullptr, CBM_ERR_ARG, "CLVD needs cell_edge >= skin");
  if (list && (k.n_max_neighbors < 1 ||
               (k.neighbors == CBM_NEIGH_VERLET_DISPLACEMENT && k.n_max_neighbors > kVdSortMax)))
    return fail(nullptr, CBM_ERR_ARG, "n_max_neighbors must be in [1, %d]",
                k.neighbors == CBM_NEIGH_VERLET_DISPLACEMENT ? kVdSortMax : (1 << 20));
  if (k.medium) {
    for (int d = 0; d < k.dims; ++d)
      if (k.n_medium[d] < 1) return fail(nullptr, CBM_ERR_ARG, "n_medium[%d] must be >= 1", d);
  }
  if (!(k.uptake >= 0) || k.uptake > 1e300)
    return fail(nullptr, CBM_ERR_ARG, "uptake must be finite and >= 0");
  if (k.uptake != 0 && !k.medium) return fail(nullptr, CBM_ERR_ARG, "uptake needs a medium");

  cbm_ctx* c = new cbm_ctx;
  c->cfg = k;
  c->tsize = k.precision == CBM_F64 ? 8 : 4;
  cudaGetDevice(&c->device);
  cudaDeviceGetAttribute(&c->n_sm, cudaDevAttrMultiProcessorCount, c->device);
  cudaError_t se = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking);
  if (se != cudaSuccess) {
    int rc = fail(nullptr, CBM_ERR_CUDA, "cudaStreamCreate failed (is a CUDA device present?)");
    delete c;
    return rc;
  }
  if (k.medium) {
    // Where the exchange is by lists the agents' kernels, which nothing of the
    // field's delays for long, go first (2e5 agents on 256^3 nodes 180 us a
    // step without, 175 with); the gather is on the field's side, and waits
    // for it would then grow (2D, 2e5 agents on 1024^2: 54.7 without, 58.8).
    int least = 0, greatest = 0;
    se = cudaDeviceGetStreamPriorityRange(&least, &greatest);
    if (se == cudaSuccess)
      se = cudaStreamCreateWithPriority(&c->side, cudaStreamNonBlocking,
                                        exchange_by_lists(k) ? greatest : least);
    for (cudaEvent_t* e :
         {&c->fork_ev, &c->join_ev, &c->links_ev, &c->field_ev, &c->de_ev, &c->update_ev})
      if (se == cudaSuccess) se = cudaEventCreateWithFlags(e, cudaEventDisableTiming);
  }
  if (se != cudaSuccess) {
    int rc = fail(nullptr, CBM_ERR_CUDA, "creating the branch of the step graph failed");
    free_all(c);
    delete c;
    return rc;
  }
  const size_t n = (size_t)(k.n_max > 0 ? k.n_max : 1);
  const size_t S = c->tsize, S4 = 4 * c->tsize;
  c->n_blocks = grid_blocks((long long)n);
  c->grid_exposed = cells;
  c->has_list = list;
  // slots are sorted by cell for every algorithm; without a grid there is one cell
  if (cells || k.neighbors == CBM_NEIGH_VERLET_DISPLACEMENT) {
    double e = k.neighbors == CBM_NEIGH_VERLET_DISPLACEMENT ? k.skin : k.cell_edge;
    long long nc = 1;
    for (int d = 0; d < k.dims; ++d) {
      // nCells_ = ceil((hi - lo) / edge + 2), neighbors.jl:605 (Float64 on the host)
      double v = std::ceil((k.box_hi[d] - k.box_lo[d]) / e + 2.0);
      if (!(v >= 1 && v < 2.0e9)) {
        int rc = fail(nullptr, CBM_ERR_ARG, "cell grid too large on axis %d", d);
        free_all(c);
        delete c;
        return rc;
      }
      c->n_cells_d[d] = (int)v;
      nc *= (long long)v;
    }
    if (nc >= (1ll << 31) - 1) {
      int rc = fail(nullptr, CBM_ERR_ARG, "cell grid has too many cells (%lld)", nc);
      free_all(c);
      delete c;
      return rc;
    }
    c->n_cells = (int)nc;
  }
  c->n_scan_tiles = (c->n_cells + kScanTile - 1) / kScanTile;
  if (k.medium) {
    long long nn = 1;
    for (int d = 0; d < k.dims; ++d) nn *= k.n_medium[d];
    if (nn >= (1ll << 31)) {
      int rc = fail(nullptr, CBM_ERR_ARG, "medium grid too large");
      free_all(c);
      delete c;
      return rc;
    }
    c->n_nodes = (int)nn;
  }

  bool ok = true;
  c->PA = dalloc(c, n * S4, &ok);
  c->PB = dalloc(c, n * S4, &ok);
  c->VA = dalloc(c, n * S, &ok);
  c->VB = dalloc(c, n * S, &ok);
  c->FA = dalloc(c, n * S4, &ok);
  c->FB = dalloc(c, n * S4, &ok);
  c->IA = (int*)dalloc(c, n * 4, &ok);
  c->IB = (int*)dalloc(c, n * 4, &ok);
  if (k.walls == CBM_WALLS_REFLECT) c->U = dalloc(c, n * S4, &ok);
  if (k.integrator == CBM_INT_HEUN || k.integrator == CBM_INT_RK4 ||
      k.integrator == CBM_INT_EULER_HEUN)
    for (int q = 0; q < 3; ++q) c->stage[q] = dalloc(c, n * S4, &ok);
  if (list) c->POLD = dalloc(c, n * S4, &ok);
  c->inv = (int*)dalloc(c, n * 4, &ok);
  c->cell_of_slot = (int*)dalloc(c, n * 4, &ok);
  c->G = dalloc(c, n * S, &ok);
  c->ID = (long long*)dalloc(c, n * 8, &ok);
  c->PAR = (long long*)dalloc(c, n * 8, &ok);
  for (int d = 0; d < 3; ++d) {
    c->hx[d] = dalloc(c, n * S, &ok);
    c->hf[d] = dalloc(c, n * S, &ok);
  }
  c->hv = dalloc(c, n * S, &ok);
  c->fate = (unsigned char*)dalloc(c, n, &ok);
  c->holes = (int*)dalloc(c, n * 4, &ok);
  c->fate_state = (unsigned long long*)dalloc(c, (size_t)c->n_blocks * 8, &ok);
  c->s_cell = (int*)dalloc(c, n * 4, &ok);
  c->s_rank = (int*)dalloc(c, n * 4, &ok);
  c->s_key = (int*)dalloc(c, n * 4, &ok);
  c->cell_count = (int*)dalloc(c, (size_t)c->n_cells * 4, &ok);
  c->cell_start = (int*)dalloc(c, ((size_t)c->n_cells + 1) * 4, &ok);
  c->scan_state = (unsigned long long*)dalloc(c, (size_t)c->n_scan_tiles * 8, &ok);
  c->scratch_int = (int*)dalloc(c, n * 4, &ok);
  {
    // one partner-list region per resident block of the force kernel
    int bps = 1;
    dispatch<DEOccupancy>(c, &bps);
    const long long resident = (long long)c->n_sm * bps;
    c->de_blocks = (int)(resident < c->n_blocks ? resident : c->n_blocks);
    if (walk_by_tile(k)) {
      dispatch<TileOccupancy>(c, &bps);
      const long long tiles = (long long)(n + 31) / 32, warps = (long long)c->n_sm * bps;
      c->tile_blocks = (int)(warps < tiles ? warps : tiles);
    }
    const bool threads = walk_by_thread(k) || may_be_sparse(k);
    if (threads)
      c->pair_list = dalloc(c, (size_t)c->de_blocks * kTile * kPairCap4 * sizeof(int4), &ok);
    // the filter's copies of the committed positions (a walk of reflected
    // positions reads those)
    const bool copies = threads && k.walls != CBM_WALLS_REFLECT;
    if (copies && c->tsize == 8) c->pos32 = dalloc(c, n * sizeof(float4), &ok);
    if (copies && c->tsize == 4) {
      c->rows_stride = (int)((n + 3) & ~(size_t)3);  // rows start on 16 bytes
      c->pos_rows = dalloc(c, 3 * (size_t)c->rows_stride * sizeof(float), &ok);
    }
  }
  if (list) {
    c->nbr_n = (int*)dalloc(c, n * 4, &ok);
    c->nbr_list = (int*)dalloc(c, n * (size_t)k.n_max_neighbors * 4, &ok);
  }
  if (k.medium) {
    for (int q = 0; q < 2; ++q) {
      c->c[q] = dalloc(c, (size_t)c->n_nodes * S, &ok);
      for (int d = 0; d < 3; ++d) c->grad[q][d] = dalloc(c, (size_t)c->n_nodes * S, &ok);
    }
    if (k.dims == 3 && vec_medium(c)) c->split = walk_by_thread(k) ? kThreadCarveout : kTileCarveout;
    if (orders_exchange(k)) {
      size_t nb = 0;
      for (int d = 0; d < k.dims; ++d) nb += 2 * (size_t)k.n_medium[d];
      c->gather_box = (int*)dalloc(c, nb * 4, &ok);
    }
    if (exchange_by_lists(k)) {
      const unsigned long long ne = list_entries(k);
      c->link_buckets = 1024;
      while (c->link_buckets < ne) c->link_buckets *= 2;
      c->link_head = (unsigned*)dalloc(c, link_head_bytes(c), &ok);
      c->link = (uint4*)dalloc(c, ne * sizeof(uint4), &ok);
      if (S == 8) c->link_w = dalloc(c, ne * S, &ok);
      c->link_sort = (unsigned long long*)dalloc(c, ne * 8, &ok);
    }
  }
  c->ctr = (Counters*)dalloc(c, sizeof(Counters), &ok);
  if (ok && cudaMallocHost((void**)&c->h_ctr, sizeof(Counters)) != cudaSuccess) {
    c->h_ctr = nullptr;
    ok = false;
  }
  if (!ok) {
    int rc = fail(nullptr, CBM_ERR_NOMEM, "device allocation failed for n_max=%lld", (long long)k.n_max);
    free_all(c);
    delete c;
    return rc;
  }
  if (c->gather_box) {
    int nmax = 1;
    for (int d = 0; d < k.dims; ++d) nmax = k.n_medium[d] > nmax ? (int)k.n_medium[d] : nmax;
    const unsigned blocks = (unsigned)((nmax + 255) / 256);
    if (c->tsize == 8)
      k_gather_box<double><<<blocks, 256, 0, c->stream>>>(params<double>(c, 0), c->gather_box, k.dims);
    else
      k_gather_box<float><<<blocks, 256, 0, c->stream>>>(params<float>(c, 0), c->gather_box, k.dims);
  }
  cudaMemsetAsync(c->cell_count, 0, (size_t)c->n_cells * 4, c->stream);
  cudaMemsetAsync(c->scan_state, 0, (size_t)c->n_scan_tiles * 8, c->stream);
  cudaMemsetAsync(c->fate_state, 0, (size_t)c->n_blocks * 8, c->stream);
  cudaMemsetAsync(c->ctr, 0, sizeof(Counters), c->stream);
  if (cudaStreamSynchronize(c->stream) != cudaSuccess) {
    int rc = fail(nullptr, CBM_ERR_CUDA, "device initialisation failed");
    free_all(c);
    delete c;
    return rc;
  }
  *out = c;
  return CBM_OK;
}

void cbm_destroy(cbm_ctx* ctx) {
  if (!ctx) return;
  cudaSetDevice(ctx->device);
  cudaStreamSynchronize(ctx->stream);
  free_all(ctx);
  delete ctx;
}

// ids 1..N for an upload that gives none (Community numbers its agents from 1)
static __global__ void k_default_ids(long long* id, int n) {
  const int i = blockIdx.x * kTile + threadIdx.x;
  if (i < n) id[i] = (long long)i + 1;
}

// Ranges of words to clear: the absent fields of an upload and the rows beyond N.
struct ClearList {
  unsigned* at[12];
  long long words[12];
  int n;
};
static __global__ void __launch_bounds__(kTile) k_clear(ClearList L) {
  for (int k = 0; k < L.n; ++k)
    for (long long i = (long long)blockIdx.x * kTile + threadIdx.x; i < L.words[k];
         i += (long long)gridDim.x * kTile)
      L.at[k][i] = 0u;
}

// An upload's counters; the epochs go on from those they replace, so that
// stale tile states never match.
static __global__ void k_load_counters(Counters* C, Counters h) {
  h.scan_epoch = C->scan_epoch + 1u;
  h.fate_epoch = C->fate_epoch + 1u;
  *C = h;
}

int cbm_upload(cbm_ctx* c, const cbm_state_view* h) {
  if (!c || !h) return fail(c, CBM_ERR_ARG, "null argument");
  cudaSetDevice(c->device);
  const cbm_config& k = c->cfg;
  if (h->N < 0 || h->N > k.n_max)
    return fail(c, CBM_ERR_ARG, "N=%lld exceeds n_max=%lld", (long long)h->N, (long long)k.n_max);
  const size_t N = (size_t)h->N, S = c->tsize, nm = (size_t)k.n_max;
  for (int d = 0; d < k.dims; ++d)
    if (N && !h->pos[d]) return fail(c, CBM_ERR_ARG, "pos[%d] is NULL", d);
  if (k.growth && N && (!h->v || !h->g)) return fail(c, CBM_ERR_ARG, "growth needs v and g");
  cudaStream_t st = c->stream;
  // staging: index order; absent fields are zeros (loadToPlatform! pads with
  // zeros), and so is every field beyond N.  A field given by the caller is
  // copied into [0, N) and cleared beyond it only.
  // (one kernel clears all of them)
  ClearList clear{};
  auto stage = [&](void* dst, const void* src, size_t elem) -> cudaError_t {
    const size_t from = (src && N) ? N : 0;
    if (nm > from) {
      clear.at[clear.n] = (unsigned*)((char*)dst + from * elem);
      clear.words[clear.n++] = (long long)((nm - from) * (elem / 4));
    }
    return from ? cudaMemcpyAsync(dst, src, N * elem, cudaMemcpyHostToDevice, st) : cudaSuccess;
  };
  for (int d = 0; d < 3; ++d) {
    CUDA_TRY(c, stage(c->hx[d], d < k.dims ? h->pos[d] : nullptr, S));
    CUDA_TRY(c, stage(c->hf[d], d < k.dims ? h->f[d] : nullptr, S));
  }
  CUDA_TRY(c, stage(c->hv, h->v, S));
  CUDA_TRY(c, stage(c->G, h->g, S));
  CUDA_TRY(c, stage(c->PAR, h->parent, 8));
  // ids: the caller's (copied straight from its array), else 1..N; zero beyond N
  CUDA_TRY(c, stage(c->ID, h->id, 8));
  k_clear<<<2 * c->n_sm, kTile, 0, st>>>(clear);
  if (N && !h->id) k_default_ids<<<grid_blocks((long long)N), kTile, 0, st>>>(c->ID, (int)N);
  if (k.medium) {
    const size_t nb = (size_t)c->n_nodes * S;
    for (int q = 0; q < 2; ++q) {
      // over the bus once; the second copy is the device's own
      if (h->medium_c)
        CUDA_TRY(c, q == 0 ? cudaMemcpyAsync(c->c[0], h->medium_c, nb, cudaMemcpyHostToDevice, st)
                           : cudaMemcpyAsync(c->c[1], c->c[0], nb, cudaMemcpyDeviceToDevice, st));
      else CUDA_TRY(c, cudaMemsetAsync(c->c[q], 0, nb, st));
      for (int d = 0; d < 3; ++d) {
        if (d < k.dims && h->medium_grad[d])
          CUDA_TRY(c, q == 0 ? cudaMemcpyAsync(c->grad[0][d], h->medium_grad[d], nb,
                                               cudaMemcpyHostToDevice, st)
                             : cudaMemcpyAsync(c->grad[1][d], c->grad[0][d], nb,
                                               cudaMemcpyDeviceToDevice, st));
        else CUDA_TRY(c, cudaMemsetAsync(c->grad[q][d], 0, nb, st));
      }
    }
  }
  CUDA_TRY(c, cudaMemsetAsync(c->cell_count, 0, (size_t)c->n_cells * 4, st));
  Counters hc;
  memset(&hc, 0, sizeof hc);
  hc.N[0] = hc.N[1] = h->N;
  hc.step[0] = hc.step[1] = h->step;
  hc.t[0] = hc.t[1] = h->t;
  hc.id_max = h->id_max > 0 ? h->id_max : h->N;
  hc.slots = h->N;
  hc.resort = 1;  // flagRecomputeNeighbors_ = [1] and computeNeighbors! at load (communityStructure.jl:480,648)
  k_load_counters<<<1, 1, 0, st>>>(c->ctr, hc);
  c->parity = 0;
  reset_stage_flags(c);
  c->loaded = true;
  c->n_loaded = h->N;
  dispatch<Pack>(c, (int)N);
  dispatch<FirstSort>(c);
  int rc = check_launch(c);
  if (rc) return rc;
  return cbm_sync(c);
}

int cbm_download(cbm_ctx* c, cbm_state_view* h, int32_t which) {
  if (!c || !h) return fail(c, CBM_ERR_ARG, "null argument");
  if (!c->loaded) return fail(c, CBM_ERR_STATE, "community not uploaded");
  cudaSetDevice(c->device);
  Counters hc;
  int rc = read_counters(c, &hc);
  if (rc) return rc;
  const cbm_config& k = c->cfg;
  const int p = c->parity;
  const long long N = hc.N[p];
  if (h->capacity < N)
    return fail(c, CBM_ERR_ARG, "host capacity %lld < N=%lld", (long long)h->capacity, N);
  h->N = N;
  h->t = hc.t[p];
  h->step = hc.step[p];
  h->id_max = hc.id_max;
  const size_t S = c->tsize, nb = (size_t)N * S;
  const bool nw = which == CBM_VIEW_NEW;
  const int src = nw && c->de_done ? 1 : (nw && c->rule_done && c->U ? 2 : 0);
  if (N) {
    dispatch<Gather>(c, (int)N, src);
    rc = check_launch(c);
    if (rc) return rc;
  }
  // the copies follow the gather on the context's stream, one
  // synchronisation for all of them
  cudaStream_t st = c->stream;
  for (int d = 0; d < k.dims; ++d) {
    if (h->pos[d] && N) CUDA_TRY(c, cudaMemcpyAsync(h->pos[d], c->hx[d], nb, cudaMemcpyDeviceToHost, st));
    if (h->f[d] && N) CUDA_TRY(c, cudaMemcpyAsync(h->f[d], c->hf[d], nb, cudaMemcpyDeviceToHost, st));
  }
  if (h->v && N) CUDA_TRY(c, cudaMemcpyAsync(h->v, c->hv, nb, cudaMemcpyDeviceToHost, st));
  if (h->g && N) CUDA_TRY(c, cudaMemcpyAsync(h->g, c->G, nb, cudaMemcpyDeviceToHost, st));
  if (h->id && N) CUDA_TRY(c, cudaMemcpyAsync(h->id, c->ID, (size_t)N * 8, cudaMemcpyDeviceToHost, st));
  if (h->parent && N)
    CUDA_TRY(c, cudaMemcpyAsync(h->parent, c->PAR, (size_t)N * 8, cudaMemcpyDeviceToHost, st));
  if (k.medium) {
    const size_t mb = (size_t)c->n_nodes * S;
    const int qc = nw && c->mde_done ? p ^ 1 : p;
    const int qg = nw && c->mrule_done ? p ^ 1 : p;
    if (h->medium_c) CUDA_TRY(c, cudaMemcpyAsync(h->medium_c, c->c[qc], mb, cudaMemcpyDeviceToHost, st));
    for (int d = 0; d < k.dims; ++d)
      if (h->medium_grad[d])
        CUDA_TRY(c, cudaMemcpyAsync(h->medium_grad[d], c->grad[qg][d], mb, cudaMemcpyDeviceToHost, st));
  }
  CUDA_TRY(c, cudaStreamSynchronize(st));
  return CBM_OK;
}

int cbm_agent_step_rule(cbm_ctx* c) {
  if (!c) return CBM_ERR_ARG;
  if (!c->loaded) return fail(c, CBM_ERR_STATE, "community not uploaded");
  cudaSetDevice(c->device);
  dispatch<StageRule>(c);
  if (c->cfg.medium && c->cfg.chemotaxis != 0) c->mrule_done = true;
  c->rule_done = true;
  return check_launch(c);
}

int cbm_agent_step_de(cbm_ctx* c) {
  if (!c) return CBM_ERR_ARG;
  if (!c->loaded) return fail(c, CBM_ERR_STATE, "community not uploaded");
  cudaSetDevice(c->device);
  const cbm_config& k = c->cfg;
  if (!c->rule_done && k.walls == CBM_WALLS_REFLECT)
    CUDA_TRY(c, cudaMemcpyAsync(c->U, c->PA, (size_t)k.n_max * 4 * c->tsize,
                                cudaMemcpyDeviceToDevice, c->stream));
  dispatch<StageDE>(c);
  c->de_done = true;
  return check_launch(c);
}

int cbm_medium_step_rule(cbm_ctx* c) {
  if (!c) return CBM_ERR_ARG;
  if (!c->loaded) return fail(c, CBM_ERR_STATE, "community not uploaded");
  cudaSetDevice(c->device);
  if (!c->mrule_done) dispatch<StageMediumRule>(c);
  if (c->cfg.medium && c->cfg.chemotaxis != 0) c->mrule_done = true;
  return check_launch(c);
}

int cbm_medium_step_de(cbm_ctx* c) {
  if (!c) return CBM_ERR_ARG;
  if (!c->loaded) return fail(c, CBM_ERR_STATE, "community not uploaded");
  cudaSetDevice(c->device);
  dispatch<StageMediumDE>(c);
  if (c->cfg.medium) c->mde_done = true;
  return check_launch(c);
}

int cbm_update(cbm_ctx* c) {
  if (!c) return CBM_ERR_ARG;
  if (!c->loaded) return fail(c, CBM_ERR_STATE, "community not uploaded");
  cudaSetDevice(c->device);
  const cbm_config& k = c->cfg;
  int copy_agents = c->de_done ? 0 : 1;
  int use_u = (c->rule_done && k.walls == CBM_WALLS_REFLECT) ? 1 : 0;
  int copy_c = (k.medium && !c->mde_done) ? 1 : 0;
  int copy_grad = (k.medium && !c->mrule_done) ? 1 : 0;
  dispatch<StageUpdate>(c, copy_agents, use_u, copy_c, copy_grad);
  c->parity ^= 1;
  reset_stage_flags(c);
  return check_launch(c);
}

int cbm_compute_neighbors(cbm_ctx* c) {
  if (!c) return CBM_ERR_ARG;
  if (!c->loaded) return fail(c, CBM_ERR_STATE, "community not uploaded");
  cudaSetDevice(c->device);
  dispatch<StageNeighbors>(c);
  return check_launch(c);
}

int cbm_sync(cbm_ctx* c) {
  if (!c) return CBM_ERR_ARG;
  cudaSetDevice(c->device);
  Counters hc;
  int rc = read_counters(c, &hc);
  if (rc) return rc;
  if (hc.err) {
    int code = flags_to_status(hc.err);
    int zero = 0;
    CUDA_TRY(c, cudaMemcpy(&c->ctr->err, &zero, sizeof zero, cudaMemcpyHostToDevice));
    const char* what = code == CBM_ERR_AGENT_OVERFLOW
                           ? "agent capacity n_max reached: births were dropped"
                           : code == CBM_ERR_NEIGHBOR_OVERFLOW
                                 ? "a Verlet row exceeded n_max_neighbors: list truncated"
                                 : "a bounded device-side wait gave up";
    return fail(c, code, "%s (device flags 0x%x)", what, hc.err);
  }
  return CBM_OK;
}

}  // extern "C"

// A fate-free CellLinked community small enough for one cluster launch of all
// its steps (cbm_small.cuh)
bool small_eligible(const cbm_ctx* c) {
  const cbm_config& k = c->cfg;
  return k.neighbors == CBM_NEIGH_CELL_LINKED && k.fate == CBM_FATE_NONE && !k.growth &&
         !k.medium && k.force_mode == CBM_FORCE_DIRECT &&
         (k.integrator == CBM_INT_EULER || k.integrator == CBM_INT_EM) &&
         c->n_cells <= kSmallMaxCells && c->n_loaded > 0 &&
         c->n_loaded <= (c->tsize == 8 ? kSmallMaxAgents<double> : kSmallMaxAgents<float>);
}

template <typename T, int D>
struct SmallSteps {
  static void run(cbm_ctx* c, int nsteps, cudaError_t* err) {
    Params<T> P0 = params<T>(c, c->parity), P1 = params<T>(c, c->parity ^ 1);
    int n_cells = c->n_cells;
    const size_t smem = (size_t)(n_cells + 1) * sizeof(int);
    auto kern = k_small_steps<T, D>;
    // one cluster of sixteen blocks, of the threads that four lanes an agent
    // need (a community of a few agents: of as many blocks as it fills)
    const long long lanes = c->n_loaded * kSmallLanes;
    int blocks = (int)std::max<long long>(
        1, std::min<long long>((lanes + kSmallMinThreads - 1) / kSmallMinThreads, kSmallMaxBlocks));
    const long long each = ((lanes + blocks - 1) / blocks + 31) / 32 * 32;
    const int threads = (int)std::max<long long>(kSmallMinThreads, std::min<long long>(each, kSmallMaxThreads));
    *err = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (*err != cudaSuccess) return;
    cudaLaunchConfig_t lc = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    lc.blockDim = dim3((unsigned)threads);
    lc.dynamicSmemBytes = smem;
    lc.stream = c->stream;
    lc.attrs = attr;
    lc.numAttrs = 1;
    for (;; blocks /= 2) {  // the largest cluster the device can schedule
      attr[0].val.clusterDim.x = (unsigned)blocks;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      lc.gridDim = dim3((unsigned)blocks);
      int clusters = 0;
      if ((cudaOccupancyMaxActiveClusters(&clusters, kern, &lc) == cudaSuccess && clusters > 0) ||
          blocks == 1)
        break;
    }
    *err = cudaLaunchKernelEx(&lc, kern, P0, P1, nsteps, n_cells);
  }
};

extern "C" {

int cbm_step(cbm_ctx* c, int32_t nsteps, int32_t flags) {
  if (!c) return CBM_ERR_ARG;
  if (!c->loaded) return fail(c, CBM_ERR_STATE, "community not uploaded");
  if (nsteps < 0) return fail(c, CBM_ERR_ARG, "nsteps must be >= 0");
  cudaSetDevice(c->device);
  if (c->rule_done || c->de_done || c->mrule_done || c->mde_done)
    return fail(c, CBM_ERR_STATE, "a step is half done through the stage calls; call cbm_update first");
  const bool use_graph = !(flags & CBM_NO_GRAPH);
  if (use_graph && nsteps > 0 && !c->graph_timing && small_eligible(c)) {
    cudaError_t e = cudaSuccess;
    dispatch<SmallSteps>(c, (int)nsteps, &e);
    if (e != cudaSuccess) return fail(c, CBM_ERR_CUDA, "small-community launch failed: %s", cudaGetErrorString(e));
    if (nsteps & 1) c->parity ^= 1;
    if (flags & CBM_SYNC) return cbm_sync(c);
    return CBM_OK;
  }
  for (int s = 0; s < nsteps; ++s) {
    const int p = c->parity;
    if (use_graph && !c->graph_timing && c->side && nsteps - s >= kChainSteps) {
      if (!c->chain[p]) {
        cudaGraph_t g = nullptr;
        CUDA_TRY(c, cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal));
        dispatch<ChainSteps>(c, p);
        cudaError_t e = cudaStreamEndCapture(c->stream, &g);
        if (e != cudaSuccess) return fail(c, CBM_ERR_CUDA, "graph capture failed: %s", cudaGetErrorString(e));
        e = cudaGraphInstantiate(&c->chain[p], g, instantiate_flags(c));
        cudaGraphDestroy(g);
        if (e != cudaSuccess) return fail(c, CBM_ERR_CUDA, "graph instantiate failed: %s", cudaGetErrorString(e));
      }
      CUDA_TRY(c, cudaGraphLaunch(c->chain[p], c->stream));
      s += kChainSteps - 1;  // an even count: the parity is unchanged
      continue;
    }
    if (use_graph) {
      cudaGraphExec_t* graphs = c->graph_timing ? c->tgraph : c->graph;
      if (!graphs[p]) {
        cudaGraph_t g = nullptr;
        CUDA_TRY(c, cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal));
        if (c->graph_timing) {  // event records around each kernel become graph nodes
          c->prof = true;
          c->prof_set = &c->gmarks[p];
          c->prof_used = &c->gmark_used[p];
          c->gmark_used[p] = 0;
        }
        dispatch<FullStep>(c, p);
        c->prof = false;
        c->prof_set = nullptr;
        c->prof_used = nullptr;
        cudaError_t e = cudaStreamEndCapture(c->stream, &g);
        if (e != cudaSuccess) return fail(c, CBM_ERR_CUDA, "graph capture failed: %s", cudaGetErrorString(e));
        e = cudaGraphInstantiate(&graphs[p], g, instantiate_flags(c));
        cudaGraphDestroy(g);
        if (e != cudaSuccess) return fail(c, CBM_ERR_CUDA, "graph instantiate failed: %s", cudaGetErrorString(e));
      }
      CUDA_TRY(c, cudaGraphLaunch(graphs[p], c->stream));
    } else {
      dispatch<FullStep>(c, p);
      int rc = check_launch(c);
      if (rc) return rc;
    }
    c->parity ^= 1;
  }
  if (flags & CBM_SYNC) return cbm_sync(c);
  return CBM_OK;
}

int cbm_step_noise(cbm_ctx* c, const void* noise, int32_t flags) {
  if (!c) return CBM_ERR_ARG;
  if (!c->loaded) return fail(c, CBM_ERR_STATE, "community not uploaded");
  if (c->cfg.integrator != CBM_INT_EM)
    return fail(c, CBM_ERR_ARG, "external noise needs the Euler-Maruyama integrator");
  if (c->rule_done || c->de_done || c->mrule_done || c->mde_done)
    return fail(c, CBM_ERR_STATE, "a step is half done through the stage calls; call cbm_update first");
  cudaSetDevice(c->device);
  Counters hc;
  int rc = read_counters(c, &hc);
  if (rc) return rc;
  const long long N = hc.N[c->parity];
  const size_t bytes = (size_t)N * (size_t)c->cfg.dims * c->tsize;
  if (N > 0 && !noise) return fail(c, CBM_ERR_ARG, "noise is NULL");
  if (!c->ext_noise) {
    CUDA_TRY(c, cudaMalloc(&c->ext_noise,
                           (size_t)(c->cfg.n_max > 0 ? c->cfg.n_max : 1) * c->cfg.dims * c->tsize));
    c->allocs.push_back(c->ext_noise);
  }
  if (bytes) CUDA_TRY(c, cudaMemcpyAsync(c->ext_noise, noise, bytes, cudaMemcpyHostToDevice, c->stream));
  c->ext_noise_on = true;  // read by params() for this step only; the step graphs keep the stream
  dispatch<FullStep>(c, c->parity);
  c->ext_noise_on = false;
  rc = check_launch(c);
  if (rc) return rc;
  c->parity ^= 1;
  // the host buffer is borrowed for the call only
  CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  if (flags & CBM_SYNC) return cbm_sync(c);
  return CBM_OK;
}

int cbm_get_counters(cbm_ctx* c, int64_t* N, int64_t* n_add, int64_t* n_remove, int64_t* id_max,
                     int32_t* flag_recompute, int64_t* stepc) {
  if (!c) return CBM_ERR_ARG;
  cudaSetDevice(c->device);
  Counters hc;
  int rc = read_counters(c, &hc);
  if (rc) return rc;
  const int p = c->parity;
  if (N) *N = hc.N[p];
  if (n_add) *n_add = hc.n_add;
  if (n_remove) *n_remove = hc.n_remove;
  if (id_max) *id_max = hc.id_max;
  // flag of the step in flight, or of the step that just ended
  if (flag_recompute) *flag_recompute = (c->rule_done || c->de_done) ? hc.flag[p] : hc.flag[p ^ 1];
  if (stepc) *stepc = hc.step[p];
  return CBM_OK;
}

int cbm_grid_shape(cbm_ctx* c, int32_t* n3) {
  if (!c || !n3) return CBM_ERR_ARG;
  for (int d = 0; d < 3; ++d) n3[d] = c->grid_exposed ? c->n_cells_d[d] : 1;
  return CBM_OK;
}

int cbm_get_grid(cbm_ctx* c, int32_t* agent_cell, int32_t* cell_start, int32_t* cell_count,
                 int32_t* cell_agents) {
  if (!c) return CBM_ERR_ARG;
  if (!c->grid_exposed) return fail(c, CBM_ERR_STATE, "this neighbor algorithm has no cell grid");
  cudaSetDevice(c->device);
  Counters hc;
  int rc = read_counters(c, &hc);
  if (rc) return rc;
  const long long N = hc.N[c->parity];
  std::vector<int> start((size_t)c->n_cells + 1), ia((size_t)N), inv((size_t)N), cos((size_t)N);
  CUDA_TRY(c, cudaMemcpy(start.data(), c->cell_start, start.size() * 4, cudaMemcpyDeviceToHost));
  if (N) {
    CUDA_TRY(c, cudaMemcpy(ia.data(), c->IA, (size_t)N * 4, cudaMemcpyDeviceToHost));
    CUDA_TRY(c, cudaMemcpy(inv.data(), c->inv, (size_t)N * 4, cudaMemcpyDeviceToHost));
    CUDA_TRY(c, cudaMemcpy(cos.data(), c->cell_of_slot, (size_t)N * 4, cudaMemcpyDeviceToHost));
  }
  for (int q = 0; q < c->n_cells; ++q) {
    if (cell_start) cell_start[q] = start[q];
    if (cell_count) cell_count[q] = start[q + 1] - start[q];
  }
  for (long long i = 0; i < N; ++i) {
    if (cell_agents) cell_agents[i] = ia[(size_t)i];  // slots are in cell order
    if (agent_cell) agent_cell[i] = cos[(size_t)inv[(size_t)i]];
  }
  return CBM_OK;
}

int cbm_get_neighbors(cbm_ctx* c, int32_t* counts, int32_t* list, int64_t cap) {
  if (!c) return CBM_ERR_ARG;
  if (!c->has_list) return fail(c, CBM_ERR_STATE, "this neighbor algorithm has no Verlet list");
  cudaSetDevice(c->device);
  int rc = ensure_list(c);
  if (rc) return rc;
  Counters hc;
  rc = read_counters(c, &hc);
  if (rc) return rc;
  const long long N = hc.N[c->parity];
  const long long M = c->cfg.n_max_neighbors, nmax = c->cfg.n_max;
  if (list && cap < N * M) return fail(c, CBM_ERR_ARG, "list capacity %lld < N*n_max_neighbors", (long long)cap);
  std::vector<int> n((size_t)N), ia((size_t)N), inv((size_t)N), col;
  if (N) {
    CUDA_TRY(c, cudaMemcpy(n.data(), c->nbr_n, (size_t)N * 4, cudaMemcpyDeviceToHost));
    CUDA_TRY(c, cudaMemcpy(ia.data(), c->IA, (size_t)N * 4, cudaMemcpyDeviceToHost));
    CUDA_TRY(c, cudaMemcpy(inv.data(), c->inv, (size_t)N * 4, cudaMemcpyDeviceToHost));
  }
  if (list && N) {
    col.resize((size_t)(nmax * M));
    CUDA_TRY(c, cudaMemcpy(col.data(), c->nbr_list, col.size() * 4, cudaMemcpyDeviceToHost));
  }
  for (long long i = 0; i < N; ++i) {
    const long long s = inv[(size_t)i];
    if (counts) counts[i] = n[(size_t)s];
    if (list)
      for (long long q = 0; q < M; ++q)
        list[i * M + q] = q < n[(size_t)s] ? ia[(size_t)col[(size_t)(q * nmax + s)]] : -1;
  }
  return CBM_OK;
}

int cbm_count_neighbors(cbm_ctx* c, double radius, int32_t* out) {
  if (!c || !out) return CBM_ERR_ARG;
  if (!c->loaded) return fail(c, CBM_ERR_STATE, "community not uploaded");
  cudaSetDevice(c->device);
  Counters hc;
  int rc = read_counters(c, &hc);
  if (rc) return rc;
  const long long N = hc.N[c->parity];
  dispatch<CountNeighbors>(c, radius, c->scratch_int);
  rc = check_launch(c);
  if (rc) return rc;
  CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  if (N) CUDA_TRY(c, cudaMemcpy(out, c->scratch_int, (size_t)N * 4, cudaMemcpyDeviceToHost));
  return CBM_OK;
}

int cbm_rng_fill(cbm_ctx* c, int32_t kind, double a, double b, int64_t n, int64_t stepc, void* out) {
  if (!c || !out || n < 0) return CBM_ERR_ARG;
  if (kind < 0 || kind > 2) return fail(c, CBM_ERR_ARG, "kind must be 0, 1 or 2");
  cudaSetDevice(c->device);
  void* buf = nullptr;
  const size_t bytes = (size_t)(n > 0 ? n : 1) * c->tsize;
  CUDA_TRY(c, cudaMallocAsync(&buf, bytes, c->stream));
  const int blocks = grid_blocks(n);
  if (n > 0) {
    if (c->cfg.precision == CBM_F64)
      k_rng_fill<double><<<blocks, kTile, 0, c->stream>>>(c->cfg.seed, c->cfg.community, stepc, kind, a,
                                                         b, n, (double*)buf);
    else
      k_rng_fill<float><<<blocks, kTile, 0, c->stream>>>(c->cfg.seed, c->cfg.community, stepc, kind,
                                                        (float)a, (float)b, n, (float*)buf);
  }
  int rc = check_launch(c);
  if (!rc && n > 0) {
    cudaError_t e = cudaMemcpyAsync(out, buf, (size_t)n * c->tsize, cudaMemcpyDeviceToHost, c->stream);
    if (e != cudaSuccess) rc = fail(c, CBM_ERR_CUDA, "copy failed: %s", cudaGetErrorString(e));
  }
  cudaFreeAsync(buf, c->stream);
  cudaError_t e = cudaStreamSynchronize(c->stream);
  if (!rc && e != cudaSuccess) rc = fail(c, CBM_ERR_CUDA, "rng fill failed: %s", cudaGetErrorString(e));
  return rc;
}

void* cbm_stream(cbm_ctx* c) { return c ? (void*)c->stream : nullptr; }

int cbm_profile_step(cbm_ctx* c, int32_t max_kernels, float* ms, const char** names,
                     int32_t* n_kernels) {
  if (!c || !n_kernels) return CBM_ERR_ARG;
  if (!c->loaded) return fail(c, CBM_ERR_STATE, "community not uploaded");
  if (c->rule_done || c->de_done || c->mrule_done || c->mde_done)
    return fail(c, CBM_ERR_STATE, "a step is half done through the stage calls; call cbm_update first");
  cudaSetDevice(c->device);
  c->prof = true;
  c->mark_used = 0;
  dispatch<FullStep>(c, c->parity);
  c->prof = false;
  int rc = check_launch(c);
  if (rc) return rc;
  c->parity ^= 1;
  CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  *n_kernels = (int32_t)c->mark_used;
  for (size_t q = 0; q < c->mark_used && (int)q < max_kernels; ++q) {
    float t = 0.f;
    CUDA_TRY(c, cudaEventElapsedTime(&t, c->marks[q].ev[0], c->marks[q].ev[1]));
    if (ms) ms[q] = t;
    if (names) names[q] = c->marks[q].name;
  }
  return cbm_sync(c);
}

int cbm_kernels_per_step(cbm_ctx* c) { return c ? kernels_per_step(c) : 0; }

int cbm_set_kernel_timing(cbm_ctx* c, int32_t on) {
  if (!c) return CBM_ERR_ARG;
  cudaSetDevice(c->device);
  CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  c->graph_timing = on != 0;  // the two sets of step graphs are kept apart
  return CBM_OK;
}

int cbm_kernel_times(cbm_ctx* c, int32_t max_kernels, float* ms, const char** names,
                     int32_t* n_kernels) {
  if (!c || !n_kernels) return CBM_ERR_ARG;
  if (!c->graph_timing) return fail(c, CBM_ERR_STATE, "kernel timing is off (cbm_set_kernel_timing)");
  cudaSetDevice(c->device);
  const int p = c->parity ^ 1;  // the parity of the step replayed last
  if (!c->tgraph[p]) return fail(c, CBM_ERR_STATE, "no step graph has been replayed yet");
  CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  *n_kernels = (int32_t)c->gmark_used[p];
  for (size_t q = 0; q < c->gmark_used[p] && (int)q < max_kernels; ++q) {
    float t = 0.f;
    CUDA_TRY(c, cudaEventElapsedTime(&t, c->gmarks[p][q].ev[0], c->gmarks[p][q].ev[1]));
    if (ms) ms[q] = t;
    if (names) names[q] = c->gmarks[p][q].name;
  }
  return CBM_OK;
}

}  // extern "C"
