// cbm_tile.cuh — the 3D force walk by tiles of 32 agents.
//
// One warp owns 32 consecutive slots.  Slots are sorted by cell, so its agents
// sit in one or a few cells of one row and share nearly all their candidates.
// The filter (which candidates may lie within the cutoff) is a contraction:
//     |xi - xj|^2 - R^2 = (|xi|^2 - R^2) + |xj|^2 - 2 xi . xj
// over the coordinates relative to the tile, in units of the cutoff's power of
// two (cbm_tile_filter.h), so 16 agents x 8 candidates are one mma.m16n8k8 (half inputs, float accumulators), and the sign of an
// accumulator is the decision: one funnel shift per pair collects it into a
// word of 32 decisions (against about eleven instructions per pair when a
// thread tests its own candidates).  The filter only has to keep every pair
// that the evaluation's exact test keeps (tile_row); the evaluation then
// walks each agent's own words in candidate order and computes the terms
// exactly as the reference does, so the sums are unchanged, bit for bit.
#pragma once
#include <cuda_fp16.h>

#include "cbm_kernels.cuh"
#include "cbm_tile_filter.h"

namespace cbm {

// Decisions are kept as a ring of words of 32 candidates per agent: 27 cells
// at 4 agents per unit volume (edge 3.3) are about 126 words.  The agents of
// a tile find their partners in different parts of the walk (one near the
// lower face of its cell mostly in the plane below), so each consumes its
// words at its own pace, and the ring is refilled when the slowest has
// consumed a third of it.  A ring of 48 words (6 KB a warp) and thirteen
// warps an SM leave 124 KB of L1 to the partners' positions: measured on the
// colony of 1e6 agents, 96 words and fifteen warps 2.28 ms (28 KB of L1), 80
// and sixteen 2.14, 64 and sixteen 2.17 (60 KB), 48 and thirteen 2.05 (124
// KB), 40 and fifteen 2.26, 40 and ten 2.31 (156 KB).
constexpr int kTileWords = 48;
constexpr int kTileRefill = 16;
constexpr int kTileWarps = 13;    // one-warp blocks an SM
constexpr int kTileCarveout = 58; // percent: 132 KB of shared memory
static_assert(kTileWords % 4 == 0 && kTileRefill % 4 == 0, "the filter takes four words at a time");
// bytes between the records of two words: 32 records of 16 bytes and a shift
// of 8 banks, so that the eight rows of an ldmatrix (two records of each of
// four words) fall into different banks
constexpr int kTileWordStride = 32 * 16 + 32;
template <typename S>
__device__ __forceinline__ void tile_begin(S& s) {  // the empty word
  s.word[kTileWords * 32 + (threadIdx.x & 31)] = 0u;
  s.base[kTileWords] = 0;
}

// Near candidates a lane holds when it walks its own; its runs lie above them.
constexpr int kNearQueue = 24;
static_assert(kNearQueue * 32 + 2 * 9 * 32 <= kTileWords * 32, "queue and runs fit the words");
struct TileSmem {
  // decisions of word w, agent a; then an empty word
  alignas(8) unsigned word[(kTileWords + 1) * 32];
  int base[kTileWords + 1];              // first slot of word w
  unsigned short info[kTileWords];       // run (0..8) | number of candidates << 8
  __align__(16) unsigned char rec[4 * kTileWordStride];  // records of four words
};

__device__ __forceinline__ unsigned half2_bits(float lo, float hi) {
  const __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const unsigned*>(&h);
}

__device__ __forceinline__ void ldmatrix4(unsigned* r, unsigned addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}

// d = a b + (ca, ca, cb, cb): rows g and g + 8 of 16 agents against 8 candidates
__device__ __forceinline__ void mma_16x8x8(float* d, unsigned a0, unsigned a1, unsigned b, float ca,
                                           float cb) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
      "{%7,%7,%8,%8};\n"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(b), "f"(ca), "f"(cb));
}

// The records of tile_candidate and tile_row as eight halves: k = 0 .. 7 of
// the contraction.
__device__ __forceinline__ uint4 tile_record(const TileRecord& r) {
  return make_uint4(half2_bits(r.v[0], r.v[1]), half2_bits(r.v[2], r.v[3]),
                    half2_bits(r.v[4], 0.f), 0u);
}

// The branch-free form's coefficients (cbm_pair.cuh) of the model.
template <typename T>
__device__ __forceinline__ PairLine<T> pair_line(const Params<T>& P) {
  return make_pair_line<T>(P.cut2, P.k_rep, P.r_rep, P.k_att, P.r_att,
                           P.att_form == CBM_ATT_FROM_REP);
}

// The terms of four partners at positions v, added to acc in order; an entry
// that is the agent itself adds nothing.  `plain`: the positions are within
// kTileReach of one another and L.mid holds.  Returns the entries within the
// cutoff (bit u).
template <typename T>
__device__ __forceinline__ int pair_terms4(const PairCoef<T>& c, const PairLine<T>& L, bool plain,
                                            const T* xi, const typename V4T<T>::type* v, int s,
                                            const int* qq, T* acc) {
  if constexpr (std::is_same<T, float>::value) {
    const bool none[4] = {qq[0] == s, qq[1] == s, qq[2] == s, qq[3] == s};
    if (plain) {
      const int in = pair_terms4_mid<false>(L, xi, v, none, acc);
      if (in >= 0) return in;
    }
  }
  if constexpr (std::is_same<T, double>::value) {
    double e[4][3], n2[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      double xj[3];
      to3<double>(v[u], xj);
      const double d2 = pair_diff<double, 3>(xi, xj, e[u]);
      n2[u] = qq[u] == s ? -L.nfar2 : d2;
    }
    if (plain && fmin(fmin(n2[0], n2[1]), fmin(n2[2], n2[3])) > 1e-12 && mid_root(n2[0]) &&
        mid_root(n2[1]) && mid_root(n2[2]) && mid_root(n2[3])) {
      double sc[4];
      int in = 0;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        double y;
        const double d = sqrt_mid(n2[u], &y);
        const bool rep = d < -L.nrrep;
        const double F = (rep ? L.krep : L.katt) * ((rep ? L.rrep : L.abase) - d);
        const double q = div_mid(F, d, y);
        sc[u] = d < -L.nreach ? q : 0.0;
        in |= d < -L.nreach ? 1 << u : 0;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int k = 0; k < 3; ++k) acc[k] = acc[k] + sc[u] * e[u][k];
      return in;
    }
  }
  int in = 0;
#pragma unroll
  for (int u = 0; u < 4; ++u)
    if (qq[u] != s) {
      T xj[3], e[3];
      to3<T>(v[u], xj);
      const T d2 = pair_diff<T, 3>(xi, xj, e);
      if (pair_term<T, 3>(c, e, d2, acc)) in |= 1 << u;
    }
  return in;
}

// The pair forces of the 32 slots from s0 on (lanes beyond N idle), summed
// into acc in the reference's order; partner(slot) is told of every pair with
// a force, in that order.
template <typename T, typename F>
__device__ __forceinline__ void tile_forces(const Params<T>& P, TileSmem& S, const int N,
                                            const int s0, const T* xi, T* acc, F&& partner) {
  using V4 = typename V4T<T>::type;
  const int lane = threadIdx.x & 31;
  const bool in = s0 + lane < N;
  const int s = in ? s0 + lane : N - 1;
  const V4* const U = P.PA;
  const PairCoef<T> coef = pair_coef<T>(P);
  const int nx = P.n_cells_d[0], ny = P.n_cells_d[1], nz = P.n_cells_d[2];
  const int cell = ld(P.cell_of_slot + s);
  const int q0 = cell % nx, q1 = (cell / nx) % ny, q2 = cell / (nx * ny);
  // the nine runs of the agent's 27 cells: rows (dy, dz), each the slots of
  // up to three cells along x
  const int xa = q0 > 0 ? q0 - 1 : 0, xb = q0 < nx - 1 ? q0 + 1 : nx - 1;
  const int row0 = nx * (q1 - 1 + ny * (q2 - 1));
  int lo[9], hi[9], cand = 0;
#pragma unroll
  for (int r = 0; r < 9; ++r) {
    const int py = q1 + r % 3 - 1, pz = q2 + r / 3 - 1;
    lo[r] = hi[r] = 0;
    if (py >= 0 && py < ny && pz >= 0 && pz < nz) {
      const int row = tile_run_row(row0, nx, ny, r);
      lo[r] = ld(P.cell_start + row + xa);
      hi[r] = ld(P.cell_start + row + xb + 1);
    }
    cand += hi[r] - lo[r];
  }
  // agents of the same row of cells share their nine runs (up to their ends
  // along x): the tile is processed row by row
  const unsigned live = __ballot_sync(kFull, in);
  const unsigned peers = __match_any_sync(kFull, in ? cell / nx : -1);
  const unsigned leaders = __ballot_sync(kFull, in && (peers & ((1u << lane) - 1u)) == 0u);
  const int n_rows = __popc(leaders);
  const int cell0 = __shfl_sync(kFull, cell, 0);
  const bool ranged = __any_sync(kFull, in && cell != cell0);
  int u0 = 0, u1 = 0;  // lane r < 9: the run r of the current row of agents
  auto unite = [&](unsigned gm) -> int {
    const bool member = (gm >> lane) & 1u;
    int words = 0;
#pragma unroll
    for (int r = 0; r < 9; ++r) {
      const int a = __reduce_min_sync(kFull, member && hi[r] > lo[r] ? lo[r] : 0x7fffffff);
      const int b = __reduce_max_sync(kFull, member ? hi[r] : 0);
      const int len = b > a ? b - a : 0;
      words += (len + 31) >> 5;
      if (lane == r) {
        u0 = len ? a : 0;
        u1 = len ? b : 0;
      }
    }
    return words;
  };
  // A word costs the warp about 75 instructions, a row of agents about 350,
  // and a candidate tested by each lane about 20: sparse tiles, whose agents
  // lie in many cells with a few candidates each, test their own.  (All tiles
  // by words against all by lanes: the young colony's kernel 46 us against
  // 76, the 256^3 medium's 159 against 55, the adjoint's 65536 agents at 0.13
  // per unit volume 195 against 115 us a step.)
  const int most = __reduce_max_sync(kFull, in ? cand : 0);
  bool by_tile = 20 * most > 350 * n_rows && P.tile_scale != (T)0;
  if (by_tile) {
    int words = 0;
    for (unsigned l = leaders; l; l &= l - 1u)
      words += unite(__shfl_sync(kFull, peers, __ffs(l) - 1));
    by_tile = 75 * words + 350 * n_rows < 20 * most;
  }
  const PairLine<T> line = pair_line(P);
  if (!by_tile) {
    // Each lane walks its own candidates, four at a time, passing over empty
    // runs (most of a sparse tile's are), the next four's positions in flight; those that may be near wait in the lane's column of
    // S.word and are evaluated together.  Runs as first slot and end, by lane.
    int2* const runs = reinterpret_cast<int2*>(S.word + 32 * kNearQueue);
#pragma unroll
    for (int r = 0; r < 9; ++r) runs[r * 32 + lane] = make_int2(lo[r], hi[r]);
    int r = 0, q = lo[0], e = in ? hi[0] : lo[0], nq = 0;
    if (!in) r = 8;
    auto take = [&](int* qq, V4* v) {
      while (q >= e && r < 8) {
        const int2 run = runs[++r * 32 + lane];
        q = run.x;
        e = run.y;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) qq[u] = q + u < e ? q + u : s;
      q += 4;
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = U[qq[u]];
    };
    auto evaluate = [&]() {
      for (int k = 0; __any_sync(kFull, k < nq); k += 4) {
        int qq[4];
        V4 v[4];
        bool plain = line.mid;
#pragma unroll
        for (int u = 0; u < 4; ++u) qq[u] = k + u < nq ? (int)S.word[(k + u) * 32 + lane] : s;
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = U[qq[u]];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          T xj[3], d[3];
          to3<T>(v[u], xj);
          plain = plain && pair_diff<T, 3>(xi, xj, d) < (T)1e12;
        }
        const int hit = pair_terms4<T>(coef, line, plain, xi, v, s, qq, acc);
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if ((hit >> u) & 1) partner(qq[u]);
      }
      nq = 0;
    };
    int qq[4];
    V4 v[4];
    take(qq, v);
    while (true) {
      const bool more = __any_sync(kFull, q < e || r < 8);
      int qn[4];
      V4 vn[4];
      if (more) take(qn, vn);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        T xj[3], d[3];
        to3<T>(v[u], xj);
        S.word[nq * 32 + lane] = (unsigned)qq[u];  // kept when it may be near (or is NaN)
        nq += qq[u] != s && !(pair_diff<T, 3>(xi, xj, d) >= coef.cut2) ? 1 : 0;
      }
      if (!more || __any_sync(kFull, nq > kNearQueue - 5)) evaluate();
      if (!more) break;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        qq[u] = qn[u];
        v[u] = vn[u];
      }
    }
    __syncwarp();
    return;
  }

  const float c = P.tile_cut;
  // The filter's unit, a power of two: the fused operation that scales rounds
  // as the difference alone does.  (A constant operand in Float32, where a
  // register for it made the walk of 1e6 agents 2.056 ms instead of 2.037; a
  // register in Float64, without which that of 1.5e5 took 255 us, not 245.)
  std::conditional_t<sizeof(T) == 4, const T&, const T> scale = P.tile_scale;
  const int g = lane >> 2, q4 = lane & 3;
  const unsigned rec = (unsigned)__cvta_generic_to_shared(S.rec);
  unsigned row_a[4];       // A fragments: agents 0-7, 8-15, 16-23, 24-31
  float start[4];          // accumulator starts of agents g, g + 8, g + 16, g + 24
  T org[3];  // minus the middle of the row's cells, in the filter's unit
  bool member = false;
  unsigned rem = leaders;
  int run = 9, k0 = 0, k1 = 0;   // next candidate and end of the run being queued
  // words are counted from 0; word n sits at n modulo kTileWords.  made:
  // words filtered; free_to: the ring has room below it; next: this lane's
  // next word, at ring position `at`; bits: what is left of its current word.
  int made = 0, ring = 0, free_to = kTileWords, next = 0, at = 0, base = 0;
  unsigned bits = 0u;
  bool far = false;  // a candidate or agent out of reach
  for (;;) {
    while (made < free_to && (run < 9 || rem)) {
      if (run == 9) {  // the next row of agents
        const int lead = __ffs(rem) - 1;
        const unsigned gm = __shfl_sync(kFull, peers, lead);
        rem &= rem - 1u;
        member = (gm >> lane) & 1u;
        if (n_rows > 1) unite(gm);
        const int qa = __shfl_sync(kFull, q0, lead), qb = __shfl_sync(kFull, q0, 31 - __clz(gm));
        org[0] = -scale * (P.box_lo[0] + ((T)(qa + qb) * (T)0.5 - (T)0.5) * P.edge);
        org[1] = -scale * (P.box_lo[1] + ((T)__shfl_sync(kFull, q1, lead) - (T)0.5) * P.edge);
        org[2] = -scale * (P.box_lo[2] + ((T)__shfl_sync(kFull, q2, lead) - (T)0.5) * P.edge);
        const T xs[3] = {fma(xi[0], scale, org[0]), fma(xi[1], scale, org[1]),
                         fma(xi[2], scale, org[2])};
        float st;
        far = far || !(fabs(xs[0]) + fabs(xs[1]) + fabs(xs[2]) <= (T)kTileReach);
        *reinterpret_cast<uint4*>(S.rec + lane * 16) =
            tile_record(tile_row((float)xs[0], (float)xs[1], (float)xs[2], c, member, &st));
#pragma unroll
        for (int k = 0; k < 4; ++k) start[k] = __shfl_sync(kFull, st, g + 8 * k);
        __syncwarp();
        ldmatrix4(row_a, rec + lane * 16);
        __syncwarp();
        run = 0;
        k0 = __shfl_sync(kFull, u0, 0);
        k1 = __shfl_sync(kFull, u1, 0);
        if (member) {  // the words before are other agents'
          next = made;
          at = ring;
        }
      }
      // queue words of the row's runs, as many as there is room for
      int n = 0, pos = ring;
      while (run < 9 && made + n < free_to) {
        const int left = (k1 - k0 + 31) >> 5, room = free_to - made - n;
        const int take = left < room ? left : room;
        for (int k = lane; k < take; k += 32) {
          const int b = k0 + 32 * k;
          int w = pos + k;
          w = w >= kTileWords ? w - kTileWords : w;
          S.base[w] = b;
          S.info[w] = tile_info(run, k1 - b < 32 ? k1 - b : 32);
        }
        n += take;
        pos += take;
        pos = pos >= kTileWords ? pos - kTileWords : pos;
        k0 += 32 * take;
        if (k0 >= k1) {
          ++run;
          k0 = __shfl_sync(kFull, u0, run);
          k1 = __shfl_sync(kFull, u1, run);
        }
      }
      for (; n & 3; ++n) {  // whole groups of four
        S.base[pos] = 0;
        S.info[pos] = kTilePad;
        ++pos;
      }
      __syncwarp();
      // filter: four words (128 candidates) at a time; lane `lane` prepares
      // candidate `lane` of each word, and the loads of the next four words
      // are in flight while these are multiplied
      V4 v[4];
      auto fetch = [&](int w) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          v[j] = U[lane < (S.info[w + j] >> 8) ? S.base[w + j] + lane : s];
      };
      int w = ring, cur = -1, rlo = 0, rhi = 0;
      if (n) fetch(w);
      for (int k = 0; k < n; k += 4) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          T xj[3];
          to3<T>(v[j], xj);
          *reinterpret_cast<uint4*>(S.rec + j * kTileWordStride + lane * 16) = tile_record(
              tile_candidate((float)fma(xj[0], scale, org[0]), (float)fma(xj[1], scale, org[1]),
                             (float)fma(xj[2], scale, org[2]), lane < (S.info[w + j] >> 8), &far));
        }
        __syncwarp();
        const int wn = w + 4 == kTileWords ? 0 : w + 4;
        if (k + 4 < n) fetch(wn);
        // column n of multiplication t is candidate 2t + (n & 1) of word n / 2:
        // thread (g, q4) then holds candidates 2t and 2t + 1 of word q4
        const unsigned addr = rec + ((lane & 7) >> 1) * kTileWordStride + (lane & 1) * 16 +
                              (lane >> 3) * 32;
        unsigned m[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int t4 = 0; t4 < 4; ++t4) {
          unsigned b[4];
          ldmatrix4(b, addr + t4 * 128);
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            float d[8];
            mma_16x8x8(d, row_a[0], row_a[1], b[t], start[0], start[1]);
            mma_16x8x8(d + 4, row_a[2], row_a[3], b[t], start[2], start[3]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              m[i] = __funnelshift_l(__float_as_uint(d[2 * i]), m[i], 1);
              m[i] = __funnelshift_l(__float_as_uint(d[2 * i + 1]), m[i], 1);
            }
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) S.word[(w + q4) * 32 + g + 8 * i] = m[i];
        __syncwarp();
        if (ranged && member) {  // keep the agent's own cells of the shared runs
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int r = S.info[w + j] & 255, b = S.base[w + j];
            if (r != cur) {
              cur = r;
              const int row = tile_run_row(row0, nx, ny, r);
              rlo = ld(P.cell_start + row + xa);
              rhi = ld(P.cell_start + row + xb + 1);
            }
            const int skip = rlo - b, keep = rhi - b;
            unsigned own = 0xffffffffu;
            if (skip > 0) own = skip < 32 ? own >> skip : 0u;
            if (keep < 32) own &= keep > 0 ? ~(0xffffffffu >> keep) : 0u;
            S.word[(w + j) * 32 + lane] &= own;
          }
        }
        w = wn;
      }
      ring = w;
      made += n;
    }
    const bool last = run == 9 && rem == 0u;

    // evaluation: each lane walks its own words, four partners at a time (the
    // positions of four are in flight together; their terms are added in
    // order), until the slowest has freed kTileRefill words, or to the end.
    // The next word is read one ahead of its use; position kTileWords is empty.
    const bool plain = line.mid && !__any_sync(kFull, far);
    const int goal = last ? made : free_to - kTileWords + kTileRefill;
    unsigned nbits;
    int nbase;
    auto read = [&]() {
      const int p = next < made ? at : kTileWords;
      nbits = S.word[p * 32 + lane];
      nbase = S.base[p];
    };
    read();
    while (__any_sync(kFull, next < goal || (last && bits != 0u))) {
      int qq[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const bool adv = bits == 0u;
        bits = adv ? nbits : bits;
        base = adv ? nbase : base;
        const int step = adv && next < made ? 1 : 0;
        next += step;
        at += step;
        at = at == kTileWords ? 0 : at;
        read();
        const int k = __clz(bits);
        qq[u] = bits ? base + k : s;
        bits &= ~(0x80000000u >> (k & 31));
      }
      V4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = U[qq[u]];
      const int hit = pair_terms4<T>(coef, line, plain, xi, v, s, qq, acc);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if ((hit >> u) & 1) partner(qq[u]);
    }
    if (last) return;
    free_to += kTileRefill;
  }
}

// agentStepDE! over the cell walk in 3D: CellLinked, and CLVD in a step with
// births or deaths (every other CLVD step is k_agent_de's).  One warp a
// block, as many as are resident; tile t is block t's, further ones come from
// a ticket counter that the last block to finish resets.
template <typename T>
__global__ void __launch_bounds__(32, kTileWarps) k_agent_de_tile(Params<T> P) {
  __shared__ TileSmem S;
  pdl_wait();
  Counters* C = P.ctr;
  if (P.neighbors == CBM_NEIGH_CLVD && !clvd_walks_cells(P)) return;
  const int N = (int)C->N[P.parity];
  const int n_tiles = (N + 31) >> 5;
  const int lane = threadIdx.x & 31;
  tile_begin(S);
  int tile = (int)blockIdx.x;
  while (tile < n_tiles) {
    const int s = tile * 32 + lane;
    T xi[3], acc[3] = {(T)0, (T)0, (T)0};
    to3<T>(P.PA[s < N ? s : N - 1], xi);
    tile_forces<T>(P, S, N, tile * 32, xi, acc, [](int) {});
    if (s < N) finish_agent<T, 3>(P, s, xi, acc);
    __syncwarp();
    int t = 0;
    if (lane == 0) t = (int)atomicAdd(&C->de_ticket, 1u);
    tile = (int)gridDim.x + __shfl_sync(kFull, t, 0);
  }
  if (lane == 0) {
    __threadfence();
    if (atomicAdd(&C->de_done, 1u) == gridDim.x - 1) {
      C->de_ticket = 0u;
      C->de_done = 0u;
    }
  }
}

}  // namespace cbm
