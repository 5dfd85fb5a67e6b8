// cbm_tile_filter.h — the arithmetic of the tiled force walk's candidate
// filter (cbm_tile.cuh), for the device and for a host compiler.
//
// A candidate may lie within the cutoff of an agent when
//     start + sum_k row.v[k] * candidate.v[k] < 0,
// the expansion of |xi - xj|^2 - R^2 over coordinates relative to the tile.
// The records hold halves, whose relative precision ends at 6e-5, so lengths
// are counted in a unit that brings the cutoff into [1, 2): a power of two,
// by which scaling is exact.
#pragma once
#include <cmath>
#ifdef __CUDACC__
#include <cuda_fp16.h>
#define CBM_FILTER_HD __host__ __device__ __forceinline__
#else
#define CBM_FILTER_HD inline
#endif

namespace cbm {

// Largest |coordinate| (in the unit) that the half records hold with the
// bounds of tile_row; farther agents and candidates are always kept.
constexpr float kTileReach = 100.f;
// The filter serves cutoffs from 2^-60, above which the squared distances of
// pairs near the cutoff are normal numbers in Float32, to 50, below which
// those of all agents in reach of a tile (346 cutoffs at most) stay inside
// the branch-free terms' range; and cells of up to 25 cutoffs, whose
// neighbors are in reach.  Other cells and cutoffs keep the walk by threads.
constexpr double kTileMinCutoff = 8.673617379884035e-19;
constexpr double kTileMaxCutoff = 50.0;
constexpr double kTileMaxEdge = 25.0;

// What lengths are multiplied by; 0: the filter does not serve.
inline double tile_scale(double cutoff, double edge) {
  if (!(cutoff >= kTileMinCutoff && cutoff <= kTileMaxCutoff && edge <= kTileMaxEdge * cutoff))
    return 0.0;
  return std::ldexp(1.0, -std::ilogb(cutoff));
}
// The cutoff in the unit, raised by more than the roundings of the exact
// test (a few 2^-24).
inline float tile_cut(double cutoff, double edge) {
  return (float)(cutoff * tile_scale(cutoff, edge) * (1.0 + 1e-5));
}

CBM_FILTER_HD float half_round(float v) {
#ifdef __CUDACC__
  return __half2float(__float2half_rn(v));
#else
  return (float)(_Float16)v;
#endif
}

// Runs r = 0 .. 8 of a walk are the rows of cells (dy, dz) = (r % 3 - 1,
// r / 3 - 1) around an agent's own.  First cell of the row of run r; row0: of
// run 0, which is negative for agents in the grid's first layers (those below
// the box, or with a NaN coordinate), where the rows outside the grid have no
// run.
CBM_FILTER_HD int tile_run_row(int row0, int nx, int ny, int r) {
  return row0 + nx * (r % 3 + ny * (r / 3));
}
// What the queue notes of a word: its run and its candidates.
CBM_FILTER_HD unsigned short tile_info(int run, int candidates) {
  return (unsigned short)(run | (candidates << 8));
}
// An empty word that fills a group of four.  Its agents look its run up too:
// their own row, which every grid has.
constexpr unsigned short kTilePad = 4;

struct TileRecord {
  float v[5];  // stored as halves
};

// A candidate's record (x, y, z, nh, nl), with nh + nl its squared norm.  A
// candidate out of reach (or not a number) is kept whatever the agent, one
// beyond its run never.
CBM_FILTER_HD TileRecord tile_candidate(float x, float y, float z, bool valid, bool* far) {
  const float hx = half_round(x), hy = half_round(y), hz = half_round(z);
  const float n = fmaf(hz, hz, fmaf(hy, hy, hx * hx));
  const float nh = half_round(n);
  TileRecord r{{hx, hy, hz, nh, n - nh}};
  // (a NaN fails the test of n, whatever fmaxf makes of it)
  if (!(fmaxf(fmaxf(fabsf(x), fabsf(y)), fabsf(z)) <= kTileReach) || !(n < 60000.f)) {
    r = TileRecord{{0.f, 0.f, 0.f, -60000.f, 0.f}};
    *far = true;
  }
  if (!valid) r = TileRecord{{0.f, 0.f, 0.f, 65504.f, 0.f}};
  return r;
}

// An agent's record (-2x, -2y, -2z, 1, 1) and the start of its accumulator,
// |x|^2 - R^2, for the cutoff c of tile_cut.  With u = 2^-11 (half rounding)
// and X the agent's largest |coordinate|, a candidate inside the cutoff has
// coordinates of at most X + c, so each component of the difference of the
// rounded positions is within E = u (2X + c) + 2^-24 (two roundings below
// half's normal range; float's roundings of the relative coordinates are
// inside the excess of 4.886e-4 over u) of the exact one, and the rounded
// distance is below R = c + sqrt(3) E.  What is left are roundings in
// M = (|x| + R)^2, which bounds both squared norms and is at least 1: of n
// and of the sums in float, 2^-23 M each, of the contraction's six addends,
// 2^-22 M each if they are truncated at the largest one's last place, and of
// nh + nl, 2^-22 M or, below half's normal range, 2^-25.  They stay below
// 2^-18 M; the start is lowered by 2^-16 M.  Agents out of reach keep every
// candidate of their runs, lanes outside the tile's row none.
CBM_FILTER_HD TileRecord tile_row(float x, float y, float z, float c, bool member, float* start) {
  const float X = fmaxf(fmaxf(fabsf(x), fabsf(y)), fabsf(z));
  const float hx = half_round(x), hy = half_round(y), hz = half_round(z);
  const float n = fmaf(hz, hz, fmaf(hy, hy, hx * hx));
  const float R = c + 1.7320509f * (4.886e-4f * (2.f * X + c) + 3e-6f);
  const float m = sqrtf(n) + R;
  *start = n - R * R - 1.52587890625e-5f * (m * m);
  TileRecord r{{-2.f * hx, -2.f * hy, -2.f * hz, 1.f, 1.f}};
  if (!(X <= kTileReach)) {
    r = TileRecord{{0.f, 0.f, 0.f, 1.f, 1.f}};
    *start = -61000.f;
  }
  if (!member) {
    r = TileRecord{{0.f, 0.f, 0.f, 0.f, 0.f}};
    *start = 1.f;
  }
  return r;
}

}  // namespace cbm
