"""The tiled force walk's candidate filter against the pair test itself, on the
CPU: every pair with a force must be kept, whatever the unit of length, with
the stated bound of the contraction's roundings held against it, and few
others may be.  And the cells that a word's agents look up, which must exist."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>
#include "cbm_tile_filter.h"
using namespace cbm;

// Agents of cell q and candidates of the 27 cells around it; `off`: the cell's
// distance from the origin, in cells.
template <typename T>
int run(const char* name, double cutoff, double edge_, double off, int n) {
  std::mt19937_64 g(5);
  std::uniform_real_distribution<double> u(0.0, 1.0);
  const double scale_ = tile_scale(cutoff, edge_);
  if (scale_ == 0.0) {
    std::printf("%s cutoff %g: not served\n", name, cutoff);
    return 1;
  }
  const T scale = (T)scale_, edge = (T)edge_, lo = (T)(-off * edge_);
  const float c = (float)(cutoff * scale_ * (1.0 + 1e-5));
  const int q = (int)off + 1;  // cell q holds lo + (q - 1) edge .. lo + q edge
  const T org = -scale * (lo + ((T)q - (T)0.5) * edge);
  auto place = [&](double from, double cells, T* x, float* xs) {
    for (int d = 0; d < 3; ++d) {
      x[d] = (T)(-off * edge_ + (q - 1 + from + cells * u(g)) * edge_);
      xs[d] = (float)std::fma(x[d], scale, org);
    }
  };
  std::vector<T> cx(3 * (size_t)n);
  std::vector<TileRecord> cr((size_t)n);
  bool far = false;
  for (int j = 0; j < n; ++j) {
    float xs[3];
    place(-1.0, 3.0, &cx[3 * j], xs);
    cr[j] = tile_candidate(xs[0], xs[1], xs[2], true, &far);
  }
  long partners = 0, lost = 0, kept = 0;
  for (int i = 0; i < n / 4; ++i) {
    T x[3];
    float xs[3], start;
    place(0.0, 1.0, x, xs);
    const TileRecord r = tile_row(xs[0], xs[1], xs[2], c, true, &start);
    const double X = std::sqrt((double)xs[0] * xs[0] + (double)xs[1] * xs[1] + (double)xs[2] * xs[2]);
    const double R = c * 1.01, M = (X + R) * (X + R);
    for (int j = 0; j < n; ++j) {
      T s2 = (T)0;
      for (int d = 0; d < 3; ++d) {
        const T e = x[d] - cx[3 * j + d];
        s2 = s2 + e * e;
      }
      const bool partner = std::sqrt(s2) < (T)cutoff;
      double s = start;
      for (int k = 0; k < 5; ++k) s += (double)half_round(r.v[k]) * half_round(cr[j].v[k]);
      partners += partner;
      lost += partner && !(s + M * 3.814697265625e-06 < 0.0);  // 2^-18
      kept += s < 0.0;
    }
  }
  const double per = partners ? (double)kept / partners : 0.0;
  const bool bad = lost != 0 || far || (partners > 1000 && per > 1.1);
  if (bad || partners < 100)
    std::printf("%s cutoff %g off %g: partners %ld lost %ld kept %.3f far %d\n", name, cutoff, off,
                partners, lost, per, far);
  return bad || partners < 100;
}

int main() {
  int bad = 0;
  for (int e = -7; e <= 1; ++e)
    for (double m : {1.0, 1.5, 2.0, 3.7, 5.0, 7.3})
      for (double off : {0.0, 3.0, 40.0}) {
        const double c = m * std::pow(10.0, e);
        if (c > kTileMaxCutoff) continue;
        bad |= run<double>("f64", c, 1.1 * c, off, 800);
        bad |= run<float>("f32", c, 1.1 * c, off, 800);
      }
  bad |= run<double>("f64", 3e-15, 3.3e-15, 2.0, 800);
  bad |= run<float>("f32", 3e-15, 3.3e-15, 2.0, 800);
  bad |= run<double>("f64", 2.0, 40.0, 2.0, 8000);  // cells of many cutoffs
  bad |= run<float>("f32", 1e-4, 2e-3, 2.0, 8000);
  // out of reach: kept; beyond a run: never kept; lanes of another row: nothing kept
  bool far = false;
  float start, other;
  const TileRecord a = tile_row(3.f, 2.f, 1.f, 1.5f, true, &start), z = tile_row(3.f, 2.f, 1.f, 1.5f, false, &other);
  const TileRecord o = tile_row(1e9f, 0.f, 0.f, 1.5f, true, &other);
  auto sum = [](float s, const TileRecord& r, const TileRecord& c) {
    for (int k = 0; k < 5; ++k) s += half_round(r.v[k]) * half_round(c.v[k]);
    return s;
  };
  const TileRecord f = tile_candidate(1e9f, 0.f, 0.f, true, &far);
  const TileRecord nan = tile_candidate(NAN, 0.f, 0.f, true, &far), inf = tile_candidate(0.f, -INFINITY, 0.f, true, &far);
  const TileRecord no = tile_candidate(3.f, 2.f, 1.f, false, &far), near = tile_candidate(3.f, 2.f, 1.f, true, &far);
  for (const TileRecord& r : {a, o})
    for (const TileRecord& k : {f, nan, inf}) {
      const float s = r.v[0] == 0.f ? -61000.f : start;
      if (!(sum(s, r, k) < 0.f)) bad |= 1, std::puts("a far candidate is lost");
    }
  if (!(sum(-61000.f, o, near) < 0.f)) bad |= 1, std::puts("a far agent loses a candidate");
  if (sum(-61000.f, o, no) < 0.f || sum(start, a, no) < 0.f) bad |= 1, std::puts("an entry beyond the run is kept");
  if (sum(1.f, z, near) < 0.f) bad |= 1, std::puts("a lane of another row keeps a candidate");
  // not served: these keep the walk by threads
  for (double c : {0.0, 1e-19, 51.0, 1e5, -1.0, (double)NAN})
    if (tile_scale(c, c) != 0.0) bad |= 1, std::puts("served");
  if (tile_scale(1.0, 26.0) != 0.0) bad |= 1, std::puts("served");
  return bad;
}
"""

# The masks of words shared by agents of several cells read cell_start at the
# first cell and one past the last of the word's run, for every word that the
# queue writes: those of the rows that the grid has, and the filling of a
# group of four.  Agents sit in every cell, the outermost layers included.
ROWS = r"""
#include <cstdio>
#include "cbm_tile_filter.h"
using namespace cbm;
int main() {
  int bad = 0;
  for (int nx = 1; nx <= 4; ++nx)
    for (int ny = 1; ny <= 4; ++ny)
      for (int nz = 1; nz <= 4; ++nz)
        for (int c = 0; c < nx * ny * nz; ++c) {
          const int q0 = c % nx, q1 = (c / nx) % ny, q2 = c / (nx * ny);
          const int row0 = nx * (q1 - 1 + ny * (q2 - 1));
          const int xa = q0 > 0 ? q0 - 1 : 0, xb = q0 < nx - 1 ? q0 + 1 : nx - 1;
          auto look = [&](unsigned short info) {
            const int row = tile_run_row(row0, nx, ny, info & 255);
            if (row + xa < 0 || row + xb + 1 > nx * ny * nz) {
              if (!bad) std::printf("grid %d %d %d cell %d run %d: row %d\n", nx, ny, nz, c, info & 255, row);
              bad = 1;
            }
          };
          for (int r = 0; r < 9; ++r) {
            const int py = q1 + r % 3 - 1, pz = q2 + r / 3 - 1;
            if (py >= 0 && py < ny && pz >= 0 && pz < nz) look(tile_info(r, 32));
          }
          look(kTilePad);
        }
  return bad | (kTilePad >> 8);
}
"""


def run_program(tmp_path, source):
    src = tmp_path / "filter.cpp"
    src.write_text(source)
    exe = tmp_path / "filter"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "cellbasedmodels.jl_b200", "csrc"), str(src), "-o",
                    str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


def test_filter_keeps_every_partner(tmp_path):
    run_program(tmp_path, PROGRAM)


def test_words_look_up_existing_cells(tmp_path):
    run_program(tmp_path, ROWS)
