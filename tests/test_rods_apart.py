"""The rods' contact filter against the contact force itself, on the CPU: a
pair that cbm_rod_apart rejects must have no contact in cbm_rod_forces, for
random, nearly parallel, collinear and crossing rods, lengths of zero, unequal
and negative, coordinates far from the origin, infinities and NaN; and it must
reject most of the candidates a cell walk meets."""
import subprocess

import pytest

import os

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <limits>
#include <random>
#include "cbm_rods_math.h"
template <typename T>
int run(const char* name, long rounds) {
  std::mt19937_64 g(7);
  std::uniform_real_distribution<double> u(-1.0, 1.0);
  std::uniform_int_distribution<int> pick(0, 9);
  const CbmRodCoef<T> k{(T)2, (T)2.2, (T)2.2, (T)0.1};
  const T odd[] = {std::numeric_limits<T>::quiet_NaN(), std::numeric_limits<T>::infinity(),
                   -std::numeric_limits<T>::infinity(), (T)0, std::numeric_limits<T>::max()};
  long wrong = 0, contacts = 0, plain = 0, kept = 0;
  for (long r = 0; r < rounds; ++r) {
    const int form = pick(g);
    // form 0 is a candidate of a 3 x 3 cell walk
    const double at = form == 1 ? 1e4 : form == 2 ? 1e6 : 60.0;
    const double reach = form == 3 ? 2.5 : form == 4 ? 40.0 : 8.0;
    CbmRodGeom<T> a, b;
    a.x = (T)(at * u(g));
    a.y = (T)(at * u(g));
    const double th = 3.2 * u(g);
    double th2 = 3.2 * u(g), bx = reach * u(g), by = reach * u(g);
    if (form >= 5 && form <= 7) {  // near parallel, and mostly along its line
      th2 = th + u(g) * std::pow(10.0, -1.0 - 6.0 * std::fabs(u(g)));
      const double along = 8.0 * u(g), off = u(g) * (form == 5 ? 2.0 : 0.3);
      bx = along * std::cos(th) - off * std::sin(th);
      by = along * std::sin(th) + off * std::cos(th);
    }
    a.c = (T)std::cos(th);
    a.s = (T)std::sin(th);
    b.c = (T)std::cos(th2);
    b.s = (T)std::sin(th2);
    b.x = (T)(a.x + bx);
    b.y = (T)(a.y + by);
    a.l = (T)(form == 8 ? 2.0 * u(g) : 1.5 + u(g));
    b.l = (T)(form == 8 ? 6.0 * u(g) : 1.5 + u(g));
    T d1 = (T)(form == 8 ? u(g) : 1.0), d2 = (T)(form == 8 ? u(g) : 1.0);
    if (form == 9) {
      // (the cosine and sine of an angle are both NaN or both of unit length)
      T* v[] = {&a.x, &a.y, &a.l, &b.x, &b.l, &d1, &d2, &b.y};
      const int w = pick(g);
      if (w < 8) *v[w] = odd[pick(g) % 5];
      else if (w == 8) a.c = a.s = odd[0];
      else b.c = b.s = odd[0];
    }
    T fx, fy, w;
    const bool hit = cbm_rod_forces<T>(a, d1, (T)0.1, (T)-0.2, (T)1, b, d2, (T)0, (T)0.3, k, &fx,
                                       &fy, &w);
    const bool apart = cbm_rod_apart<T>(a, d1, b, d2);
    contacts += hit;
    wrong += hit && apart;
    if (form == 0) {
      ++plain;
      kept += !apart;
    }
  }
  std::printf("%s contacts %ld wrong %ld kept %.3f\n", name, contacts, wrong, (double)kept / plain);
  return wrong != 0 || contacts < rounds / 100 || kept * 2 > plain;
}
int main(int argc, char** argv) {
  const long n = std::atol(argv[1]);
  return run<double>("f64", n) | run<float>("f32", n);
}
"""


@pytest.mark.parametrize("rounds", [3_000_000])
def test_apart_never_loses_a_contact(tmp_path, rounds):
    src = tmp_path / "apart.cpp"
    src.write_text("#include <cstdlib>\n" + PROGRAM)
    exe = tmp_path / "apart"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "include"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe), str(rounds)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
