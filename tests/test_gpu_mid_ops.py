"""The branch-free square root and quotient of the pair terms (sqrt_mid,
div_mid) and the terms made of them, against the general operations, bit for
bit.  Float32: every root and every reciprocal of the range that they are used
in.  Float64: what their proof (beside them) leaves to a check, which are
finitely many operands, and random ones."""
import importlib.util
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "cellbasedmodels.jl_b200")
pytestmark = pytest.mark.gpu


def hard_roots():
    """Float64 x in [1, 4) whose root is within 12 u^2 (relative, u = 2^-53) of
    a midpoint m of two numbers: with M = m / u odd, x / u^2 = M^2 + j for a
    |j| below 96, and x a multiple of 2 u (below 2) or 4 u."""
    found = []
    for bits, lo, hi in ((54, 1 << 106, 1 << 107), (55, 1 << 107, 1 << 108)):
        for j in range(-96, 97):
            roots = [1]  # odd M with M^2 + j = 0 modulo 2^k, k growing to bits
            for k in range(3, bits + 1):
                step = 1 << (k - 2)
                roots = {m for r in (roots if k > 3 else (1, 3, 5, 7)) for m in
                         ((r, r + step, r + 2 * step, r + 3 * step) if k > 3 else (r,))
                         if (m * m + j) % (1 << k) == 0 and m < (1 << k)}
                if not roots:
                    break
            for r in roots:
                for m in range(r, 1 << 55, 1 << bits):
                    x = m * m + j
                    if (1 << 53) < m < (1 << 54) and lo <= x < hi:
                        assert x % (1 << bits) == 0
                        found.append(x / 2.0 ** 106)  # exact: 53 bits
    return sorted(set(found))


PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "cbm_tile.cuh"
using namespace cbm;
typedef unsigned long long u64;
__device__ u64 g_bad[8];
__device__ u64 g_first[8];
__device__ int g_eps;      // largest |1 - d inv| seen, in quarters of 2^-53
__device__ float g_approx; // largest relative error of the hardware's approximation

__device__ u64 mix(u64 z) {  // splitmix64
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
__device__ void check(int what, bool ok, u64 which) {
  if (!ok && atomicAdd(&g_bad[what], 1ull) == 0) g_first[what] = which;
}
__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }
__device__ bool same(double a, double b) {
  return __double_as_longlong(a) == __double_as_longlong(b);
}

// every Float32 of the range: root of squared distances, reciprocal of distances
__global__ void roots32(unsigned lo, unsigned hi) {
  for (unsigned i = lo + blockIdx.x * blockDim.x + threadIdx.x; i < hi; i += gridDim.x * blockDim.x)
    check(0, same(sqrt_mid(__uint_as_float(i)), __fsqrt_rn(__uint_as_float(i))), i);
}
__global__ void reciprocals32(unsigned lo, unsigned hi) {
  for (unsigned i = lo + blockIdx.x * blockDim.x + threadIdx.x; i < hi; i += gridDim.x * blockDim.x) {
    const float b = __uint_as_float(i);
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
    y = __fmaf_rn(__fmaf_rn(-b, y, 1.f), y, y);
    check(1, same(y, __frcp_rn(b)), i);
  }
}
// quotients by every significand: random numerators, and numerators whose
// quotient is next to a midpoint of two numbers
__global__ void quotients32(int rounds) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < 1u << 23; i += gridDim.x * blockDim.x) {
    const float b = __uint_as_float(0x3f800000u | i);
    for (int r = 0; r < rounds; ++r) {
      const u64 z = mix((u64)i * 1024 + r);
      const float any = __uint_as_float(0x3f800000u | (unsigned)(z & 0x7fffff));
      const double mid = (double)any + ldexp(1.0, -24);
      const float at = __double2float_rn(mid * (double)b);
      const float a[4] = {any, at, __uint_as_float(__float_as_uint(at) + 1),
                          __uint_as_float(__float_as_uint(at) - 1)};
      for (int k = 0; k < 4; ++k) check(2, same(div_mid(a[k], b), __fdiv_rn(a[k], b)), i);
    }
    for (int n = 0; n < 32; ++n) {
      if (i >= (1u << 23) - 16) {  // both near the top of their binade
        const float a = __uint_as_float(0x407fffffu - n);
        check(2, same(div_mid(a, b), __fdiv_rn(a, b)), i);
      }
    }
  }
}

__device__ void root64(double x, double* d, double* inv, u64 which) {
  *d = sqrt_mid(x, inv);
  check(3, same(*d, __dsqrt_rn(x)), which);
  const int eps = (int)ceil(fabs(__fma_rn(-*d, *inv, 1.0)) * 4.0 * 9007199254740992.0);
  if (eps > g_eps) atomicMax(&g_eps, eps);
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const float rel = (float)fabs(__fma_rn(-y * y, x, 1.0)) * 0.5f;
  if (rel > g_approx) atomicMax((int*)&g_approx, __float_as_int(rel));
}
__device__ void quotient64(double a, double x, double d, double inv, u64 which) {
  if (mid_root(x)) check(4, same(div_mid(a, d, inv), __ddiv_rn(a, d)), which);
}
__global__ void random64(int rounds) {
  const u64 t = (u64)blockIdx.x * blockDim.x + threadIdx.x;
  for (int r = 0; r < rounds; ++r) {
    const u64 z = mix(t * rounds + r), w = mix(~z);
    const int e = (int)(w % 80) - 40;  // 1e-12 .. 1e12
    double x = ldexp(__longlong_as_double(0x3ff0000000000000ll | (long long)(z >> 12)), e);
    double d, inv;
    root64(x, &d, &inv, z);
    const double any = __longlong_as_double(0x3ff0000000000000ll | (long long)(w >> 12));
    quotient64(any, x, d, inv, z);
    quotient64(-any, x, d, inv, z);
    // a numerator whose quotient is next to a midpoint
    const double at = __fma_rn(any, d, d * 1.1102230246251565e-16);
    quotient64(at, x, d, inv, z);
    quotient64(__longlong_as_double(__double_as_longlong(at) + 1), x, d, inv, z);
    quotient64(__longlong_as_double(__double_as_longlong(at) - 1), x, d, inv, z);
    // a root next to a midpoint
    x = __fma_rn(any, any, any * 2.220446049250313e-16);
    root64(x, &d, &inv, z);
    // the approximation looks at the upper word alone: all of them, two exponents
    if (r == 0 && t < 1ull << 21)
      root64(__longlong_as_double(0x3ff0000000000000ll + (long long)(t << 32)), &d, &inv, t);
  }
}
// the finitely many cases that the proof leaves, at every even exponent of the range
__global__ void hard64(const double* x, int n) {
  for (int i = threadIdx.x; i < n; i += blockDim.x)
    for (int e = -40; e <= 40; e += 2) {
      double d, inv;
      root64(ldexp(x[i], e), &d, &inv, i);
    }
  // divisors 2 - k 2^-52, whose reciprocals are nearest to midpoints, from
  // every x that has them as its root
  const int k = threadIdx.x;
  if (k < 1 || k > 64) return;
  const double top = 2.0 - k * ldexp(1.0, -52);
  const double around = __dmul_rn(top, top);
  for (int o = -4; o <= 4; ++o)
    for (int e = -40; e <= 38; e += 2) {
      const double xs = ldexp(__longlong_as_double(__double_as_longlong(around) + o), e);
      double d, inv;
      root64(xs, &d, &inv, k);
      if (d != ldexp(top, e / 2)) continue;
      if (k == 1) check(5, !mid_root(xs), k);
      else check(5, same(div_mid(1.0, d, inv), __drcp_rn(d)), k);
      for (int j = 0; j < 256; ++j) {
        quotient64(4.0 - j * ldexp(1.0, -51), xs, d, inv, k);
        quotient64(2.0 + j * ldexp(1.0, -51), xs, d, inv, k);
        quotient64(2.0 - j * ldexp(1.0, -52), xs, d, inv, k);
      }
    }
}

// the terms of four partners against one by one
template <typename T>
__global__ void terms(int what, int rounds) {
  using V4 = typename V4T<T>::type;
  const u64 t = (u64)blockIdx.x * blockDim.x + threadIdx.x;
  for (int r = 0; r < rounds; ++r) {
    u64 z = mix(t * rounds + r);
    auto u = [&]() { z = mix(z); return (double)(z >> 11) * 1.1102230246251565e-16; };
    const double scale = exp2(12.0 * u() - 10.0), k1 = exp2(20.0 * u() - 10.0), k2 = exp2(20.0 * u() - 10.0);
    const T rrep = (T)(scale * (0.2 + 0.8 * u())), ratt = (T)(scale * (u() < 0.2 ? 0.1 : 1.0 + u()));
    const bool from_rep = u() < 0.5;
    const T cut = rrep > ratt ? rrep : ratt;
    PairCoef<T> c;
    c.cut2 = (T)((double)cut * cut * (1.0 + 3e-5));
    c.rrep = rrep;
    c.ratt = ratt;
    c.krep = (T)(u() < 0.1 ? 0.0 : k1);
    c.katt = (T)(u() < 0.1 ? 0.0 : k2);
    c.from_rep = from_rep;
    const PairLine<T> line = make_pair_line<T>(c.cut2, c.krep, c.rrep, c.katt, c.ratt, from_rep);
    T xi[3], a[3], b[3];
    V4 v[4];
    int q[4];
    for (int d = 0; d < 3; ++d) {
      xi[d] = (T)(100.0 * scale * u());
      a[d] = b[d] = (T)0;
    }
    for (int k = 0; k < 4; ++k) {
      V4 p;
      const double s = u() < 0.1 ? 1e-3 * scale : scale * 1.3;
      p.x = xi[0] + (T)(s * (2.0 * u() - 1.0));
      p.y = xi[1] + (T)(s * (2.0 * u() - 1.0));
      p.z = xi[2] + (T)(s * (2.0 * u() - 1.0));
      p.w = (T)0;
      q[k] = u() < 0.1 ? 7 : k;
      if (q[k] == 7) { p.x = xi[0]; p.y = xi[1]; p.z = xi[2]; }
      v[k] = p;
    }
    const int in = pair_terms4<T>(c, line, line.mid, xi, v, 7, q, a);
    int ref = 0;
    for (int k = 0; k < 4; ++k)
      if (q[k] != 7) {
        T xj[3], e[3];
        to3<T>(v[k], xj);
        const T s2 = pair_diff<T, 3>(xi, xj, e);
        if (pair_term<T, 3>(c, e, s2, b)) ref |= 1 << k;
      }
    check(what, in == ref && same(a[0], b[0]) && same(a[1], b[1]) && same(a[2], b[2]), t);
  }
}

int main() {
  const std::vector<double> hard = {HARD};
  double* x = nullptr;
  if (cudaMalloc(&x, hard.size() * 8) != cudaSuccess) return 2;
  cudaMemcpy(x, hard.data(), hard.size() * 8, cudaMemcpyHostToDevice);
  const float lo2 = 1e-12f, hi2 = 1e12f, lo = 1e-6f, hi = 1e6f;
  auto bits = [](float v) { unsigned u; memcpy(&u, &v, 4); return u; };
  roots32<<<148 * 8, 256>>>(bits(lo2), bits(hi2) + 1);
  reciprocals32<<<148 * 8, 256>>>(bits(lo), bits(hi) + 1);
  quotients32<<<148 * 8, 256>>>(32);
  random64<<<8192, 256>>>(128);
  hard64<<<1, 256>>>(x, (int)hard.size());
  terms<float><<<8192, 256>>>(6, 64);
  terms<double><<<8192, 256>>>(7, 64);
  u64 bad[8], first[8];
  int eps = 0;
  float approx = 0;
  if (cudaDeviceSynchronize() != cudaSuccess) return 2;
  cudaMemcpyFromSymbol(bad, g_bad, sizeof bad);
  cudaMemcpyFromSymbol(first, g_first, sizeof first);
  cudaMemcpyFromSymbol(&eps, g_eps, 4);
  cudaMemcpyFromSymbol(&approx, g_approx, 4);
  const char* name[] = {"roots f32", "reciprocals f32", "quotients f32", "roots f64", "quotients f64",
                        "hard reciprocals f64", "terms f32", "terms f64"};
  int rc = 0;
  for (int k = 0; k < 8; ++k) {
    if (bad[k]) rc = 1;
    std::printf("%s: %llu differ (first %llu)\n", name[k], bad[k], first[k]);
  }
  // what the proof takes of the approximation and of the inverse root
  std::printf("approximation %g, inverse root %g u, hard roots %zu\n", approx, eps / 4.0, hard.size());
  if (!(approx < 3.8e-6f) || eps > 14 || hard.empty()) rc = 1;
  return rc;
}
"""


def test_mid_operations_are_the_general_ones(gpu_lib, tmp_path):
    spec = importlib.util.spec_from_file_location("cbm_build", os.path.join(PKG, "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    src, exe = tmp_path / "mid.cu", tmp_path / "mid"
    hard = ", ".join(float.hex(x) for x in hard_roots())
    src.write_text("#include <cstring>\n" + PROGRAM.replace("{HARD}", "{" + hard + "}"))
    subprocess.run([build._nvcc(), *build.FLAGS, "-I", os.path.join(PKG, "csrc"), "-o", str(exe),
                    str(src)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    print(out.stdout)
    assert out.returncode == 0, out.stdout
