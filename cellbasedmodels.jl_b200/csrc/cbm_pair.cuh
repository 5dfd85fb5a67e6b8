// cbm_pair.cuh — soft-sphere pair terms of several partners at once, without
// branches (Float32).
#pragma once
#include "cbm_common.cuh"

namespace cbm {

// Packed pairs of float operations (sm_100 f32x2): one instruction, and per
// element the same IEEE rounding as the scalar operation.
__device__ __forceinline__ float2 f2_sub(float2 a, float2 b) {
  unsigned long long r;
  asm("sub.rn.f32x2 %0, %1, %2;"
      : "=l"(r)
      : "l"(*reinterpret_cast<unsigned long long*>(&a)),
        "l"(*reinterpret_cast<unsigned long long*>(&b)));
  return *reinterpret_cast<float2*>(&r);
}
__device__ __forceinline__ float2 f2_mul(float2 a, float2 b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;"
      : "=l"(r)
      : "l"(*reinterpret_cast<unsigned long long*>(&a)),
        "l"(*reinterpret_cast<unsigned long long*>(&b)));
  return *reinterpret_cast<float2*>(&r);
}

__device__ __forceinline__ float2 f2_add(float2 a, float2 b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;"
      : "=l"(r)
      : "l"(*reinterpret_cast<unsigned long long*>(&a)),
        "l"(*reinterpret_cast<unsigned long long*>(&b)));
  return *reinterpret_cast<float2*>(&r);
}

__device__ __forceinline__ float2 f2_fma(float2 a, float2 b, float2 c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(r)
      : "l"(*reinterpret_cast<unsigned long long*>(&a)),
        "l"(*reinterpret_cast<unsigned long long*>(&b)),
        "l"(*reinterpret_cast<unsigned long long*>(&c)));
  return *reinterpret_cast<float2*>(&r);
}

// Coefficients of the pair term in a form without branches: base and
// stiffness are selected, and every pair beyond the cutoff, or the agent
// itself, adds a zero.  In Float32 all of it is kept negated (-d^2, -d), which
// leaves no negations between the packed operations.
template <typename T>
struct PairLine {
  T nfar2, nreach, nrrep, krep, katt, rrep, abase;
  bool mid;  // the stiffnesses are far from the ends of the exponent range
};
// cut2: a squared distance of cut2 is a distance >= the cutoff for certain.
// -(a (d - r)) and a (r - d) are the same number; so are -(a (c - d)) and
// (-a) (c - d).
template <typename T>
__device__ __forceinline__ PairLine<T> make_pair_line(T cut2, T k_rep, T r_rep, T k_att, T r_att,
                                                      bool from_rep) {
  auto mid = [](T k) { return k == (T)0 || (fabs(k) > (T)1e-12 && fabs(k) < (T)1e12); };
  return PairLine<T>{-cut2, -(r_rep > r_att ? r_rep : r_att), -r_rep, k_rep,
                     from_rep ? k_att : -k_att, r_rep, from_rep ? r_rep : r_att,
                     mid(k_rep) && mid(k_att)};
}

// The terms of four partners at positions v, added to acc in order; an entry
// with none[u] adds nothing.  Returns the entries that lie within the cutoff
// (bit u), or -1, with acc as it was, for distances that need the general
// square root and quotient (coincident agents; with kFar also infinities, NaN
// and distances above 1e6).  L.mid must hold.  Square root and quotient are
// sqrt_mid and div_mid on pairs of values.
template <bool kFar>
__device__ __forceinline__ int pair_terms4_mid(const PairLine<float>& L, const float* xi,
                                                const float4* v, const bool* none, float* acc) {
  const float2 ixy = make_float2(xi[0], xi[1]);
  float2 exy[4], n2[2];
  float ez[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    exy[u] = f2_sub(ixy, make_float2(v[u].x, v[u].y));
    ez[u] = xi[2] - v[u].z;
    const float2 q = f2_mul(exy[u], exy[u]);
    const float n = (-q.x - q.y) - ez[u] * ez[u];
    (u & 1 ? n2[u >> 1].y : n2[u >> 1].x) = none[u] ? L.nfar2 : n;
  }
  if (!(fmaxf(fmaxf(n2[0].x, n2[0].y), fmaxf(n2[1].x, n2[1].y)) < -1e-12f)) return -1;
  // (a NaN fails the sum's test, and none's own difference is not looked at)
  if (kFar && !((n2[0].x + n2[0].y) + (n2[1].x + n2[1].y) > -1e12f)) return -1;
  int in = 0;
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    const float2 x = n2[p], half = make_float2(0.5f, 0.5f);
    float2 y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y.x) : "f"(-x.x));
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y.y) : "f"(-x.y));
    float2 g = f2_mul(x, y), h = f2_mul(half, y);
    const float2 r = f2_fma(g, h, half);
    g = f2_fma(g, r, g);
    h = f2_fma(h, r, h);
    const float2 d = f2_fma(f2_fma(g, g, x), h, g);  // minus the distances
    const bool r0 = d.x > L.nrrep, r1 = d.y > L.nrrep;
    const float2 k = make_float2(r0 ? L.krep : L.katt, r1 ? L.krep : L.katt);
    const float2 b = make_float2(r0 ? L.rrep : L.abase, r1 ? L.rrep : L.abase);
    const float2 F = f2_mul(k, f2_add(b, d));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y.x) : "f"(-d.x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y.y) : "f"(-d.y));
    y = f2_fma(y, f2_fma(d, y, make_float2(1.f, 1.f)), y);
    float2 q = f2_mul(F, y);
    q = f2_fma(f2_fma(d, q, F), y, q);
    const bool i0 = d.x > L.nreach, i1 = d.y > L.nreach;
    in |= (i0 ? 1 << 2 * p : 0) | (i1 ? 2 << 2 * p : 0);
    const float c0 = i0 ? q.x : 0.f, c1 = i1 ? q.y : 0.f;
    const float2 t0 = f2_mul(make_float2(c0, c0), exy[2 * p]);
    const float2 t1 = f2_mul(make_float2(c1, c1), exy[2 * p + 1]);
    // scalar sums: a packed product and a packed sum came out fused
    acc[0] = (acc[0] + t0.x) + t1.x;
    acc[1] = (acc[1] + t0.y) + t1.y;
    acc[2] = (acc[2] + c0 * ez[2 * p]) + c1 * ez[2 * p + 1];
  }
  return in;
}

}  // namespace cbm
