// cbm_stencil_vec.cuh — 3D medium stencils on 16-byte vectors of nodes.
//
// A thread owns one vector of nodes along x (four Float32, two Float64) and
// marches a run of planes along z with the planes below, at and above it in
// registers; the rows y - 1 and y + 1 and the two nodes beside the vector are
// loads that its block's other threads have brought into L1.  No shared
// memory and no barriers: a plane is five loads and one (FTCS) or three
// (gradient) vector stores a thread, so the kernels are bound by HBM instead
// of by the scalar shared-memory reads and the instructions of a tile.
// Threads are numbered along the plane, so any row length that is a whole
// number of vectors keeps every lane busy; blocks of 256 cover 1024 Float32
// nodes.  Six blocks an SM hide the loads (measured at 256^3 Float32, FTCS
// and gradient: 34 and 49 us with six, 42 and 53 with four, 35 and 58 with
// eight; planes staged in shared memory by TMA took 50 and 52; HBM alone 21
// and 41).
//
// Same expressions as k_medium_grad / k_medium_de: lap = (l_x + l_y) + l_z,
// the DE reading medium_in() of every value, the divisions by dx^2 and 2 dx
// as over_dx2 / over_2dx.
#pragma once
#include "cbm_kernels.cuh"

namespace cbm {

template <typename T>
struct NodeVec;
template <>
struct NodeVec<float> {
  using type = float4;
  static constexpr int n = 4;
};
template <>
struct NodeVec<double> {
  using type = double2;
  static constexpr int n = 2;
};

template <typename T>
__device__ __forceinline__ void vec_load(const T* p, T* v) {
  *reinterpret_cast<typename NodeVec<T>::type*>(v) =
      *reinterpret_cast<const typename NodeVec<T>::type*>(p);
}
template <typename T>
__device__ __forceinline__ void vec_store(T* p, const T* v) {
  *reinterpret_cast<typename NodeVec<T>::type*>(p) =
      *reinterpret_cast<const typename NodeVec<T>::type*>(v);
}

template <typename T>
__device__ __forceinline__ void vec_store_cs(T* p, const T* v) {
  __stcs(reinterpret_cast<typename NodeVec<T>::type*>(p),
         *reinterpret_cast<const typename NodeVec<T>::type*>(v));
}

template <typename T, bool kDE, bool kScale>
__device__ __forceinline__ void stencil_3d_vec(const Params<T>& P, int z_run) {
  constexpr int V = NodeVec<T>::n;
  const int nx = P.n_medium[0], ny = P.n_medium[1], nz = P.n_medium[2];
  const int row = nx / V;
  const int plane = nx * ny;
  const int t = blockIdx.x * kTile + threadIdx.x;
  if (t >= row * ny) return;
  const int y = t / row, x = (t - y * row) * V;
  const int za = blockIdx.y * z_run;
  const int zb = za + z_run < nz ? za + z_run : nz;
  const bool iny = y > 0 && y < ny - 1;
  const int o = y * nx + x;  // in the plane
  const int left = x > 0 ? o - 1 : o, right = x + V < nx ? o + V : o;
  const int up = iny ? o + nx : o, down = iny ? o - nx : o;
  const T* const c = P.c_cur;
  auto in_val = [&](T v) { return kDE ? medium_in(P, v) : v; };
  alignas(16) T lo[V], mid[V], hi[V];
  const T* p = c + (size_t)za * plane;  // plane z
  vec_load(p + (za > 0 ? o - plane : o), lo);
  vec_load(p + o, mid);
#pragma unroll
  for (int k = 0; k < V; ++k) {
    lo[k] = in_val(lo[k]);
    mid[k] = in_val(mid[k]);
  }
  for (int z = za; z < zb; ++z, p += plane) {
    alignas(16) T yu[V], yd[V], out[V];
    vec_load(p + (z < nz - 1 ? o + plane : o), hi);
    vec_load(p + up, yu);
    vec_load(p + down, yd);
    const T xl = in_val(p[left]), xr = in_val(p[right]);
#pragma unroll
    for (int k = 0; k < V; ++k) {
      hi[k] = in_val(hi[k]);
      yu[k] = in_val(yu[k]);
      yd[k] = in_val(yd[k]);
    }
    const bool inyz = iny && z > 0 && z < nz - 1;
    const size_t at = (size_t)z * plane + o;
    if (kDE) {
#pragma unroll
      for (int k = 0; k < V; ++k) {
        const T u = mid[k];
        const T l0 = over_dx2<kScale>(P, 0, ((k < V - 1 ? mid[k + 1 < V ? k + 1 : k] : xr) - (T)2 * u) +
                                                (k > 0 ? mid[k > 0 ? k - 1 : 0] : xl));
        const T l1 = over_dx2<kScale>(P, 1, (yu[k] - (T)2 * u) + yd[k]);
        const T l2 = over_dx2<kScale>(P, 2, (hi[k] - (T)2 * u) + lo[k]);
        const T lap = (l0 + l1) + l2;
        const T kk = P.diff_D * lap - P.decay * u;
        const bool in = inyz && x + k > 0 && x + k < nx - 1;
        out[k] = in ? u + P.dt * kk : u;
      }
      vec_store(P.c_nxt + at, out);
    } else {
      alignas(16) T gy[V], gz[V];
#pragma unroll
      for (int k = 0; k < V; ++k) {
        const bool in = inyz && x + k > 0 && x + k < nx - 1;
        const T r = k < V - 1 ? mid[k + 1 < V ? k + 1 : k] : xr;
        const T l = k > 0 ? mid[k > 0 ? k - 1 : 0] : xl;
        out[k] = in ? over_2dx<kScale>(P, 0, r - l) : (T)0;
        gy[k] = in ? over_2dx<kScale>(P, 1, yu[k] - yd[k]) : (T)0;
        gz[k] = in ? over_2dx<kScale>(P, 2, hi[k] - lo[k]) : (T)0;
      }
      // streamed past the field, which the exchange and the FTCS read next
      vec_store_cs(P.grad_nxt[0] + at, out);
      vec_store_cs(P.grad_nxt[1] + at, gy);
      vec_store_cs(P.grad_nxt[2] + at, gz);
    }
#pragma unroll
    for (int k = 0; k < V; ++k) {
      lo[k] = mid[k];
      mid[k] = hi[k];
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(kTile, 6) k_medium_grad_3d_vec(Params<T> P, int z_run) {
  if (P.exact_scale) stencil_3d_vec<T, false, true>(P, z_run);
  else stencil_3d_vec<T, false, false>(P, z_run);
}

template <typename T>
__global__ void __launch_bounds__(kTile, 6) k_medium_de_3d_vec(Params<T> P, int z_run) {
  if (P.exact_scale) stencil_3d_vec<T, true, true>(P, z_run);
  else stencil_3d_vec<T, true, false>(P, z_run);
}

}  // namespace cbm
