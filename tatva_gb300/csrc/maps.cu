// Operator maps: eval / grad / integration weights / integrate / deterministic sums /
// gather and the reverse-mode transposes (K1-K3).
//
// Reference semantics (tatva/operator.py):
//   eval                     :358-377  out[e,q,v]   = sum_a N_a(xi_q) u[conn[e,a], v]
//   grad                     :379-397  out[e,q,v,d] = sum_a dN_a/dx_d u[conn[e,a], v]
//   get_integration_weights  :172-192  out[e,q]     = detJ(e,q) * w_q
//   _integrate_quad_array    :344-356  out[e,v]     = sum_q quad[e,q,v] w[e,q]
//   integrate                :307-319  sum over elements
#include "tg_common.cuh"
#include "tg_dispatch.cuh"
#include "tg_hex.cuh"

namespace tg {

constexpr int TPB_T = 256;

// ------------------------------------------------------------------ 32-byte access
// A thread per element writes (reads) its element's values as one contiguous run.  In
// 4-byte accesses a warp touches 32 cache lines per instruction; 32-byte accesses are whole
// memory sectors, so the runs cost no more L2 transactions than coalesced rows would.
__device__ __forceinline__ void st32(float* p, const float* v) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0]),
               "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
               : "memory");
}
__device__ __forceinline__ void st32(double* p, const double* v) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(v[0]), "d"(v[1]),
               "d"(v[2]), "d"(v[3])
               : "memory");
}
__device__ __forceinline__ void ld32(const float* p, float* v) {
  asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]),
                 "=f"(v[6]), "=f"(v[7])
               : "l"(p));
}
__device__ __forceinline__ void ld32(const double* p, double* v) {
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
               : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3])
               : "l"(p));
}
// N consecutive values (N a multiple of 32 bytes); VEC: p is 32-byte aligned
template <bool VEC, int N, class T>
__device__ __forceinline__ void store_run(T* p, const T (&v)[N]) {
  if constexpr (VEC) {
    constexpr int W = 32 / sizeof(T);
    static_assert(N % W == 0, "whole 32-byte words");
#pragma unroll
    for (int k = 0; k < N; k += W) st32(p + k, v + k);
  } else {
#pragma unroll
    for (int k = 0; k < N; ++k) p[k] = v[k];
  }
}
template <bool VEC, int N, class T>
__device__ __forceinline__ void load_run(const T* p, T (&v)[N]) {
  if constexpr (VEC) {
    constexpr int W = 32 / sizeof(T);
    static_assert(N % W == 0, "whole 32-byte words");
#pragma unroll
    for (int k = 0; k < N; k += W) ld32(p + k, v + k);
  } else {
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = p[k];
  }
}

// Whether a value is infinite or NaN, on its bits (FP64: without the FP64 pipe).  The forms
// that subtract a corner's value first turn one infinite nodal value into NaN all over its
// element, and overflow from an eighth of the largest number on; an element with such a result
// is done again as the weighted sum that defines it.
__device__ __forceinline__ unsigned magnitude_bits(float v) {
  return __float_as_uint(v) & 0x7fffffffu;
}
__device__ __forceinline__ unsigned magnitude_bits(double v) {
  return (unsigned)__double2hiint(v) & 0x7fffffffu;
}
template <int N, class T>
__device__ __forceinline__ bool any_nonfinite(const T (&v)[N]) {
  unsigned m = 0;
#pragma unroll
  for (int k = 0; k < N; ++k) m = max(m, magnitude_bits(v[k]));
  return m >= (sizeof(T) == 4 ? 0x7f800000u : 0x7ff00000u);
}

// ------------------------------------------------------------------ eval
template <int ET, class T>
__global__ void eval_kernel(const T* __restrict__ nodal, int V, const int32_t* __restrict__ conn,
                            int64_t n_elems, T* __restrict__ out) {
  using E = Elem<ET>;
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t total = n_elems * E::Q * V;
  if (tid >= total) return;
  const int v = (int)(tid % V);
  const int64_t eq = tid / V;
  const int q = (int)(eq % E::Q);
  const int64_t e = eq / E::Q;
  T acc = T(0);
#pragma unroll
  for (int a = 0; a < E::NN; ++a) {
    const int64_t n = __ldg(conn + e * E::NN + a);
    acc += E::template N<T>(q, a) * nodal[n * V + v];
  }
  out[tid] = acc;
}

// ------------------------------------------------------------------ gather coords
template <int ET, class T>
__device__ __forceinline__ void gather_coords(const T* __restrict__ coords,
                                              const int32_t* __restrict__ conn, int64_t e,
                                              T (&X)[Elem<ET>::NN][Elem<ET>::D],
                                              int (&nid)[Elem<ET>::NN]) {
  using E = Elem<ET>;
#pragma unroll
  for (int a = 0; a < E::NN; ++a) {
    nid[a] = __ldg(conn + e * E::NN + a);
#pragma unroll
    for (int d = 0; d < E::D; ++d) X[a][d] = coords[(int64_t)nid[a] * E::D + d];
  }
}

// ------------------------------------------------------------------ simplex grad
// A warp's 32 element runs of N values each, moved between the lanes (a run per lane) and
// memory (32 consecutive values per instruction) through shared memory; odd row stride.
// n_here: elements of the warp that exist.
constexpr int SIMPLEX_THREADS = 128;
template <int N>
constexpr int run_stride() { return N | 1; }
template <int N, class T>
__device__ __forceinline__ void warp_store_runs(T* __restrict__ dst, T* tile, const T (&v)[N],
                                                int n_here) {
  const int lane = threadIdx.x & 31;
  __syncwarp();
#pragma unroll
  for (int i = 0; i < N; ++i) tile[lane * run_stride<N>() + i] = v[i];
  __syncwarp();
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int k = i * 32 + lane, row = k / N;
    if (row < n_here) dst[k] = tile[row * run_stride<N>() + (k - row * N)];
  }
}
template <int N, class T>
__device__ __forceinline__ void warp_load_runs(const T* __restrict__ src, T* tile, T (&v)[N],
                                               int n_here) {
  const int lane = threadIdx.x & 31;
  __syncwarp();
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int k = i * 32 + lane, row = k / N;
    if (row < n_here) tile[row * run_stride<N>() + (k - row * N)] = __ldg(src + k);
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = tile[lane * run_stride<N>() + i];
}

// Tri3 / Tet4: thread per element through the edge vectors from node 0 (gradient = R D f,
// D_k f = f_{k+1} - f_0, R the inverse of the coordinates' D).  NV = V in {1, 2, 3}; NV = 0:
// any V, a component at a time.  FP64 is bound by the FP64 pipe (about 95 operations for
// V = 3), FP32 by memory.  A result that is not finite is done again as the sum over the nodes
// (sum_a G_a f_a, with G_0 = -sum_k R_k): in the differences an infinite f_0 is in every term.
template <int ET, class T>
__device__ __forceinline__ void simplex_inverse(const T* __restrict__ coords,
                                                const int32_t* __restrict__ conn, int64_t e,
                                                int (&nid)[Elem<ET>::NN],
                                                T (&R)[Elem<ET>::D][Elem<ET>::D]) {
  constexpr int D = Elem<ET>::D;
  T X[Elem<ET>::NN][D], J[D][D];
  gather_coords<ET, T>(coords, conn, e, X, nid);
#pragma unroll
  for (int k = 0; k < D; ++k)
#pragma unroll
    for (int d = 0; d < D; ++d) J[k][d] = X[k + 1][d] - X[0][d];
  invD<T, D>(J, R);
}

// the gradient of one component as the sum over the nodes (not inlined: the compiler would run
// it for every element, FP64 Tri3 46 -> 74 us)
template <class T, int D>
struct SimplexVec {
  T v[D];
};
template <int ET, class T>
__device__ __noinline__ SimplexVec<T, Elem<ET>::D> simplex_grad_nodal(
    const T* __restrict__ nodal, const T* __restrict__ coords, int V, int v,
    const int32_t* __restrict__ conn, int64_t e) {
  constexpr int D = Elem<ET>::D;
  int nid[Elem<ET>::NN];
  T R[D][D];
  simplex_inverse<ET, T>(coords, conn, e, nid, R);
  SimplexVec<T, D> g;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    T g0 = T(0);
#pragma unroll
    for (int k = 0; k < D; ++k) g0 -= R[d][k];
    g.v[d] = g0 * nodal[(int64_t)nid[0] * V + v];
#pragma unroll
    for (int k = 0; k < D; ++k) g.v[d] += R[d][k] * nodal[(int64_t)nid[k + 1] * V + v];
  }
  return g;
}
template <int ET, class T, int NV>
__global__ void __launch_bounds__(SIMPLEX_THREADS)
    simplex_grad_kernel(const T* __restrict__ nodal, const T* __restrict__ coords, int V,
                        const int32_t* __restrict__ conn, int64_t n_elems,
                        T* __restrict__ out) {
  using E = Elem<ET>;
  constexpr int NN = E::NN, D = E::D, N = (NV ? NV : 1) * D;
  __shared__ T tiles[NV ? SIMPLEX_THREADS / 32 * 32 * run_stride<N>() : 1];
  const int64_t e = (int64_t)blockIdx.x * SIMPLEX_THREADS + threadIdx.x;
  const int64_t e0 = e - (threadIdx.x & 31);
  if (e0 >= n_elems) return;  // whole warps
  const int64_t ec = e < n_elems ? e : n_elems - 1;
  int nid[NN];
  T R[D][D];
  simplex_inverse<ET, T>(coords, conn, ec, nid, R);
  auto gradient = [&](int v, T* o) {
    const T f0 = nodal[(int64_t)nid[0] * V + v];
    T g[D];
#pragma unroll
    for (int k = 0; k < D; ++k) {
      const T f = nodal[(int64_t)nid[k + 1] * V + v] - f0;
#pragma unroll
      for (int d = 0; d < D; ++d) g[d] = k == 0 ? R[d][0] * f : fma(R[d][k], f, g[d]);
    }
    if (any_nonfinite(g)) {
      const auto t = simplex_grad_nodal<ET, T>(nodal, coords, V, v, conn, ec);
#pragma unroll
      for (int d = 0; d < D; ++d) g[d] = t.v[d];
    }
#pragma unroll
    for (int d = 0; d < D; ++d) o[d] = g[d];
  };
  if constexpr (NV) {
    V = NV;
    T o[N];
#pragma unroll
    for (int v = 0; v < NV; ++v) gradient(v, o + v * D);
    warp_store_runs<N>(out + e0 * N, tiles + (threadIdx.x >> 5) * 32 * run_stride<N>(), o,
                       (int)(n_elems - e0 < 32 ? n_elems - e0 : 32));
  } else {
    if (e < n_elems)
      for (int v = 0; v < V; ++v) gradient(v, out + (e * V + v) * D);
  }
}

// ------------------------------------------------------------------ Hex8 maps
// Thread per element, in the modal form of tg_hex.cuh.  FP64 is bound by the FP64 pipe (the
// operation count), FP32 by the element-sized runs of quadrature values in memory: NV = V in
// {1, 2, 3} moves them in 32-byte accesses where the array is aligned (VEC); NV = 0 takes
// any V in groups of three components with 4- or 8-byte accesses.  The four points of a
// plane of constant xi3 share their reference gradients: df/dxi1 takes two values there,
// df/dxi2 two and df/dxi3 four.  FP32 holds both planes of an element (24 NV values) in
// registers, FP64 one at a time.
// Brick of 96 x 80 x 112, FP32, V = 3 (860,160 elements), against a point or a node per
// thread and 4-byte accesses: eval 125 -> 20 us (82 MB written, 5.2 TB/s with the gathers),
// grad 329 -> 65 us (248 MB, 4.2 TB/s), transpose of grad 156 -> 77 us for the elements, of
// eval 236 -> 21 us for the elements + 38 us for the nodes.  61 x 67 x 59 distorted, FP64,
// V = 1: grad 389 -> 263 us, its transpose 408 -> 282 us; with the adjugate instead of the
// inverse (one value: three products by the reciprocal determinant, not nine) 240 and 246.
template <int NV>
constexpr int hex_group() { return NV ? NV : 3; }
template <class T>
constexpr int hex_planes() { return sizeof(T) == 4 ? 2 : 1; }

// 8 df/dxi_i of C components at the points of plane sz: d0 by side of xi2, d1 by side of
// xi1, d2 by both
template <class T, int C>
struct HexPlane {
  T d0[2][C], d1[2][C], d2[2][2][C];
  __device__ __forceinline__ void set(const T (&m)[8][C], T sz) {
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const T a0 = fma(sz, m[5][c], m[1][c]), a1 = fma(sz, m[7][c], m[3][c]);
      d0[0][c] = a0 - a1;
      d0[1][c] = a0 + a1;
      const T b0 = fma(sz, m[6][c], m[2][c]), b1 = fma(sz, m[7][c], m[3][c]);
      d1[0][c] = b0 - b1;
      d1[1][c] = b0 + b1;
      const T e0 = m[4][c] - m[5][c], e1 = m[4][c] + m[5][c];
      const T h0 = m[6][c] - m[7][c], h1 = m[6][c] + m[7][c];
      d2[0][0][c] = e0 - h0;
      d2[0][1][c] = e0 + h0;
      d2[1][0][c] = e1 - h1;
      d2[1][1][c] = e1 + h1;
    }
  }
  __device__ __forceinline__ void at(int p, T (&D)[3][C]) const {
    const int ix = (p == 1 || p == 2), iy = p >= 2;
#pragma unroll
    for (int c = 0; c < C; ++c) {
      D[0][c] = d0[iy][c];
      D[1][c] = d1[ix][c];
      D[2][c] = d2[ix][iy][c];
    }
  }
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int c = 0; c < C; ++c) {
      d0[0][c] = d0[1][c] = d1[0][c] = d1[1][c] = T(0);
      d2[0][0][c] = d2[0][1][c] = d2[1][0][c] = d2[1][1][c] = T(0);
    }
  }
  // adjoint of at: adds F to the plane's values
  __device__ __forceinline__ void add(int p, int c, T f0, T f1, T f2) {
    const int ix = (p == 1 || p == 2), iy = p >= 2;
    d0[iy][c] += f0;
    d1[ix][c] += f1;
    d2[ix][iy][c] += f2;
  }
  // adjoint of set: adds the plane's values to the scaled-mode weights
  __device__ __forceinline__ void fold(T (&w)[8][C], T sz) const {
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const T s0 = d0[1][c] + d0[0][c], t0 = d0[1][c] - d0[0][c];
      const T s1 = d1[1][c] + d1[0][c], t1 = d1[1][c] - d1[0][c];
      const T e0 = d2[0][0][c] + d2[0][1][c], e1 = d2[1][0][c] + d2[1][1][c];
      const T h0 = d2[0][1][c] - d2[0][0][c], h1 = d2[1][1][c] - d2[1][0][c];
      const T t = t0 + t1;
      w[1][c] += s0;
      w[2][c] += s1;
      w[3][c] += t;
      w[4][c] += e0 + e1;
      w[5][c] += fma(sz, s0, e1 - e0);
      w[6][c] += fma(sz, s1, h0 + h1);
      w[7][c] += fma(sz, t, h1 - h0);
    }
  }
};

// the geometry of an element: scaled coordinate modes and, for a parallelepiped (bitwise
// what the per-point evaluation gives), its one inverse
template <class T, bool UNSCALED>
struct HexGeometry {
  T mx[8][3], R[3][3], r;
  bool constant;
  // R: the inverse, or, UNSCALED, the adjugate, and r: the reciprocal determinant
  __device__ __forceinline__ void invert(const T (&J)[3][3]) {
    if constexpr (UNSCALED) r = T(1) / adjugate3(J, R);
    else inv3(J, R);
  }
  __device__ __forceinline__ T scaled(T v) const { return UNSCALED ? v * r : v; }
  __device__ __forceinline__ void load(const T* __restrict__ coords,
                                       const int32_t* __restrict__ conn, int64_t e,
                                       int (&nid)[8]) {
    gather_coords<TG_HEX8, T>(coords, conn, e, mx, nid);
    hex_modes8<T, 3>(mx);
    hex_scale_gauss<T, 3>(mx);
    constant = hex_constant_jacobian(mx);
    if (constant) {
      const T J[3][3] = {{mx[1][0], mx[1][1], mx[1][2]},
                         {mx[2][0], mx[2][1], mx[2][2]},
                         {mx[4][0], mx[4][1], mx[4][2]}};
      invert(J);
    }
  }
  __device__ __forceinline__ void plane(HexPlane<T, 3>& jx, T sz) const {
    if (!constant) jx.set(mx, sz);
  }
  __device__ __forceinline__ void at(const HexPlane<T, 3>& jx, int p) {
    if (!constant) {
      T J[3][3];
      jx.at(p, J);
      invert(J);
    }
  }
};

template <class T, int NV>
__device__ __forceinline__ void hex_load_values(const T* __restrict__ nodal, int V, int v0, int nv,
                                                const int (&nid)[8], T (&m)[8][hex_group<NV>()]) {
#pragma unroll
  for (int a = 0; a < 8; ++a)
#pragma unroll
    for (int k = 0; k < hex_group<NV>(); ++k)
      m[a][k] = (NV || k < nv) ? nodal[(int64_t)nid[a] * V + v0 + k] : T(0);
}

// out[e, q, v, d] = sum_i R[d][i] 8 dU_v/dxi_i
template <class T, int NV, bool VEC>
__global__ void __launch_bounds__(128) hex_grad_kernel(const T* __restrict__ nodal,
                                                       const T* __restrict__ coords, int V,
                                                       const int32_t* __restrict__ conn,
                                                       int64_t n_elems, T* __restrict__ out) {
  constexpr int G = hex_group<NV>(), NP = hex_planes<T>();
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n_elems) return;
  HexGeometry<T, NV == 1> geo;
  int nid[8];
  geo.load(coords, conn, e, nid);
  if (NV) V = NV;
  for (int v0 = 0; v0 < V; v0 += G) {
    const int nv = (V - v0) < G ? (V - v0) : G;
    T mu[8][G];
    hex_load_values<T, NV>(nodal, V, v0, nv, nid, mu);
    hex_modes8<T, G>(mu);
    hex_scale_gauss<T, G>(mu);
#pragma unroll 1
    for (int z0 = 0; z0 < 2; z0 += NP) {
      T o[NP * 12 * G];
#pragma unroll
      for (int z = 0; z < NP; ++z) {
        const T sz = (z0 + z) ? T(1) : T(-1);
        HexPlane<T, 3> jx;
        HexPlane<T, G> ju;
        geo.plane(jx, sz);
        ju.set(mu, sz);
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          geo.at(jx, p);
          T H[3][G];
          ju.at(p, H);
#pragma unroll
          for (int k = 0; k < G; ++k)
#pragma unroll
            for (int d = 0; d < 3; ++d)
              o[((z * 4 + p) * G + k) * 3 + d] =
                  geo.scaled(fma(geo.R[d][2], H[2][k],
                                 fma(geo.R[d][1], H[1][k], geo.R[d][0] * H[0][k])));
        }
      }
      T* dst = out + ((e * 8 + z0 * 4) * V + v0) * 3;
      if constexpr (NV) {
        store_run<VEC>(dst, o);
      } else {
#pragma unroll
        for (int p = 0; p < 4 * NP; ++p)
#pragma unroll
          for (int k = 0; k < 3 * G; ++k)
            if (k < 3 * nv) dst[p * 3 * V + k] = o[p * 3 * G + k];
      }
    }
  }
}

// contrib[e, a, v] = sum_q sum_d dN_a/dx_d flux[e, q, v, d]: the adjoint of hex_grad_kernel
template <class T, int NV, bool VEC>
__global__ void __launch_bounds__(128)
    hex_grad_transpose_elem_kernel(const T* __restrict__ flux, const T* __restrict__ coords,
                                   int V, const int32_t* __restrict__ conn, int64_t n_elems,
                                   T* __restrict__ contrib) {
  constexpr int G = hex_group<NV>(), NP = hex_planes<T>();
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n_elems) return;
  HexGeometry<T, NV == 1> geo;
  int nid[8];
  geo.load(coords, conn, e, nid);
  if (NV) V = NV;
  for (int v0 = 0; v0 < V; v0 += G) {
    const int nv = (V - v0) < G ? (V - v0) : G;
    T w[8][G];
#pragma unroll
    for (int m = 0; m < 8; ++m)
#pragma unroll
      for (int k = 0; k < G; ++k) w[m][k] = T(0);
#pragma unroll 1
    for (int z0 = 0; z0 < 2; z0 += NP) {
      T f[NP * 12 * G];
      const T* src = flux + ((e * 8 + z0 * 4) * V + v0) * 3;
      if constexpr (NV) {
        load_run<VEC>(src, f);
      } else {
#pragma unroll
        for (int p = 0; p < 4 * NP; ++p)
#pragma unroll
          for (int k = 0; k < 3 * G; ++k) f[p * 3 * G + k] = k < 3 * nv ? src[p * 3 * V + k] : T(0);
      }
#pragma unroll
      for (int z = 0; z < NP; ++z) {
        const T sz = (z0 + z) ? T(1) : T(-1);
        HexPlane<T, 3> jx;
        HexPlane<T, G> F;
        geo.plane(jx, sz);
        F.clear();
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          geo.at(jx, p);
#pragma unroll
          for (int k = 0; k < G; ++k) {
            const T* t = f + ((z * 4 + p) * G + k) * 3;
            T r[3];
#pragma unroll
            for (int i = 0; i < 3; ++i)
              r[i] = geo.scaled(
                  fma(geo.R[2][i], t[2], fma(geo.R[1][i], t[1], geo.R[0][i] * t[0])));
            F.add(p, k, r[0], r[1], r[2]);
          }
        }
        F.fold(w, sz);
      }
    }
    hex_scale_gauss<T, G>(w);
    hex_modes8_adjoint<T, G>(w);
    T* dst = contrib + e * 8 * V + v0;
    if constexpr (NV) {
      T o[8 * G];
#pragma unroll
      for (int a = 0; a < 8; ++a)
#pragma unroll
        for (int k = 0; k < G; ++k) o[a * G + k] = w[a][k];
      store_run<VEC>(dst, o);
    } else {
#pragma unroll
      for (int a = 0; a < 8; ++a)
#pragma unroll
        for (int k = 0; k < G; ++k)
          if (k < nv) dst[a * V + k] = w[a][k];
    }
  }
}

// modes of a field times g^|m| / 8, g = 1/sqrt(3): what evaluation at the Gauss points and
// its transpose have between their two butterflies (N_a(xi_q) = 1/8 sum_m g^|m| s_m(a) s_m(q))
template <class T, int C>
__device__ __forceinline__ void hex_scale_value(T (&m)[8][C]) {
  const T e = T(0.125), g = T(HEX_GAUSS) * T(0.125), g2 = T(1.0 / 24), g3 = g2 * T(HEX_GAUSS);
#pragma unroll
  for (int c = 0; c < C; ++c) {
    m[0][c] *= e;
    m[1][c] *= g;
    m[2][c] *= g;
    m[4][c] *= g;
    m[3][c] *= g2;
    m[5][c] *= g2;
    m[6][c] *= g2;
    m[7][c] *= g3;
  }
}

// the same sums as they are written: one element's components v0 .. v0 + nv - 1 of
// sum_a N_a(xi_q) u[conn[e, a]] and of sum_q N_a(xi_q) quad[e, q]
template <class T>
__device__ __noinline__ void hex_eval_weighted(const T* __restrict__ nodal, int V, int v0, int nv,
                                               const int32_t* __restrict__ conn, T* out) {
  for (int q = 0; q < 8; ++q)
    for (int k = 0; k < nv; ++k) {
      T s = T(0);
      for (int a = 0; a < 8; ++a)
        s += Elem<TG_HEX8>::N<T>(q, a) * nodal[(int64_t)conn[a] * V + v0 + k];
      out[q * V + k] = s;
    }
}
template <class T>
__device__ __noinline__ void hex_eval_transpose_weighted(const T* quad, int V, int nv, T* out) {
  for (int a = 0; a < 8; ++a)
    for (int k = 0; k < nv; ++k) {
      T s = T(0);
      for (int q = 0; q < 8; ++q) s += Elem<TG_HEX8>::N<T>(q, a) * quad[q * V + k];
      out[a * V + k] = s;
    }
}

// out[e, q, v] = sum_a N_a(xi_q) u[conn[e, a], v]
template <class T, int NV, bool VEC>
__global__ void __launch_bounds__(128)
    hex_eval_kernel(const T* __restrict__ nodal, int V, const int32_t* __restrict__ conn,
                    int64_t n_elems, T* __restrict__ out) {
  constexpr int G = hex_group<NV>();
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n_elems) return;
  int nid[8];
#pragma unroll
  for (int a = 0; a < 8; ++a) nid[a] = __ldg(conn + e * 8 + a);
  if (NV) V = NV;
  for (int v0 = 0; v0 < V; v0 += G) {
    const int nv = (V - v0) < G ? (V - v0) : G;
    T m[8][G], base[G];
    hex_load_values<T, NV>(nodal, V, v0, nv, nid, m);
#pragma unroll
    for (int k = 0; k < G; ++k) base[k] = m[0][k];
    hex_modes8<T, G>(m);
    hex_scale_value<T, G>(m);
    hex_modes8_adjoint<T, G>(m);
    T o[8 * G];
#pragma unroll
    for (int q = 0; q < 8; ++q)
#pragma unroll
      for (int k = 0; k < G; ++k) o[q * G + k] = m[q][k] + base[k];
    T* dst = out + e * 8 * V + v0;
    if (any_nonfinite(o)) {
      hex_eval_weighted(nodal, V, v0, nv, conn + e * 8, dst);
      continue;
    }
    if constexpr (NV) {
      store_run<VEC>(dst, o);
    } else {
#pragma unroll
      for (int q = 0; q < 8; ++q)
#pragma unroll
        for (int k = 0; k < G; ++k)
          if (k < nv) dst[q * V + k] = o[q * G + k];
    }
  }
}

// contrib[e, a, v] = sum_q N_a(xi_q) quad[e, q, v]
template <class T, int NV, bool VEC>
__global__ void __launch_bounds__(128)
    hex_eval_transpose_elem_kernel(const T* __restrict__ quad, int V, int64_t n_elems,
                                   T* __restrict__ contrib) {
  constexpr int G = hex_group<NV>();
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n_elems) return;
  if (NV) V = NV;
  for (int v0 = 0; v0 < V; v0 += G) {
    const int nv = (V - v0) < G ? (V - v0) : G;
    T f[8 * G];
    const T* src = quad + e * 8 * V + v0;
    if constexpr (NV) {
      load_run<VEC>(src, f);
    } else {
#pragma unroll
      for (int q = 0; q < 8; ++q)
#pragma unroll
        for (int k = 0; k < G; ++k) f[q * G + k] = k < nv ? src[q * V + k] : T(0);
    }
    T m[8][G];
#pragma unroll
    for (int q = 0; q < 8; ++q)
#pragma unroll
      for (int k = 0; k < G; ++k) m[q][k] = f[q * G + k];
    hex_modes8<T, G>(m);
#pragma unroll
    for (int k = 0; k < G; ++k) m[0][k] = fma(T(8), f[k], m[0][k]);
    hex_scale_value<T, G>(m);
    hex_modes8_adjoint<T, G>(m);
    T* dst = contrib + e * 8 * V + v0;
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
      for (int k = 0; k < G; ++k) f[a * G + k] = m[a][k];
    if (any_nonfinite(f)) {
      hex_eval_transpose_weighted(src, V, nv, dst);
      continue;
    }
    if constexpr (NV) {
      store_run<VEC>(dst, f);
    } else {
#pragma unroll
      for (int a = 0; a < 8; ++a)
#pragma unroll
        for (int k = 0; k < G; ++k)
          if (k < nv) dst[a * V + k] = f[a * G + k];
    }
  }
}

// the kernel variant of V components and of arrays (quadrature side and workspace) that are
// 32-byte aligned or not
inline bool aligned32(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 31u) == 0; }
template <class F>
void simplex_variant(int V, F&& f) {
  if (V == 1) f(IntC<1>{});
  else if (V == 2) f(IntC<2>{});
  else if (V == 3) f(IntC<3>{});
  else f(IntC<0>{});
}
template <class F>
void hex_variant(int V, bool vec, F&& f) {
  if (V == 1) vec ? f(IntC<1>{}, IntC<1>{}) : f(IntC<1>{}, IntC<0>{});
  else if (V == 2) vec ? f(IntC<2>{}, IntC<1>{}) : f(IntC<2>{}, IntC<0>{});
  else if (V == 3) vec ? f(IntC<3>{}, IntC<1>{}) : f(IntC<3>{}, IntC<0>{});
  else f(IntC<0>{}, IntC<0>{});
}

// ------------------------------------------------------------------ weights
template <int ET, class T>
__global__ void weights_kernel(const T* __restrict__ coords, const int32_t* __restrict__ conn,
                               int64_t n_elems, T* __restrict__ out) {
  using E = Elem<ET>;
  constexpr int NN = E::NN, D = E::D;
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n_elems) return;
  T X[NN][D];
  int nid[NN];
  gather_coords<ET, T>(coords, conn, e, X, nid);
#pragma unroll
  for (int q = 0; q < E::Q; ++q) {
    T G[NN][D];
    const T det = qp_geometry<ET, T>(q, X, G);
    out[e * E::Q + q] = det * E::template w<T>(q);
  }
}

// ------------------------------------------------------------------ integrate quad array
template <class T>
__global__ void integrate_quad_kernel(const T* __restrict__ quad, const T* __restrict__ w,
                                      int64_t n_elems, int Q, int V, T* __restrict__ out) {
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (tid >= n_elems * V) return;
  const int v = (int)(tid % V);
  const int64_t e = tid / V;
  T acc = T(0);
  for (int q = 0; q < Q; ++q) acc += quad[(e * Q + q) * V + v] * w[e * Q + q];
  out[tid] = acc;
}

// ------------------------------------------------------------------ deterministic row sums
// Stage 1: a fixed number of chunks (independent of the GPU), each summed by one
// block in a fixed strided + tree order, accumulated in FP64.  Stage 2: one block
// sums the chunk partials in a fixed tree order.
constexpr int SUM_CHUNKS = 512;
constexpr int SUM_THREADS = 256;

template <class T>
__global__ void __launch_bounds__(SUM_THREADS)
    rowsum_stage1(const T* __restrict__ in, int64_t n_rows, int V, double* __restrict__ part) {
  __shared__ double sh[SUM_THREADS];
  const int64_t chunk = (n_rows + SUM_CHUNKS - 1) / SUM_CHUNKS;
  const int64_t r0 = blockIdx.x * chunk;
  const int64_t r1 = min(n_rows, r0 + chunk);
  for (int v = 0; v < V; ++v) {
    double acc = 0.0;
    for (int64_t r = r0 + threadIdx.x; r < r1; r += SUM_THREADS) acc += (double)in[r * V + v];
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int s = SUM_THREADS / 2; s > 0; s >>= 1) {
      if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
      __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x * V + v] = sh[0];
    __syncthreads();
  }
}

template <class T>
__global__ void __launch_bounds__(SUM_THREADS)
    rowsum_stage2(const double* __restrict__ part, int V, T* __restrict__ out) {
  __shared__ double sh[SUM_THREADS];
  for (int v = 0; v < V; ++v) {
    double acc = 0.0;
    for (int b = threadIdx.x; b < SUM_CHUNKS; b += SUM_THREADS) acc += part[b * V + v];
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int s = SUM_THREADS / 2; s > 0; s >>= 1) {
      if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
      __syncthreads();
    }
    if (threadIdx.x == 0) out[v] = (T)sh[0];
    __syncthreads();
  }
}

// ------------------------------------------------------------------ gather
template <class T>
__global__ void gather_nodal_kernel(const T* __restrict__ nodal, int V,
                                    const int32_t* __restrict__ conn, int64_t n_entries,
                                    T* __restrict__ out) {
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (tid >= n_entries * V) return;
  const int v = (int)(tid % V);
  const int64_t k = tid / V;
  out[tid] = nodal[(int64_t)__ldg(conn + k) * V + v];
}

// ------------------------------------------------------------------ transposes
// Phase 1: element e's contribution to each of its nodes, c[e][a][v] = sum_q sum_d
// dNdX[e,q,d,a] flux[e,q,v,d] (the adjoint of the gradient kernels).
template <int ET, class T, int NV>
__global__ void __launch_bounds__(SIMPLEX_THREADS)
    simplex_grad_transpose_elem_kernel(const T* __restrict__ flux, const T* __restrict__ coords,
                                       int V, const int32_t* __restrict__ conn, int64_t n_elems,
                                       T* __restrict__ contrib) {
  using E = Elem<ET>;
  constexpr int NN = E::NN, D = E::D, N = (NV ? NV : 1) * D, M = (NV ? NV : 1) * NN;
  constexpr int ROW = run_stride<N>() > run_stride<M>() ? run_stride<N>() : run_stride<M>();
  __shared__ T tiles[NV ? SIMPLEX_THREADS / 32 * 32 * ROW : 1];
  const int64_t e = (int64_t)blockIdx.x * SIMPLEX_THREADS + threadIdx.x;
  const int64_t e0 = e - (threadIdx.x & 31);
  if (e0 >= n_elems) return;  // whole warps
  const int64_t ec = e < n_elems ? e : n_elems - 1;
  int nid[NN];
  T R[D][D];
  simplex_inverse<ET, T>(coords, conn, ec, nid, R);
  // node 0's shape gradient; its share as their product with it (minus the sum of the other
  // shares is two operations less, but rounds 4 to 9 % more, and infinite fluxes meet in it
  // with both signs)
  T g0[D];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    g0[d] = -R[d][0];
#pragma unroll
    for (int k = 1; k < D; ++k) g0[d] -= R[d][k];
  }
  auto contribution = [&](const T* f, T (&c)[NN]) {
#pragma unroll
    for (int a = 0; a < NN; ++a) {
      c[a] = (a ? R[0][a ? a - 1 : 0] : g0[0]) * f[0];
#pragma unroll
      for (int d = 1; d < D; ++d) c[a] = fma(a ? R[d][a ? a - 1 : 0] : g0[d], f[d], c[a]);
    }
  };
  if constexpr (NV) {
    const int n_here = (int)(n_elems - e0 < 32 ? n_elems - e0 : 32);
    T* tile = tiles + (threadIdx.x >> 5) * 32 * ROW;
    T f[N], o[M];
    warp_load_runs<N>(flux + e0 * N, tile, f, n_here);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      T c[NN];
      contribution(f + v * D, c);
#pragma unroll
      for (int a = 0; a < NN; ++a) o[a * NV + v] = c[a];
    }
    warp_store_runs<M>(contrib + e0 * M, tile, o, n_here);
  } else {
    if (e < n_elems)
      for (int v = 0; v < V; ++v) {
        T c[NN];
        contribution(flux + (e * V + v) * D, c);
#pragma unroll
        for (int a = 0; a < NN; ++a) contrib[(e * NN + a) * V + v] = c[a];
      }
  }
}

// Phase 2: out[n] = the contributions of node n's incident (element, corner) pairs, in
// the order of the incidence CSR (increasing element): deterministic.  Each pair's load
// waits for its index, so eight pairs are in flight (a Hex8 grid node has eight; FP32, 3
// values, 881,000 nodes: 37.5 us with four, 31.7 with eight), four in FP64 (1 value, 253,000
// nodes: 8.6 us, 10.2 with eight).
template <class T>
__global__ void transpose_node_kernel(const T* __restrict__ contrib, int64_t n_nodes, int V,
                                      const int32_t* __restrict__ inc_ptr,
                                      const int32_t* __restrict__ inc_idx, T* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_nodes * V) return;
  const int64_t n = i < (int64_t)1 << 31 ? (int64_t)((unsigned)i / (unsigned)V) : i / V;
  const int v = (int)(i - n * V);
  T s = T(0);
  int k = __ldg(inc_ptr + n);
  const int k1 = __ldg(inc_ptr + n + 1);
  auto run = [&](auto count) {
    constexpr int C = decltype(count)::value;
    for (; k + C <= k1; k += C) {
      int j[C];
      T c[C];
#pragma unroll
      for (int t = 0; t < C; ++t) j[t] = __ldg(inc_idx + k + t);
#pragma unroll
      for (int t = 0; t < C; ++t) c[t] = __ldg(contrib + (int64_t)j[t] * V + v);
#pragma unroll
      for (int t = 0; t < C; ++t) s += c[t];
    }
  };
  if constexpr (sizeof(T) == 4) run(std::integral_constant<int, 8>{});
  run(std::integral_constant<int, 4>{});
  run(std::integral_constant<int, 1>{});
  out[i] = s;
}

// One-point elements: a thread per (node, component), four incident elements' loads in flight.
template <int ET, class T>
__global__ void simplex_eval_transpose_kernel(const T* __restrict__ quad, int64_t n_nodes, int V,
                                              const int32_t* __restrict__ inc_ptr,
                                              const int32_t* __restrict__ inc_idx,
                                              T* __restrict__ out) {
  using E = Elem<ET>;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_nodes * V) return;
  const int64_t n = i / V;
  const int v = (int)(i - n * V);
  const T w0 = E::template N<T>(0, 0), w1 = E::template N<T>(0, 1);
  T s = T(0);
  int k = __ldg(inc_ptr + n);
  const int k1 = __ldg(inc_ptr + n + 1);
  for (; k < k1; k += 4) {
    T c[4], w[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int ea = k + t < k1 ? __ldg(inc_idx + k + t) : -1;
      const int e = ea / E::NN;
      w[t] = ea < 0 ? T(0) : (ea == e * E::NN ? w0 : w1);
      c[t] = ea < 0 ? T(0) : __ldg(quad + (int64_t)e * V + v);
    }
#pragma unroll
    for (int t = 0; t < 4; ++t) s = fma(w[t], c[t], s);
  }
  out[i] = s;
}

template <int ET, class T>
__global__ void eval_transpose_kernel(const T* __restrict__ quad, int64_t n_nodes, int V,
                                      const int32_t* __restrict__ inc_ptr,
                                      const int32_t* __restrict__ inc_idx, T* __restrict__ out) {
  using E = Elem<ET>;
  const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= n_nodes) return;
  for (int v = 0; v < V; ++v) {
    T acc = T(0);
    for (int k = inc_ptr[n]; k < inc_ptr[n + 1]; ++k) {
      const int ea = inc_idx[k];
      const int64_t e = ea / E::NN;
      const int a = ea % E::NN;
      for (int q = 0; q < E::Q; ++q) acc += E::template N<T>(q, a) * quad[(e * E::Q + q) * V + v];
    }
    out[n * V + v] = acc;
  }
}

template <class T>
__global__ void integrate_quad_transpose_kernel(const T* __restrict__ g, const T* __restrict__ w,
                                                int64_t n_elems, int Q, int V,
                                                T* __restrict__ out) {
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (tid >= n_elems * Q * V) return;
  const int v = (int)(tid % V);
  const int64_t eq = tid / V;
  const int64_t e = eq / Q;
  out[tid] = g[e * V + v] * w[eq];
}

}  // namespace tg

using namespace tg;

extern "C" int tg_integrate_quad_transpose(int prec, const void* g, const void* weights,
                                           int64_t n_elems, int n_quad, int n_vals, void* out,
                                           void* stream) {
  TG_TRY(check_sizes(n_elems, 0, n_vals));
  if (n_quad <= 0) return set_error(TG_ERR_VALUE, "n_quad must be positive");
  if (n_elems == 0) return TG_OK;
  TG_TRY(check_ptr(g, "g"));
  TG_TRY(check_ptr(weights, "weights"));
  TG_TRY(check_ptr(out, "out"));
  return dispatch_prec(prec, [&](auto t) -> int {
    using T = decltype(t);
    const int64_t total = n_elems * n_quad * n_vals;
    integrate_quad_transpose_kernel<T><<<grid_for(total, TPB_T), TPB_T, 0, as_stream(stream)>>>(
        (const T*)g, (const T*)weights, n_elems, n_quad, n_vals, (T*)out);
    return launch_check("tg_integrate_quad_transpose");
  });
}

extern "C" int tg_scatter_nodal(int prec, const void* vals, int64_t n_nodes, int n_vals,
                                int nodes_per_elem, const int32_t* inc_ptr,
                                const int32_t* inc_idx, void* out, void* stream) {
  (void)nodes_per_elem;
  TG_TRY(check_sizes(0, n_nodes, n_vals));
  if (n_nodes == 0) return TG_OK;
  TG_TRY(check_ptr(inc_ptr, "inc_ptr"));
  TG_TRY(check_ptr(out, "out"));
  return dispatch_prec(prec, [&](auto t) -> int {
    using T = decltype(t);
    transpose_node_kernel<T><<<grid_for(n_nodes * n_vals, TPB_T), TPB_T, 0, as_stream(stream)>>>(
        (const T*)vals, n_nodes, n_vals, inc_ptr, inc_idx, (T*)out);
    return launch_check("tg_scatter_nodal");
  });
}

static constexpr int TPB = 256;

extern "C" int tg_eval(int elem, int prec, const void* nodal, int64_t n_nodes, int n_vals,
                       const int32_t* conn, int64_t n_elems, void* out, void* stream) {
  TG_TRY(check_sizes(n_elems, n_nodes, n_vals));
  if (n_elems == 0) return TG_OK;
  TG_TRY(check_ptr(nodal, "nodal"));
  TG_TRY(check_ptr(conn, "conn"));
  TG_TRY(check_ptr(out, "out"));
  return dispatch_elem(elem, [&](auto et) -> int {
    constexpr int ET = decltype(et)::value;
    return dispatch_prec(prec, [&](auto t) -> int {
      using T = decltype(t);
      if constexpr (ET == TG_HEX8) {
        hex_variant(n_vals, aligned32(out), [&](auto nv, auto vec) {
          hex_eval_kernel<T, decltype(nv)::value, decltype(vec)::value != 0>
              <<<grid_for(n_elems, 128), 128, 0, as_stream(stream)>>>(
                  (const T*)nodal, n_vals, conn, n_elems, (T*)out);
        });
      } else {
        const int64_t total = n_elems * Elem<ET>::Q * n_vals;
        eval_kernel<ET, T><<<grid_for(total, TPB), TPB, 0, as_stream(stream)>>>(
            (const T*)nodal, n_vals, conn, n_elems, (T*)out);
      }
      return launch_check("tg_eval");
    });
  });
}

extern "C" int tg_grad(int elem, int prec, const void* nodal, const void* coords, int64_t n_nodes,
                       int n_vals, const int32_t* conn, int64_t n_elems, void* out, void* stream) {
  TG_TRY(check_sizes(n_elems, n_nodes, n_vals));
  if (n_elems == 0) return TG_OK;
  TG_TRY(check_ptr(nodal, "nodal"));
  TG_TRY(check_ptr(coords, "coords"));
  TG_TRY(check_ptr(conn, "conn"));
  TG_TRY(check_ptr(out, "out"));
  return dispatch_elem(elem, [&](auto et) -> int {
    constexpr int ET = decltype(et)::value;
    return dispatch_prec(prec, [&](auto t) -> int {
      using T = decltype(t);
      if constexpr (ET == TG_HEX8)
        hex_variant(n_vals, aligned32(out), [&](auto nv, auto vec) {
          hex_grad_kernel<T, decltype(nv)::value, decltype(vec)::value != 0>
              <<<grid_for(n_elems, 128), 128, 0, as_stream(stream)>>>(
                  (const T*)nodal, (const T*)coords, n_vals, conn, n_elems, (T*)out);
        });
      else
        simplex_variant(n_vals, [&](auto nv) {
          simplex_grad_kernel<ET, T, decltype(nv)::value>
              <<<grid_for(n_elems, SIMPLEX_THREADS), SIMPLEX_THREADS, 0, as_stream(stream)>>>(
                  (const T*)nodal, (const T*)coords, n_vals, conn, n_elems, (T*)out);
        });
      return launch_check("tg_grad");
    });
  });
}

extern "C" int tg_integration_weights(int elem, int prec, const void* coords, int64_t n_nodes,
                                      const int32_t* conn, int64_t n_elems, void* out,
                                      void* stream) {
  TG_TRY(check_sizes(n_elems, n_nodes, 1));
  if (n_elems == 0) return TG_OK;
  TG_TRY(check_ptr(coords, "coords"));
  TG_TRY(check_ptr(conn, "conn"));
  TG_TRY(check_ptr(out, "out"));
  return dispatch_elem(elem, [&](auto et) -> int {
    constexpr int ET = decltype(et)::value;
    return dispatch_prec(prec, [&](auto t) -> int {
      using T = decltype(t);
      weights_kernel<ET, T><<<grid_for(n_elems, 128), 128, 0, as_stream(stream)>>>(
          (const T*)coords, conn, n_elems, (T*)out);
      return launch_check("tg_integration_weights");
    });
  });
}

extern "C" int tg_integrate_quad(int prec, const void* quad, const void* weights, int64_t n_elems,
                                 int n_quad, int n_vals, void* out, void* stream) {
  TG_TRY(check_sizes(n_elems, 0, n_vals));
  if (n_quad <= 0) return set_error(TG_ERR_VALUE, "n_quad must be positive");
  if (n_elems == 0) return TG_OK;
  TG_TRY(check_ptr(quad, "quad"));
  TG_TRY(check_ptr(weights, "weights"));
  TG_TRY(check_ptr(out, "out"));
  return dispatch_prec(prec, [&](auto t) -> int {
    using T = decltype(t);
    integrate_quad_kernel<T><<<grid_for(n_elems * n_vals, TPB), TPB, 0, as_stream(stream)>>>(
        (const T*)quad, (const T*)weights, n_elems, n_quad, n_vals, (T*)out);
    return launch_check("tg_integrate_quad");
  });
}

extern "C" size_t tg_sum_rows_workspace_bytes(int prec, int n_vals) {
  (void)prec;
  return (size_t)SUM_CHUNKS * (size_t)(n_vals > 0 ? n_vals : 1) * sizeof(double);
}

extern "C" int tg_sum_rows(int prec, const void* in, int64_t n_rows, int n_vals, void* out,
                           void* workspace, size_t workspace_bytes, void* stream) {
  if (n_rows < 0 || n_vals <= 0) return set_error(TG_ERR_VALUE, "bad sizes for tg_sum_rows");
  TG_TRY(check_ptr(out, "out"));
  if (workspace_bytes < tg_sum_rows_workspace_bytes(prec, n_vals))
    return set_error(TG_ERR_WORKSPACE, "tg_sum_rows: workspace too small");
  if (n_rows > 0) TG_TRY(check_ptr(in, "in"));
  return dispatch_prec(prec, [&](auto t) -> int {
    using T = decltype(t);
    rowsum_stage1<T><<<SUM_CHUNKS, SUM_THREADS, 0, as_stream(stream)>>>(
        (const T*)in, n_rows, n_vals, (double*)workspace);
    rowsum_stage2<T><<<1, SUM_THREADS, 0, as_stream(stream)>>>((const double*)workspace, n_vals,
                                                               (T*)out);
    return launch_check("tg_sum_rows");
  });
}

extern "C" int tg_gather_nodal(int prec, const void* nodal, int64_t n_nodes, int n_vals,
                               const int32_t* conn, int64_t n_elems, int nodes_per_elem,
                               void* out, void* stream) {
  TG_TRY(check_sizes(n_elems, n_nodes, n_vals));
  if (nodes_per_elem <= 0) return set_error(TG_ERR_VALUE, "nodes_per_elem must be positive");
  if (n_elems == 0) return TG_OK;
  TG_TRY(check_ptr(nodal, "nodal"));
  TG_TRY(check_ptr(conn, "conn"));
  TG_TRY(check_ptr(out, "out"));
  const int64_t entries = n_elems * nodes_per_elem;
  return dispatch_prec(prec, [&](auto t) -> int {
    using T = decltype(t);
    gather_nodal_kernel<T><<<grid_for(entries * n_vals, TPB), TPB, 0, as_stream(stream)>>>(
        (const T*)nodal, n_vals, conn, entries, (T*)out);
    return launch_check("tg_gather_nodal");
  });
}

// workspace that pays in tg_eval_transpose_ws: Hex8 sums its eight points per element once
// (the node-centric kernel reads each element's points from all eight corners); the
// one-point elements need none
extern "C" size_t tg_eval_transpose_workspace_bytes(int elem, int prec, int64_t n_elems,
                                                    int n_vals) {
  if (elem != TG_HEX8 || n_elems <= 0 || n_vals <= 0) return 0;
  return (size_t)n_elems * 8 * n_vals * (prec == TG_F32 ? 4 : 8);
}

extern "C" int tg_eval_transpose_ws(int elem, int prec, const void* quad, int64_t n_nodes,
                                    int n_vals, const int32_t* conn, int64_t n_elems,
                                    const int32_t* inc_ptr, const int32_t* inc_idx, void* out,
                                    void* workspace, size_t workspace_bytes, void* stream) {
  TG_TRY(check_sizes(n_elems, n_nodes, n_vals));
  const size_t need = tg_eval_transpose_workspace_bytes(elem, prec, n_elems, n_vals);
  if (need == 0)
    return tg_eval_transpose(elem, prec, quad, n_nodes, n_vals, conn, n_elems, inc_ptr, inc_idx,
                             out, stream);
  if (n_nodes == 0) return TG_OK;
  if (workspace_bytes < need)
    return set_error(TG_ERR_WORKSPACE, "tg_eval_transpose_ws: workspace too small (%zu < %zu)",
                     workspace_bytes, need);
  TG_TRY(check_ptr(quad, "quad"));
  TG_TRY(check_ptr(inc_ptr, "inc_ptr"));
  TG_TRY(check_ptr(inc_idx, "inc_idx"));
  TG_TRY(check_ptr(out, "out"));
  TG_TRY(check_ptr(workspace, "workspace"));
  return dispatch_prec(prec, [&](auto t) -> int {
    using T = decltype(t);
    hex_variant(n_vals, aligned32(quad) && aligned32(workspace), [&](auto nv, auto vec) {
      hex_eval_transpose_elem_kernel<T, decltype(nv)::value, decltype(vec)::value != 0>
          <<<grid_for(n_elems, 128), 128, 0, as_stream(stream)>>>((const T*)quad, n_vals,
                                                                  n_elems, (T*)workspace);
    });
    transpose_node_kernel<T><<<grid_for(n_nodes * n_vals, 256), 256, 0, as_stream(stream)>>>(
        (const T*)workspace, n_nodes, n_vals, inc_ptr, inc_idx, (T*)out);
    return launch_check("tg_eval_transpose_ws");
  });
}

extern "C" size_t tg_grad_transpose_workspace_bytes(int elem, int prec, int64_t n_elems,
                                                    int n_vals) {
  const int NN = elem == TG_TRI3 ? 3 : (elem == TG_TET4 ? 4 : 8);
  if (n_elems <= 0 || n_vals <= 0) return 0;
  return (size_t)n_elems * NN * n_vals * (prec == TG_F32 ? 4 : 8);
}

extern "C" int tg_grad_transpose(int elem, int prec, const void* flux, const void* coords,
                                 int64_t n_nodes, int n_vals, const int32_t* conn,
                                 int64_t n_elems, const int32_t* inc_ptr, const int32_t* inc_idx,
                                 void* out, void* workspace, size_t workspace_bytes,
                                 void* stream) {
  TG_TRY(check_sizes(n_elems, n_nodes, n_vals));
  if (n_nodes == 0) return TG_OK;
  if (workspace_bytes < tg_grad_transpose_workspace_bytes(elem, prec, n_elems, n_vals))
    return set_error(TG_ERR_WORKSPACE, "tg_grad_transpose: workspace too small (%zu < %zu)",
                     workspace_bytes, tg_grad_transpose_workspace_bytes(elem, prec, n_elems, n_vals));
  TG_TRY(check_ptr(coords, "coords"));
  TG_TRY(check_ptr(inc_ptr, "inc_ptr"));
  TG_TRY(check_ptr(out, "out"));
  if (n_elems > 0) {
    TG_TRY(check_ptr(flux, "flux"));
    TG_TRY(check_ptr(conn, "conn"));
    TG_TRY(check_ptr(inc_idx, "inc_idx"));
  }
  return dispatch_elem(elem, [&](auto et) -> int {
    constexpr int ET = decltype(et)::value;
    return dispatch_prec(prec, [&](auto t) -> int {
      using T = decltype(t);
      if (n_elems > 0) {
        if constexpr (ET == TG_HEX8)
          hex_variant(n_vals, aligned32(flux) && aligned32(workspace), [&](auto nv, auto vec) {
            hex_grad_transpose_elem_kernel<T, decltype(nv)::value, decltype(vec)::value != 0>
                <<<grid_for(n_elems, 128), 128, 0, as_stream(stream)>>>(
                    (const T*)flux, (const T*)coords, n_vals, conn, n_elems, (T*)workspace);
          });
        else
          simplex_variant(n_vals, [&](auto nv) {
            simplex_grad_transpose_elem_kernel<ET, T, decltype(nv)::value>
                <<<grid_for(n_elems, SIMPLEX_THREADS), SIMPLEX_THREADS, 0, as_stream(stream)>>>(
                    (const T*)flux, (const T*)coords, n_vals, conn, n_elems, (T*)workspace);
          });
      }
      transpose_node_kernel<T><<<grid_for(n_nodes * n_vals, 256), 256, 0, as_stream(stream)>>>(
          (const T*)workspace, n_nodes, n_vals, inc_ptr, inc_idx, (T*)out);
      return launch_check("tg_grad_transpose");
    });
  });
}

extern "C" int tg_eval_transpose(int elem, int prec, const void* quad, int64_t n_nodes,
                                 int n_vals, const int32_t* conn, int64_t n_elems,
                                 const int32_t* inc_ptr, const int32_t* inc_idx, void* out,
                                 void* stream) {
  (void)conn;
  TG_TRY(check_sizes(n_elems, n_nodes, n_vals));
  if (n_nodes == 0) return TG_OK;
  TG_TRY(check_ptr(inc_ptr, "inc_ptr"));
  TG_TRY(check_ptr(out, "out"));
  if (n_elems > 0) {
    TG_TRY(check_ptr(quad, "quad"));
    TG_TRY(check_ptr(inc_idx, "inc_idx"));
  }
  return dispatch_elem(elem, [&](auto et) -> int {
    constexpr int ET = decltype(et)::value;
    return dispatch_prec(prec, [&](auto t) -> int {
      using T = decltype(t);
      if constexpr (Elem<ET>::Q == 1)
        simplex_eval_transpose_kernel<ET, T><<<grid_for(n_nodes * n_vals, TPB_T), TPB_T, 0,
                                               as_stream(stream)>>>(
            (const T*)quad, n_nodes, n_vals, inc_ptr, inc_idx, (T*)out);
      else
        eval_transpose_kernel<ET, T><<<grid_for(n_nodes, 128), 128, 0, as_stream(stream)>>>(
            (const T*)quad, n_nodes, n_vals, inc_ptr, inc_idx, (T*)out);
      return launch_check("tg_eval_transpose");
    });
  });
}
