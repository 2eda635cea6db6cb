// Structured-brick stencil of the linear-elastic Hex8 operator: the tile code shared by
// the single-solve kernels (grid.cu) and the batched request engine (bricks.cu).
//
// Linear-elastic Hex8 residual / HVP on a structured brick: the assembled operator as
// a 27-point stencil of 3 x 3 blocks.
//
// When the mesh is a tensor grid of Nx x Ny x Nz nodes with uniform spacing (hx, hy,
// hz) along each axis, node ids i + Nx (j + Ny k) and one element per cell with the
// corner order of the reference Hexahedron8 (tatva/element/base.py:478-491), every
// element has the same stiffness matrix and the HVP y = sum_e K_e v_e is, at a node
// whose eight surrounding cells all exist, a fixed stencil.  With 1-D factors on an
// axis of spacing h
//   K(0) = 2/h, K(+-1) = -1/h          (int phi_n' phi_m')
//   M(0) = 2h/3, M(+-1) = h/6          (int phi_n phi_m)
//   G(d) = -d/2                        (int phi_n' phi_{n+d})
// the 3 x 3 block for an input node at offset d = (dx, dy, dz) is
//   C_aa(d) = mu (Kx My Mz + Mx Ky Mz + Mx My Kz)(d) + (lambda + mu) D_aa(d),
//             D_xx = Kx My Mz, D_yy = Mx Ky Mz, D_zz = Mx My Kz,
//   C_ab(d) = -(lambda + mu) G(d_a) G(d_b) M(d_c)      (a != b, c the third axis),
// i.e. mu delta_ab sum_i D_ii + lambda D_ab + mu D_ba of the energy
// 1/2 sigma:eps (tests/test_sparse_benchmark.py:30-78), integrated exactly -- the
// 2 x 2 x 2 Gauss rule of the element is exact for these products -- so the stencil
// equals the element-by-element sum up to rounding.  This is what jax.jvp(jax.grad(E))
// computes for E = integrate(psi(grad u)) (README.md:93, tatva/sparse/base.py:257-265).
//
// Schedule (one launch):
//   * interior CTAs: a tile of 32 x 8 node columns (x, y) and a run of z planes.  Each
//     thread owns one column (FP32: two, below) and sweeps z; the input plane (with a
//     one-node halo, 34 x 10 nodes, 3 components in a 16-byte slot) sits in shared memory; a
//     plane adds its contributions to the outputs at z - 1, z, z + 1 (three accumulator sets), so each
//     output is complete after its upper neighbour plane.  Planes arrive through
//     registers two planes ahead (the Dirichlet mask is applied on the way) and are
//     double-buffered in shared memory: one barrier per plane.  Per node and plane:
//     nine 16-byte shared loads and ~90 FP operations, using the stencil's symmetries
//     (in-plane sums grouped by |dx|, |dy| for the diagonal blocks; signed cross sums
//     for the off-diagonal ones).
//     The z faces belong to the sweep: the 1-D matrices of a finite interval differ from
//     the infinite ones in their corner entries only, K(0), M(0) half of the interior's and
//     G(0) = -+1/2.  So a face plane's own contribution to its outputs is half the interior
//     one plus a term in (lambda - mu)/4, and the planes next to it contribute as inside.
//   * face CTAs: the x and y faces with the node's one-sided 18-point stencil (the four
//     cells around it merged, in constants): y faces a node per thread, consecutive along
//     x; x faces in 16 x 8 patches (FP64 16 x 16) whose two node columns next to the face
//     are staged in shared memory first (consecutive nodes are a grid row apart).
//   * edge CTAs: nodes on two or three faces, as the sum over the cells that exist around
//     the node of the element matrix times the cell's input values.
// Every output is written once by the thread that owns it, in a fixed order: the
// result is deterministic and needs no atomics, partial slots or second pass.
#pragma once

#include <cstddef>
#include <type_traits>

#include "tg_cg.cuh"
#include "tg_common.cuh"
#include "tg_f32x2.cuh"
#include "tg_internal.h"

namespace tg {

// Tile height (node rows per CTA) and interior planes per tile, measured on GB300 (128^3
// brick).  FP32: 128 threads, each two node columns four rows apart (grid_interior_pair);
// FP64: 256 threads, a column each (grid_interior), its kernels being FP64-pipe bound.
constexpr int GR_DEEP_TZ = 11, GR_MAX_TZ = 15;
// Unknowns up to which CG iterations run as one cooperative launch (grid_cg_kernel): at 96^3
// (2.7 M) 37.0 against 41.9 us an iteration in three launches, at 128^3 (6.4 M), where the
// vector passes want more loads in flight than one CTA per SM keeps, 90.1 against 81.5.
constexpr int64_t GRID_CG_MAX_DOFS = 3500000;
constexpr int GR_TX = 32, GR_TY = 8;
constexpr int GR_PX = GR_TX + 2, GR_PY = GR_TY + 2, GR_PLANE = GR_PX * GR_PY;  // 340
template <class T>
constexpr int grid_threads() { return sizeof(T) == 4 ? 128 : 256; }
template <class T>
constexpr int grid_ctas_per_sm() { return sizeof(T) == 4 ? 3 : 2; }
// x-face patch: GR_XT x grid_xt_z nodes
constexpr int GR_XT = 16, GR_XS = GR_XT + 2;
template <class T>
constexpr int grid_xt_z() { return grid_threads<T>() / GR_XT; }
// FP32 interior tiles: pairs of rows (r, r + GP_HALF), staged with halo as GP_SLOTS pair
// slots of 24 bytes per plane, GP_STAGES planes in flight
constexpr int GP_HALF = GR_TY / 2, GP_ROWS = GP_HALF + 2, GP_SLOTS = GR_PX * GP_ROWS;  // 204
constexpr int GP_STAGES = 4;
constexpr int GP_ENTRIES = (2 * GP_SLOTS + 127) / 128;  // node copies per thread and plane
struct GridPairStage {
  ulonglong2 xy[GP_SLOTS];  // (x of both rows), (y of both rows)
  unsigned long long z[GP_SLOTS];
};
// shared memory of one CTA
template <class T>
struct GridShared;
template <>
struct GridShared<float> {
  union {
    GridPairStage stage[GP_STAGES];
    float4 sm[2 * GR_XS * (grid_xt_z<float>() + 2)];
    float ke[8 * 8 * 9];
  };
};
template <>
struct GridShared<double> {
  union {
    double4 sm[2 * GR_PLANE];
    double ke[8 * 8 * 9];
  };
};
static_assert(2 * GR_XS * (grid_xt_z<double>() + 2) <= 2 * GR_PLANE, "x-face staging fits");

template <class T>
struct GridCoef {
  T c[3][8];   // diagonal blocks: c[a][ix + 2 iy + 4 iz], i* = |d*| in {0, 1}
  T qxy[2];    // -(lambda + mu)/4 M_z(0), M_z(1)
  T qxz[2];    // -(lambda + mu)/4 M_y(0), M_y(1)
  T qyz[2];    // -(lambda + mu)/4 M_x(0), M_x(1)
  T r1[3];     // in-plane row sum of the |dz| = 1 diagonal-block coefficients
  T kxz[2], kyz[2];  // (lambda - mu)/4 M_y, M_x: the z faces' own-plane coupling
  int nx, ny, nz;    // nodes per axis
  int tiles_x, tiles_y, tiles_z, tz;  // tiling of the interior columns: tz planes per tile
  int edge_lanes;        // lanes of a node on two or three faces
  int n_yface_ctas;      // y face nodes, one per thread
  int xt_y, xt_z;        // x-face patches per face along y and z
  int n_xface_ctas;      // 2 xt_y xt_z
  // the rest is read by the face CTAs only
  T fx[2][2][9][3][3];  // x faces (low, high): node column next to the face, 3 (dz+1) + dy+1
  T fy[2][2][9][3][3];  // y faces: node row, 3 (dz+1) + dx+1
  T ke[8][8][3][3];     // element matrix, corners cn, cm = lx + 2 ly + 4 lz
};

template <class T>
struct Vec4;
template <>
struct Vec4<float> {
  using type = float4;
};
template <>
struct Vec4<double> {
  using type = double4;
};

template <class T>
__device__ __forceinline__ typename Vec4<T>::type make4(T a, T b, T c) {
  typename Vec4<T>::type r;
  r.x = a;
  r.y = b;
  r.z = c;
  r.w = T(0);
  return r;
}

// Dirichlet masks: none, one byte per dof (the C ABI's `fixed`), or one byte per node
// with bit d set when dof 3 n + d is fixed (packed once per solve by the CG, so that a
// node's mask is one load instead of three)
// MASK_NODE_OUT: the node byte applied to the output rows only -- for inputs that are
// already zero on the fixed dofs (the CG's direction when the preconditioner is zero
// there), so the staged loads need no mask.
constexpr int MASK_NONE = 0, MASK_DOF = 1, MASK_NODE = 2, MASK_NODE_OUT = 3;

// whether the launch masks its input values (the Dirichlet columns of an HVP)
template <int MODE, int MK>
__device__ __forceinline__ constexpr bool masks_input() {
  return MODE == TG_MODE_HVP && MK != MASK_NONE && MK != MASK_NODE_OUT;
}

// p.q (or r.r) of a grid launch: per node the three products summed in T (FMAs), the node
// sums accumulated in a fixed order -- FP64 in FP64; FP32 as an unevaluated float pair (one
// two-sum per node, exact to 48 bits): a conversion and an addition in FP64 per node held
// the FP64 pipe, 64 cycles a warp instruction, about as long as the stencil takes.  The error
// of p.q is the node sums' rounding, 2^-24 each, with either (simulated: 9.4e-11 of the whole
// at 200,000 nodes, the two 2e-18 apart).
template <class T>
struct GridDotAcc;
template <>
struct GridDotAcc<double> {
  double v = 0.0;
  __device__ __forceinline__ void add3(const double (&a)[3], const double (&b)[3]) {
    v += fma(a[2], b[2], fma(a[1], b[1], a[0] * b[0]));
  }
  __device__ __forceinline__ double value() const { return v; }
};
template <>
struct GridDotAcc<float> {
  float hi = 0.f, lo = 0.f;
  __device__ __forceinline__ void add(float s) {
    const float t = hi + s, bp = t - hi;
    lo += (hi - (t - bp)) + (s - bp);
    hi = t;
  }
  __device__ __forceinline__ void add3(const float (&a)[3], const float (&b)[3]) {
    add(fmaf(a[2], b[2], fmaf(a[1], b[1], a[0] * b[0])));
  }
  __device__ __forceinline__ double value() const { return (double)hi + (double)lo; }
};

// Output of a launch: the operator applied (EPI_PLAIN; with DOT, p.q of input and
// output), or the residual y = b - A x of a right-hand side b (EPI_RESID; with DOT,
// y.y).
constexpr int EPI_PLAIN = 0, EPI_RESID = 1;

// A group of grid_threads<T>() threads works on one tile or face.  It is the CTA, or (COH:
// the persistent CG, whose CTA holds several groups) a part of it with its own barrier.
template <class T, bool COH>
__device__ __forceinline__ int group_tid() {
  return COH ? threadIdx.x & (grid_threads<T>() - 1) : threadIdx.x;
}
template <class T, bool COH>
__device__ __forceinline__ void group_sync() {
  if constexpr (COH)
    asm volatile("bar.sync %0, %1;" ::"r"(1 + threadIdx.x / grid_threads<T>()),
                 "n"(grid_threads<T>())
                 : "memory");
  else
    __syncthreads();
}

// Loads of a launch's input vector.  COH: the vector is written between the sweeps of one
// launch (the persistent CG), so a load must not be moved or served as read-only data; it
// sees the other CTAs' stores after a grid barrier (whose fence also empties the SM's L1).
template <bool COH, class T>
__device__ __forceinline__ T ld_in(const T* p) {
  if constexpr (!COH) {
    return __ldg(p);
  } else {
    T v;
    if constexpr (sizeof(T) == 4)
      asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    else
      asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
  }
}

// bit d of the mask of node g (0: free)
template <int MK>
__device__ __forceinline__ int mask_bits(const uint8_t* __restrict__ fixed, int64_t g) {
  if constexpr (MK == MASK_DOF) {
    return (__ldg(fixed + 3 * g) != 0) | (__ldg(fixed + 3 * g + 1) != 0) << 1 |
           (__ldg(fixed + 3 * g + 2) != 0) << 2;
  } else if constexpr (MK == MASK_NODE || MK == MASK_NODE_OUT) {
    return __ldg(fixed + g);
  } else {
    return 0;
  }
}

// One input plane's contributions to the outputs below (accM, z - 1), at (accP, z) and
// above (accN, z + 1) the plane, for the node column at shared-memory slot c0 (FP64: value
// form; the FP32 form is in pair_plane).  ctr: this plane's column value (out); side: +1 on
// the low, -1 on the high z face, else 0.
template <class T>
__device__ __forceinline__ void stencil_plane(const GridCoef<T>& P,
                                              const typename Vec4<T>::type* buf, int c0,
                                              T (&accM)[3], T (&accP)[3], T (&accN)[3],
                                              T (&ctr)[3], int side) {
  using V4 = typename Vec4<T>::type;
  // the nine in-plane neighbours, v[dy + 1][dx + 1]
  V4 v[3][3];
#pragma unroll
  for (int dy = 0; dy < 3; ++dy)
#pragma unroll
    for (int dx = 0; dx < 3; ++dx) v[dy][dx] = buf[c0 + (dx - 1) + GR_PX * (dy - 1)];
  const T a0[3] = {v[1][1].x, v[1][1].y, v[1][1].z};
  const T xm[3] = {v[1][0].x, v[1][0].y, v[1][0].z}, xp[3] = {v[1][2].x, v[1][2].y, v[1][2].z};
  const T ym[3] = {v[0][1].x, v[0][1].y, v[0][1].z}, yp[3] = {v[2][1].x, v[2][1].y, v[2][1].z};
  const T mm[3] = {v[0][0].x, v[0][0].y, v[0][0].z}, pm[3] = {v[0][2].x, v[0][2].y, v[0][2].z};
  const T mp[3] = {v[2][0].x, v[2][0].y, v[2][0].z}, pp[3] = {v[2][2].x, v[2][2].y, v[2][2].z};
  // a face plane adds half of these sums to the outputs in it (and the terms at the end): what
  // was there before enters twice and the whole is halved, both exact, so that the other
  // planes pay nothing for it (sums of their own cost 3 of 93 FP64 instructions)
  if (side) {
#pragma unroll
    for (int a = 0; a < 3; ++a) accP[a] += accP[a];
  }
  // diagonal blocks grouped by |dx|, |dy|
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    ctr[a] = a0[a];
    const T gx = xm[a] + xp[a], gy = ym[a] + yp[a];
    const T gc = (mm[a] + mp[a]) + (pm[a] + pp[a]);
    accP[a] = fma(P.c[a][3], gc,
                  fma(P.c[a][2], gy, fma(P.c[a][1], gx, fma(P.c[a][0], a0[a], accP[a]))));
    const T s1 = fma(P.c[a][7], gc, fma(P.c[a][6], gy, fma(P.c[a][5], gx, P.c[a][4] * a0[a])));
    accM[a] += s1;
    accN[a] += s1;
  }
  // x-y blocks: C = qxy(|dz|) dx dy, the cross sum of the in-plane corners
  const T wx = (pp[0] - pm[0]) - (mp[0] - mm[0]);
  const T wy = (pp[1] - pm[1]) - (mp[1] - mm[1]);
  accP[0] = fma(P.qxy[0], wy, accP[0]);
  accM[0] = fma(P.qxy[1], wy, accM[0]);
  accN[0] = fma(P.qxy[1], wy, accN[0]);
  accP[1] = fma(P.qxy[0], wx, accP[1]);
  accM[1] = fma(P.qxy[1], wx, accM[1]);
  accN[1] = fma(P.qxy[1], wx, accN[1]);
  // x-z blocks: C = qxz(|dy|) dx dz: odd in x, summed over dy with M_y
  const T uz_x = fma(P.qxz[1], ((pm[2] - mm[2]) + (pp[2] - mp[2])), P.qxz[0] * (xp[2] - xm[2]));
  const T ux_x = fma(P.qxz[1], ((pm[0] - mm[0]) + (pp[0] - mp[0])), P.qxz[0] * (xp[0] - xm[0]));
  // y-z blocks: C = qyz(|dx|) dy dz: odd in y, summed over dx with M_x
  const T uz_y = fma(P.qyz[1], ((mp[2] - mm[2]) + (pp[2] - pm[2])), P.qyz[0] * (yp[2] - ym[2]));
  const T uy_y = fma(P.qyz[1], ((mp[1] - mm[1]) + (pp[1] - pm[1])), P.qyz[0] * (yp[1] - ym[1]));
  // dz = plane - output: the output below (z - 1) sees dz = +1, the one above -1
  accM[0] += uz_x;
  accN[0] -= uz_x;
  accM[2] += ux_x;
  accN[2] -= ux_x;
  accM[1] += uz_y;
  accN[1] -= uz_y;
  accM[2] += uy_y;
  accN[2] -= uy_y;
  if (side) {  // half the interior's own-plane entries and the corner entries of G_z
    const T sg = T(side);
    const T zx = fma(P.kxz[1], ((pm[2] - mm[2]) + (pp[2] - mp[2])), P.kxz[0] * (xp[2] - xm[2]));
    const T xx = fma(P.kxz[1], ((pm[0] - mm[0]) + (pp[0] - mp[0])), P.kxz[0] * (xp[0] - xm[0]));
    const T zy = fma(P.kyz[1], ((mp[2] - mm[2]) + (pp[2] - pm[2])), P.kyz[0] * (yp[2] - ym[2]));
    const T yy = fma(P.kyz[1], ((mp[1] - mm[1]) + (pp[1] - pm[1])), P.kyz[0] * (yp[1] - ym[1]));
    accP[0] = fma(sg, zx, T(0.5) * accP[0]);
    accP[1] = fma(sg, zy, T(0.5) * accP[1]);
    accP[2] = fma(-sg, xx + yy, T(0.5) * accP[2]);
  }
}

// Tile of interior columns: thread (lx, ly) owns node column (x0 + lx, y0 + ly), planes
// [zs, ze) of output (the z faces among them), from the input planes ps .. pe.
template <class T, int MODE, int MK, bool DOT, int EPI = EPI_PLAIN, bool COH = false>
__device__ void grid_interior(const GridCoef<T>& P, int item, const T* __restrict__ in,
                              const T* __restrict__ vin, const uint8_t* __restrict__ fixed,
                              T* __restrict__ y, typename Vec4<T>::type* sm, GridDotAcc<T>& dot,
                              const T* __restrict__ bres = nullptr) {
  using V4 = typename Vec4<T>::type;
  const int tid = group_tid<T, COH>();
  const int nx = P.nx, ny = P.ny, nz = P.nz;
  const int tx = item % P.tiles_x;
  const int rest = item / P.tiles_x;
  const int ty = rest % P.tiles_y;
  const int tzi = rest / P.tiles_y;
  const int x0 = 1 + tx * GR_TX, y0 = 1 + ty * GR_TY;
  const int zs = tzi * P.tz, ze = min(zs + P.tz, nz);
  const int ps = max(zs - 1, 0), pe = min(ze, nz - 1);
  const int lx = tid % GR_TX, ly = tid / GR_TX;
  const int x = x0 + lx, yy = y0 + ly;
  const bool own = (x <= nx - 2) && (yy <= ny - 2);
  const int64_t plane_nodes = (int64_t)nx * ny;
  constexpr int GR_THREADS = grid_threads<T>();
  constexpr int GR_SLOTS = (GR_PLANE + GR_THREADS - 1) / GR_THREADS;

  // staged slots of this thread: s = tid + k * GR_THREADS < GR_PLANE
  int64_t soff[GR_SLOTS];  // node offset within a plane, -1: outside the grid / no slot
#pragma unroll
  for (int k = 0; k < GR_SLOTS; ++k) {
    const int s = tid + k * GR_THREADS;
    soff[k] = -1;
    if (s < GR_PLANE) {
      const int gx = x0 - 1 + s % GR_PX, gy = y0 - 1 + s / GR_PX;
      if (gx < nx && gy < ny) soff[k] = gx + (int64_t)nx * gy;
    }
  }
  // raw values and mask bits stay in registers until the plane is stored, so that no
  // load is waited for before then (the prefetch distance is two planes)
  auto load_plane = [&](int p, T (&r)[GR_SLOTS][3], int (&m)[GR_SLOTS]) {
#pragma unroll
    for (int k = 0; k < GR_SLOTS; ++k) {
      m[k] = 0;
#pragma unroll
      for (int d = 0; d < 3; ++d) r[k][d] = T(0);
      if (soff[k] >= 0 && p <= pe) {
        const int64_t g = soff[k] + plane_nodes * p;
        if (masks_input<MODE, MK>()) m[k] = mask_bits<MK>(fixed, g);
#pragma unroll
        for (int d = 0; d < 3; ++d) r[k][d] = ld_in<COH>(in + 3 * g + d);
      }
    }
  };
  auto store_plane = [&](V4* buf, const T (&r)[GR_SLOTS][3], const int (&m)[GR_SLOTS]) {
#pragma unroll
    for (int k = 0; k < GR_SLOTS; ++k) {
      const int s = tid + k * GR_THREADS;
      if (s < GR_PLANE)
        buf[s] = make4<T>((m[k] & 1) ? T(0) : r[k][0], (m[k] & 2) ? T(0) : r[k][1],
                          (m[k] & 4) ? T(0) : r[k][2]);
    }
  };

  T accM[3], accP[3], accN[3];  // outputs at z - 1, z, z + 1 of the current plane z
#pragma unroll
  for (int a = 0; a < 3; ++a) accM[a] = accP[a] = accN[a] = T(0);
  const int c0 = (lx + 1) + GR_PX * (ly + 1);

  T ctr[3];  // the column's value in the current plane
  // A warp whose row of columns is outside the grid has nothing to add: its arithmetic would
  // only take the FP64 pipe from the others' (4^3, three of eight rows exist: HVP 23 -> 13 us;
  // in the persistent CG, whose CTAs hold one tile, the branch costs 3 % at 96^3).  A face
  // plane that is another tile's output counts as an inner one.
  const bool row = COH || yy <= ny - 2;
  auto plane_step = [&](const V4* buf, int p) {
    const int side = p == 0 && zs == 0 ? 1 : (p == nz - 1 && ze == nz ? -1 : 0);
    if (row) stencil_plane<T>(P, buf, c0, accM, accP, accN, ctr, side);
  };

  // pc: the node's own input (the column's value in the output plane, masked): with
  // DOT the product input . output of the owned dofs (fixed dofs: their unmasked input,
  // which is also their output) enters the CTA's dot partial
  // the output node's mask bits, loaded one plane before its emission
  auto out_mask = [&](int z) {
    return (own && z >= zs && z < ze) ? mask_bits<MK>(fixed, x + (int64_t)nx * yy + plane_nodes * z)
                                      : 0;
  };
  auto emit = [&](int z, const T (&acc)[3], const T (&pc)[3], int m) {
    if (!own || z < zs || z >= ze) return;
    const int64_t g = x + (int64_t)nx * yy + plane_nodes * z, base = 3 * g;
    T pvs[3], vals[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      T val = acc[d], pv = pc[d];
      if (m >> d & 1) {
        val = (MODE == TG_MODE_HVP) ? ld_in<COH>(vin + base + d) : T(0);
        pv = val;
      }
      if constexpr (EPI == EPI_RESID) {
        val = __ldg(bres + base + d) - val;
        pv = val;
      }
      y[base + d] = val;
      pvs[d] = pv;
      vals[d] = val;
    }
    if constexpr (DOT) dot.add3(pvs, vals);
  };

  V4* buf0 = sm;
  V4* buf1 = sm + GR_PLANE;
  T rA[GR_SLOTS][3], rB[GR_SLOTS][3];
  int mA[GR_SLOTS], mB[GR_SLOTS];
  auto shift = [&]() {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      accM[a] = accP[a];
      accP[a] = accN[a];
      accN[a] = T(0);
    }
  };
  // prologue: plane ps into buf0; ps + 1 in flight in rB, ps + 2 in rA
  load_plane(ps, rA, mA);
  store_plane(buf0, rA, mA);
  load_plane(ps + 1, rB, mB);
  load_plane(ps + 2, rA, mA);
  int m_out = out_mask(ps - 1);  // mask of the node emitted after the next plane
  group_sync<T, COH>();
  // planes p = ps .. pe, two per trip: buf0 holds p, buf1 gets p + 1
  ctr[0] = ctr[1] = ctr[2] = T(0);
  for (int p = ps; p <= pe; p += 2) {
    T pc[3] = {ctr[0], ctr[1], ctr[2]};
    int m_now = m_out;
    m_out = out_mask(p);
    plane_step(buf0, p);
    emit(p - 1, accM, pc, m_now);
    shift();
    store_plane(buf1, rB, mB);
    load_plane(p + 3, rB, mB);
    group_sync<T, COH>();
    if (p + 1 > pe) break;
#pragma unroll
    for (int a = 0; a < 3; ++a) pc[a] = ctr[a];
    m_now = m_out;
    m_out = out_mask(p + 1);
    plane_step(buf1, p + 1);
    emit(p, accM, pc, m_now);
    shift();
    store_plane(buf0, rA, mA);
    load_plane(p + 4, rA, mA);
    group_sync<T, COH>();
  }
  if (ze == nz) emit(nz - 1, accM, ctr, m_out);  // the high z face: no plane above it
}

// ------------------------------------------------------------------ FP32 interior
// The FP32 sweep is bound by its issued instructions, so a thread owns two node columns
// (rows ly and ly + GP_HALF of the tile) in the two lanes of f32x2 arithmetic: one packed
// instruction serves both, and a plane is staged with the two rows' values of a component
// next to each other, so a neighbour costs one 16-byte and one 8-byte shared load for the
// pair.  Planes arrive by 4-byte cp.async, GP_STAGES - 1 ahead, without holding registers;
// one barrier per plane.
// HVP of a brick without / with a Dirichlet mask, the launch alone (graph replays; the call at
// 128^3 takes 32.8 us), against a column per thread staged through registers and
// element-matrix sums on all faces: 64^3 7.3 / 9.8 -> 6.6 / 8.9 us, 96^3 15.2 /
// 22.0 -> 12.8 / 18.2, 128^3 26.8 / 39.0 -> 22.7 / 30.5 us.  f32x2 runs at the scalar lane
// rate on this chip (128 lane operations a clock and SM); what it saves is issue slots, of
// which a plane of 64 nodes takes 330 (18 shared loads, 10 copies, 143 on the FMA pipe).
//
// Difference form: every block row of the stencil sums to zero (a rigid translation has no
// stiffness), so each in-plane neighbour enters as its difference to the column's value in
// that plane, and the column's own values enter as the second difference along z with the
// in-plane row sum R1 of the |dz| = 1 coefficients.  For smooth fields this keeps the FP32
// result as accurate as its rounded input allows (the value form loses a factor of ~1/h^2
// to cancellation).
struct GridPairCoef {
  f2 c[3][6];  // P.c[a][1], [2], [3], [5], [6], [7]
  f2 r1[3], qxy[2], qxz[2], qyz[2], kxz[2], kyz[2];
  __device__ __forceinline__ void set(const GridCoef<float>& P) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        c[a][i] = f2_bcast(P.c[a][1 + i]);
        c[a][3 + i] = f2_bcast(P.c[a][5 + i]);
      }
      r1[a] = f2_bcast(P.r1[a]);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      qxy[i] = f2_bcast(P.qxy[i]);
      qxz[i] = f2_bcast(P.qxz[i]);
      qyz[i] = f2_bcast(P.qyz[i]);
      kxz[i] = f2_bcast(P.kxz[i]);
      kyz[i] = f2_bcast(P.kyz[i]);
    }
  }
};

// One plane of the sweep for the column pair at slot c0.  below, here: what the planes so far
// add to the outputs below this plane and in it; on return out is the finished output below
// the plane, below and here are those sums for the next plane.  prev: the pair's values in
// the previous plane (updated); side: +1 on the low, -1 on the high z face, else 0.
__device__ __forceinline__ void pair_plane(const GridPairCoef& K, const GridPairStage& S, int c0,
                                           f2 (&below)[3], f2 (&here)[3], f2 (&prev)[3],
                                           f2 (&out)[3], int side) {
  auto load = [&](int s, f2 (&v)[3]) {
    const ulonglong2 xy = S.xy[s];
    v[0].v = xy.x;
    v[1].v = xy.y;
    v[2].v = S.z[s];
  };
  f2 a0[3], xm[3], xp[3], ym[3], yp[3], mm[3], pm[3], mp[3], pp[3];
  load(c0, a0);
  load(c0 - 1, xm);
  load(c0 + 1, xp);
  load(c0 - GR_PX, ym);
  load(c0 + GR_PX, yp);
  load(c0 - GR_PX - 1, mm);
  load(c0 - GR_PX + 1, pm);
  load(c0 + GR_PX - 1, mp);
  load(c0 + GR_PX + 1, pp);
  f2 own[3], next[3];  // to the outputs in this plane, and the even part to those next to it
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const f2 gx = (xm[a] - a0[a]) + (xp[a] - a0[a]);
    const f2 gy = (ym[a] - a0[a]) + (yp[a] - a0[a]);
    const f2 gc = ((mm[a] - a0[a]) + (mp[a] - a0[a])) + ((pm[a] - a0[a]) + (pp[a] - a0[a]));
    own[a] = fma2(K.c[a][2], gc, fma2(K.c[a][1], gy, K.c[a][0] * gx));
    next[a] = fma2(K.c[a][5], gc, fma2(K.c[a][4], gy, K.c[a][3] * gx));
    const f2 dz = a0[a] - prev[a];
    out[a] = fma2(K.r1[a], dz, below[a]);
    below[a] = fma2(K.r1[a], prev[a] - a0[a], here[a]);
    prev[a] = a0[a];
  }
  // x-y blocks: C = qxy(|dz|) dx dy, the cross sum of the in-plane corners; x-z blocks: C =
  // qxz(|dy|) dx dz, odd in x; y-z blocks: C = qyz(|dx|) dy dz, odd in y
  const f2 dl = pm[0] - mm[0], du = pp[0] - mp[0];
  const f2 el = mp[1] - mm[1], er = pp[1] - pm[1];
  const f2 wx = du - dl, wy = er - el;
  own[0] = fma2(K.qxy[0], wy, own[0]);
  own[1] = fma2(K.qxy[0], wx, own[1]);
  next[0] = fma2(K.qxy[1], wy, next[0]);
  next[1] = fma2(K.qxy[1], wx, next[1]);
  const f2 zx1 = (pm[2] - mm[2]) + (pp[2] - mp[2]), zx0 = xp[2] - xm[2];
  const f2 xx1 = dl + du, xx0 = xp[0] - xm[0];
  const f2 zy1 = (mp[2] - mm[2]) + (pp[2] - pm[2]), zy0 = yp[2] - ym[2];
  const f2 yy1 = el + er, yy0 = yp[1] - ym[1];
  if (side) {  // half the interior's own-plane entries and the corner entries of G_z
    const f2 h = f2_bcast(0.5f), sg = f2_bcast((float)side), ng = f2_bcast(-(float)side);
    own[0] = fma2(sg, fma2(K.kxz[1], zx1, K.kxz[0] * zx0), h * own[0]);
    own[1] = fma2(sg, fma2(K.kyz[1], zy1, K.kyz[0] * zy0), h * own[1]);
    own[2] = fma2(ng, fma2(K.kxz[1], xx1, K.kxz[0] * xx0) + fma2(K.kyz[1], yy1, K.kyz[0] * yy0),
                  h * own[2]);
  }
  // odd in z: dz = plane - output is +1 for the output below, -1 for the one above
  f2 odd[3];
  odd[0] = fma2(K.qxz[1], zx1, K.qxz[0] * zx0);
  odd[1] = fma2(K.qyz[1], zy1, K.qyz[0] * zy0);
  odd[2] = fma2(K.qxz[1], xx1, K.qxz[0] * xx0) + fma2(K.qyz[1], yy1, K.qyz[0] * yy0);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    out[a] = out[a] + (next[a] + odd[a]);
    below[a] = below[a] + own[a];
    here[a] = next[a] - odd[a];
  }
}

// The mask of one node as loaded: a node byte (MASK_NODE*), or the aligned words that hold
// the three dof bytes at p (the second only where byte p + 2 lies in it, so that nothing
// beyond the mask's own words is read).  Kept raw until it is applied, a plane later.
template <int MK>
struct RawMask {
  unsigned lo = 0, hi = 0;
  __device__ __forceinline__ void load(const uint8_t* __restrict__ fixed, int64_t n) {
    if constexpr (MK == MASK_DOF) {
      const uintptr_t a = reinterpret_cast<uintptr_t>(fixed + 3 * n);
      const unsigned* w = reinterpret_cast<const unsigned*>(a & ~uintptr_t(3));
      lo = __ldg(w);
      hi = (a & 3) > 1 ? __ldg(w + 1) : 0u;
    } else {
      lo = __ldg(fixed + n);
    }
  }
  __device__ __forceinline__ bool any() const { return (lo | hi) != 0; }  // may be a neighbour's
  // bit d: dof d of node n is fixed
  __device__ __forceinline__ unsigned bits(const uint8_t* __restrict__ fixed, int64_t n) const {
    if constexpr (MK == MASK_DOF) {
      const unsigned sh = (unsigned)(reinterpret_cast<uintptr_t>(fixed + 3 * n) & 3) * 8;
      const unsigned m = __funnelshift_r(lo, hi, sh);
      return ((m & 0xffu) != 0) | ((m & 0xff00u) != 0) << 1 | ((m & 0xff0000u) != 0) << 2;
    } else {
      return lo;
    }
  }
};

template <int MODE, int MK, bool DOT, bool COH = false>
__device__ void grid_interior_pair(const GridCoef<float>& P, int item,
                                   const float* __restrict__ in, const float* __restrict__ vin,
                                   const uint8_t* __restrict__ fixed, float* __restrict__ y,
                                   GridPairStage* stage, GridDotAcc<float>& dot) {
  constexpr bool MASK_IN = masks_input<MODE, MK>();
  constexpr int NT = grid_threads<float>();
  const int tid = group_tid<float, COH>();
  const int nx = P.nx, ny = P.ny, nz = P.nz;
  const int tx = item % P.tiles_x;
  const int rest = item / P.tiles_x;
  const int ty = rest % P.tiles_y;
  const int tzi = rest / P.tiles_y;
  const int x0 = 1 + tx * GR_TX, y0 = 1 + ty * GR_TY;
  const int zs = tzi * P.tz, ze = min(zs + P.tz, nz);
  const int ps = max(zs - 1, 0), pe = min(ze, nz - 1);
  const int lx = tid % GR_TX, ly = tid / GR_TX;
  const int x = x0 + lx, ya = y0 + ly, yb = ya + GP_HALF;
  const bool own_a = x <= nx - 2 && ya <= ny - 2, own_b = x <= nx - 2 && yb <= ny - 2;
  const int64_t plane_nodes = (int64_t)nx * ny;

  // node copies of this thread: entry t = tid + k NT < 2 GP_SLOTS is slot t % GP_SLOTS of
  // half t / GP_SLOTS.  goff: its node's offset within a plane (0 where there is no entry or
  // the node lies outside the grid), sxy / sz: shared-memory addresses in stage 0 of its x and
  // z word; bit k of valid: the entry is copied.  Copies outside the grid stay zero.
  unsigned goff[GP_ENTRIES], sxy[GP_ENTRIES];
  unsigned valid = 0;
  const unsigned stage0 = (unsigned)__cvta_generic_to_shared(stage);
  constexpr unsigned Z_OF = offsetof(GridPairStage, z), ST = sizeof(GridPairStage);
#pragma unroll
  for (int k = 0; k < GP_ENTRIES; ++k) {
    const int t = tid + k * NT;
    const int half = t >= GP_SLOTS, s = t - half * GP_SLOTS;
    const int gx = x0 - 1 + s % GR_PX, gy = y0 - 1 + s / GR_PX + half * GP_HALF;
    const bool slot = t < 2 * GP_SLOTS, in_grid = slot && gx < nx && gy < ny;
    goff[k] = in_grid ? (unsigned)(gx + nx * gy) : 0u;
    sxy[k] = stage0 + 16 * s + 4 * half;
    if (in_grid) valid |= 1u << k;
    if (slot && !in_grid) {
#pragma unroll
      for (int i = 0; i < GP_STAGES; ++i) {
        float* q = reinterpret_cast<float*>(stage[i].xy + s) + half;
        q[0] = 0.f;
        q[2] = 0.f;
        reinterpret_cast<float*>(stage[i].z + s)[half] = 0.f;
      }
    }
  }
  // z word of entry k: 8 bytes a slot, from its xy address (16 bytes a slot)
  auto sz = [&](int k) {
    const unsigned d = sxy[k] - stage0;
    return stage0 + Z_OF + ((d >> 4) << 3) + (d & 15u);
  };
  auto copy = [&](unsigned dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
  };
  auto issue = [&](int p, int st) {
    if (p <= pe) {
      const float* src = in + 3 * plane_nodes * p;
#pragma unroll
      for (int k = 0; k < GP_ENTRIES; ++k)
        if (valid >> k & 1) {
          const float* g = src + 3 * (size_t)goff[k];
          const unsigned d = sxy[k] + st * ST;
          copy(d, g);
          copy(d + 8, g + 1);
          copy(sz(k) + st * ST, g + 2);
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // Dirichlet masks of plane p's copies, loaded one plane before they are applied
  RawMask<MK> mw[MASK_IN ? GP_ENTRIES : 1];
  auto load_masks = [&](int p) {
    if constexpr (MASK_IN) {
#pragma unroll
      for (int k = 0; k < GP_ENTRIES; ++k)
        if ((valid >> k & 1) && p <= pe) mw[k].load(fixed, plane_nodes * p + goff[k]);
    }
  };
  auto apply_masks = [&](int p, int st) {
    if constexpr (MASK_IN) {
#pragma unroll
      for (int k = 0; k < GP_ENTRIES; ++k)
        if (mw[k].any()) {
          const unsigned m = mw[k].bits(fixed, plane_nodes * p + goff[k]);
          const unsigned d = sxy[k] + st * ST;
          if (m & 1) asm volatile("st.shared.f32 [%0], 0f00000000;" ::"r"(d) : "memory");
          if (m & 2) asm volatile("st.shared.f32 [%0], 0f00000000;" ::"r"(d + 8) : "memory");
          if (m & 4) asm volatile("st.shared.f32 [%0], 0f00000000;" ::"r"(sz(k) + st * ST) : "memory");
        }
    }
  };

  GridPairCoef K;
  K.set(P);
  const int c0 = (lx + 1) + GR_PX * (ly + 1);
  f2 below[3], here[3], prev[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) below[a] = here[a] = prev[a] = f2_zero();

  const int64_t na = x + (int64_t)nx * ya, nb = na + (int64_t)nx * GP_HALF;
  // masks of the pair's nodes in plane z
  struct OutMask {
    RawMask<MK> a, b;
  };
  auto out_mask = [&](int z) {
    OutMask m;
    if constexpr (MK != MASK_NONE) {
      if (z >= zs && z < ze) {
        if (own_a) m.a.load(fixed, na + plane_nodes * z);
        if (own_b) m.b.load(fixed, nb + plane_nodes * z);
      }
    }
    return m;
  };
  auto emit_node = [&](int64_t n, float (&val)[3], float (&pv)[3], const RawMask<MK>& raw) {
    if (MK != MASK_NONE && raw.any()) {
      const unsigned m = raw.bits(fixed, n);
#pragma unroll
      for (int d = 0; d < 3; ++d)
        if (m >> d & 1) {
          val[d] = (MODE == TG_MODE_HVP) ? ld_in<COH>(vin + 3 * n + d) : 0.f;
          pv[d] = val[d];
        }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) y[3 * n + d] = val[d];
    if constexpr (DOT) dot.add3(pv, val);
  };
  auto emit = [&](int z, const f2 (&out)[3], const f2 (&pc)[3], const OutMask& m) {
    float a[3], b[3], ca[3], cb[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      f2_split(out[d], a[d], b[d]);
      f2_split(pc[d], ca[d], cb[d]);
    }
    if (own_a) emit_node(na + plane_nodes * z, a, ca, m.a);
    if (own_b) emit_node(nb + plane_nodes * z, b, cb, m.b);
  };

  if constexpr (MASK_IN) load_masks(ps);
#pragma unroll
  for (int i = 0; i < GP_STAGES - 1; ++i) issue(ps + i, i);
  OutMask m_out;          // masks of the nodes emitted after the next plane
  int st = 0;             // stage of plane p
  for (int p = ps; p <= pe; ++p) {
    asm volatile("cp.async.wait_group %0;" ::"n"(GP_STAGES - 2) : "memory");
    apply_masks(p, st);
    // plane p complete; every thread is done with the stage refilled below
    group_sync<float, COH>();
    issue(p + GP_STAGES - 1, (st + GP_STAGES - 1) % GP_STAGES);
    if constexpr (MASK_IN) load_masks(p + 1);
    const GridPairStage& S = stage[st];
    if (p == ps) {  // no z difference to a plane below (at the low face there is none;
                    // elsewhere the first plane's outputs are another tile's)
      prev[0].v = S.xy[c0].x;
      prev[1].v = S.xy[c0].y;
      prev[2].v = S.z[c0];
    }
    const OutMask m_now = m_out;
    m_out = out_mask(p);
    const f2 pc[3] = {prev[0], prev[1], prev[2]};  // the pair's values in plane p - 1
    f2 out[3];
    // (a face plane that is another tile's output counts as an inner one)
    pair_plane(K, S, c0, below, here, prev, out,
               p == 0 && zs == 0 ? 1 : (p == nz - 1 && ze == nz ? -1 : 0));
    if (p > zs) emit(p - 1, out, pc, m_now);
    st = (st + 1) % GP_STAGES;
  }
  if (ze == nz) emit(nz - 1, below, prev, m_out);  // the high z face: no plane above it
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// Edge node t: the four edges along x with their corners (4 nx), then those along y
// (4 (ny - 2)) and z (4 (nz - 2)).
__device__ __forceinline__ void edge_node(int t, int nx, int ny, int nz, int& x, int& y, int& z) {
  if (t < 4 * nx) {
    const int e = t / nx;
    x = t - e * nx;
    y = (e & 1) ? ny - 1 : 0;
    z = (e & 2) ? nz - 1 : 0;
    return;
  }
  t -= 4 * nx;
  if (t < 4 * (ny - 2)) {
    const int e = t / (ny - 2);
    y = 1 + t - e * (ny - 2);
    x = (e & 1) ? nx - 1 : 0;
    z = (e & 2) ? nz - 1 : 0;
    return;
  }
  t -= 4 * (ny - 2);
  const int e = t / (nz - 2);
  z = 1 + t - e * (nz - 2);
  x = (e & 1) ? nx - 1 : 0;
  y = (e & 2) ? ny - 1 : 0;
}
__host__ __device__ inline int edge_nodes(int nx, int ny, int nz) {
  return 4 * nx + 4 * (ny - 2) + 4 * (nz - 2);
}

// Output of a face node: the Dirichlet rows, the residual epilogue and the dot.
template <class T, int MODE, int MK, bool DOT, int EPI, bool COH>
__device__ __forceinline__ void grid_emit_node(int x, int yy, int z, int nx, int ny,
                                               const T (&acc)[3], const T* __restrict__ in,
                                               const T* __restrict__ vin,
                                               const uint8_t* __restrict__ fixed,
                                               T* __restrict__ y, GridDotAcc<T>& dot,
                                               const T* __restrict__ bres) {
  const int64_t gn = x + (int64_t)nx * (yy + (int64_t)ny * z), base = 3 * gn;
  const int mn = mask_bits<MK>(fixed, gn);
  T pvs[3], vals[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    T val = acc[d];
    T pv = T(0);
    if constexpr (DOT && EPI == EPI_PLAIN) pv = ld_in<COH>(in + base + d);
    if (mn >> d & 1) {
      val = (MODE == TG_MODE_HVP) ? ld_in<COH>(vin + base + d) : T(0);
      pv = val;
    }
    if constexpr (EPI == EPI_RESID) {
      val = __ldg(bres + base + d) - val;
      pv = val;
    }
    y[base + d] = val;
    pvs[d] = pv;
    vals[d] = val;
  }
  if constexpr (DOT) dot.add3(pvs, vals);
}

// Edge nodes: the sum over the cells that exist around the node of the element matrix times
// the cell's input values.  P.edge_lanes lanes per node share its cells (added in a fixed
// tree): eight where one brick's latency counts (a thread walking the cells one after the
// other took 8,800 clocks, the longest path of a small brick's HVP), one in launches shared by
// many bricks, whose CTA count costs more (64 bricks in flight: 333 against 347 ms).
template <class T, int MODE, int MK, bool DOT, int EPI = EPI_PLAIN, bool COH = false>
__device__ void grid_edges(const GridCoef<T>& P, int b, const T* __restrict__ in,
                           const T* __restrict__ vin, const uint8_t* __restrict__ fixed,
                           T* __restrict__ y, T* ke, GridDotAcc<T>& dot,
                           const T* __restrict__ bres = nullptr) {
  for (int i = group_tid<T, COH>(); i < 8 * 8 * 9; i += grid_threads<T>())
    ke[i] = (&P.ke[0][0][0][0])[i];
  group_sync<T, COH>();
  const int nx = P.nx, ny = P.ny, nz = P.nz, lanes = P.edge_lanes;
  const int t = (b * grid_threads<T>() + group_tid<T, COH>()) / lanes, n = edge_nodes(nx, ny, nz);
  int x, yy, z;
  edge_node(t < n ? t : n - 1, nx, ny, nz, x, yy, z);
  const int lane = group_tid<T, COH>() & (lanes - 1);
  T acc[3] = {T(0), T(0), T(0)};
  for (int o = lane; o < 8; o += lanes) {  // cell whose corner o is this node
    const int cx = x - (o & 1), cy = yy - ((o >> 1) & 1), cz = z - (o >> 2);
    if (cx < 0 || cy < 0 || cz < 0 || cx >= nx - 1 || cy >= ny - 1 || cz >= nz - 1) continue;
    const T* kr = ke + o * 72;  // rows of corner o: [cm][a][b]
#pragma unroll
    for (int cm = 0; cm < 8; ++cm) {
      const int64_t g = (cx + (cm & 1)) + (int64_t)nx * ((cy + ((cm >> 1) & 1)) +
                                                         (int64_t)ny * (cz + (cm >> 2)));
      const int m = masks_input<MODE, MK>() ? mask_bits<MK>(fixed, g) : 0;
      const T v0 = (m & 1) ? T(0) : ld_in<COH>(in + 3 * g);
      const T v1 = (m & 2) ? T(0) : ld_in<COH>(in + 3 * g + 1);
      const T v2 = (m & 4) ? T(0) : ld_in<COH>(in + 3 * g + 2);
      const T* k9 = kr + cm * 9;
#pragma unroll
      for (int a = 0; a < 3; ++a)
        acc[a] = fma(k9[3 * a + 2], v2, fma(k9[3 * a + 1], v1, fma(k9[3 * a], v0, acc[a])));
    }
  }
  for (int s = lanes >> 1; s > 0; s >>= 1)
#pragma unroll
    for (int a = 0; a < 3; ++a) acc[a] += __shfl_down_sync(0xffffffffu, acc[a], s, lanes);
  if (lane == 0 && t < n)
    grid_emit_node<T, MODE, MK, DOT, EPI, COH>(x, yy, z, nx, ny, acc, in, vin, fixed, y, dot, bres);
}

// Nodes of the y faces (1 <= x <= nx - 2, 1 <= z <= nz - 2), one per thread, consecutive
// threads consecutive along x: the corner loads coalesce.
template <class T, int MODE, int MK, bool DOT, int EPI = EPI_PLAIN, bool COH = false>
__device__ void grid_yface(const GridCoef<T>& P, int64_t t0, const T* __restrict__ in,
                           const T* __restrict__ vin, const uint8_t* __restrict__ fixed,
                           T* __restrict__ y, GridDotAcc<T>& dot,
                           const T* __restrict__ bres = nullptr) {
  const int nx = P.nx, ny = P.ny, nz = P.nz;
  const int64_t per = (int64_t)(nx - 2) * (nz - 2);
  int64_t t = t0 + group_tid<T, COH>();
  if (t >= 2 * per) return;
  const int high = t >= per;
  if (high) t -= per;
  const int x = 1 + (int)(t % (nx - 2)), z = 1 + (int)(t / (nx - 2));
  const int yb = high ? ny - 2 : 0;  // first of the two node rows
  T acc[3] = {T(0), T(0), T(0)};
  auto stencil = [&](auto side) {
    constexpr int S = decltype(side)::value;
#pragma unroll
    for (int row = 0; row < 2; ++row)
#pragma unroll
      for (int j = 0; j < 9; ++j) {
        const int64_t g = (x + j % 3 - 1) + (int64_t)nx * ((yb + row) + (int64_t)ny * (z + j / 3 - 1));
        const int m = masks_input<MODE, MK>() ? mask_bits<MK>(fixed, g) : 0;
        const T v0 = (m & 1) ? T(0) : ld_in<COH>(in + 3 * g);
        const T v1 = (m & 2) ? T(0) : ld_in<COH>(in + 3 * g + 1);
        const T v2 = (m & 4) ? T(0) : ld_in<COH>(in + 3 * g + 2);
#pragma unroll
        for (int a = 0; a < 3; ++a)
          acc[a] = fma(P.fy[S][row][j][a][2], v2,
                       fma(P.fy[S][row][j][a][1], v1, fma(P.fy[S][row][j][a][0], v0, acc[a])));
      }
  };
  if (high) stencil(std::integral_constant<int, 1>{});
  else stencil(std::integral_constant<int, 0>{});
  grid_emit_node<T, MODE, MK, DOT, EPI, COH>(x, high ? ny - 1 : 0, z, nx, ny, acc, in, vin, fixed, y,
                                        dot, bres);
}

// Nodes of the two x faces (x = 0 and x = nx - 1, 1 <= y <= ny - 2, 1 <= z <= nz - 2),
// a GR_XT x grid_xt_z patch (y, z) per CTA.  On these faces consecutive nodes are a grid
// row apart, so per-thread corner loads would touch one cache line per thread; the CTA
// instead stages the two node columns next to the face (x = 0, 1 or nx - 2, nx - 1)
// of its patch and halo, row by row (contiguous 24-byte runs), masked on the way.
template <class T, int MODE, int MK, bool DOT, int EPI = EPI_PLAIN, bool COH = false>
__device__ void grid_xface(const GridCoef<T>& P, int item, const T* __restrict__ in,
                           const T* __restrict__ vin, const uint8_t* __restrict__ fixed,
                           T* __restrict__ y, typename Vec4<T>::type* sm, GridDotAcc<T>& dot,
                           const T* __restrict__ bres = nullptr) {
  using V4 = typename Vec4<T>::type;
  const int nx = P.nx, ny = P.ny, nz = P.nz;
  const int per_face = P.xt_y * P.xt_z;
  const int face = item / per_face, rest = item - face * per_face;
  const int ty = rest % P.xt_y, tz = rest / P.xt_y;
  const int xb = face ? nx - 2 : 0;  // first of the two staged columns
  const int y0 = 1 + ty * GR_XT, z0 = 1 + tz * grid_xt_z<T>();
  // slot s = 2 (rz GR_XS + ry) + col: node (xb + col, y0 - 1 + ry, z0 - 1 + rz)
  for (int s = group_tid<T, COH>(); s < 2 * GR_XS * (grid_xt_z<T>() + 2); s += grid_threads<T>()) {
    const int col = s & 1, r = s >> 1;
    const int gy = y0 - 1 + r % GR_XS, gz = z0 - 1 + r / GR_XS;
    T v0 = T(0), v1 = T(0), v2 = T(0);
    if (gy < ny && gz < nz) {
      const int64_t g = (xb + col) + (int64_t)nx * (gy + (int64_t)ny * gz);
      const int m = masks_input<MODE, MK>() ? mask_bits<MK>(fixed, g) : 0;
      v0 = (m & 1) ? T(0) : ld_in<COH>(in + 3 * g);
      v1 = (m & 2) ? T(0) : ld_in<COH>(in + 3 * g + 1);
      v2 = (m & 4) ? T(0) : ld_in<COH>(in + 3 * g + 2);
    }
    sm[s] = make4<T>(v0, v1, v2);
  }
  group_sync<T, COH>();
  const int ly = group_tid<T, COH>() % GR_XT, lz = group_tid<T, COH>() / GR_XT;
  const int yy = y0 + ly, z = z0 + lz;
  if (yy > ny - 2 || z > nz - 2) return;
  T acc[3] = {T(0), T(0), T(0)};
  auto stencil = [&](auto side) {
    constexpr int S = decltype(side)::value;
#pragma unroll
    for (int j = 0; j < 9; ++j)
#pragma unroll
      for (int col = 0; col < 2; ++col) {
        const V4 v = sm[2 * ((lz + j / 3) * GR_XS + ly + j % 3) + col];
#pragma unroll
        for (int a = 0; a < 3; ++a)
          acc[a] = fma(P.fx[S][col][j][a][2], v.z,
                       fma(P.fx[S][col][j][a][1], v.y, fma(P.fx[S][col][j][a][0], v.x, acc[a])));
      }
  };
  if (face) stencil(std::integral_constant<int, 1>{});
  else stencil(std::integral_constant<int, 0>{});
  grid_emit_node<T, MODE, MK, DOT, EPI, COH>(face ? nx - 1 : 0, yy, z, nx, ny, acc, in, vin, fixed, y,
                                        dot, bres);
}

// What CTA b of a brick's launch works on (grid_cta's order): the coefficients it reads are
// GridCoef's head and, on faces and edges, one of its arrays.
enum GridPart { GRID_INTERIOR, GRID_XFACE, GRID_YFACE, GRID_EDGE };
template <class T>
__device__ __forceinline__ GridPart grid_part(const GridCoef<T>& P, int b) {
  b -= P.tiles_x * P.tiles_y * P.tiles_z;
  if (b < 0) return GRID_INTERIOR;
  if (b < P.n_xface_ctas) return GRID_XFACE;
  return b - P.n_xface_ctas < P.n_yface_ctas ? GRID_YFACE : GRID_EDGE;
}

// CTA b of a launch over the brick: interior tiles first, then the shorter face and edge CTAs,
// which fill the launch's tail (faces first measured 24.3 instead of 23.3 us at 128^3)
template <class T, int MODE, int MK, bool DOT, int EPI = EPI_PLAIN, bool COH = false>
__device__ __forceinline__ void grid_cta(const GridCoef<T>& P, int b, const T* __restrict__ in,
                                         const T* __restrict__ vin,
                                         const uint8_t* __restrict__ fixed, T* __restrict__ y,
                                         GridShared<T>& sh, GridDotAcc<T>& dot,
                                         const T* __restrict__ bres = nullptr) {
  if (grid_part(P, b) == GRID_INTERIOR) {
    if constexpr (std::is_same<T, float>::value) {
      static_assert(EPI == EPI_PLAIN, "the FP32 launches apply the operator only");
      grid_interior_pair<MODE, MK, DOT, COH>(P, b, in, vin, fixed, y, sh.stage, dot);
    } else {
      grid_interior<T, MODE, MK, DOT, EPI, COH>(P, b, in, vin, fixed, y, sh.sm, dot, bres);
    }
    return;
  }
  b -= P.tiles_x * P.tiles_y * P.tiles_z;
  if (b < P.n_xface_ctas) {
    grid_xface<T, MODE, MK, DOT, EPI, COH>(P, b, in, vin, fixed, y, sh.sm, dot, bres);
    return;
  }
  b -= P.n_xface_ctas;
  if (b < P.n_yface_ctas) {
    grid_yface<T, MODE, MK, DOT, EPI, COH>(P, (int64_t)b * grid_threads<T>(), in, vin, fixed, y, dot,
                                      bres);
    return;
  }
  b -= P.n_yface_ctas;
  grid_edges<T, MODE, MK, DOT, EPI, COH>(P, b, in, vin, fixed, y, sh.ke, dot, bres);
}

// ------------------------------------------------------------------------- host
// Stencil coefficients and the element matrix from the spacings and Lame parameters,
// in FP64, then rounded to T.
template <class T>
static void grid_coefficients(const double h[3], double mu, double lam, GridCoef<T>& P) {
  double K[3][2], M[3][2];
  for (int k = 0; k < 3; ++k) {
    K[k][0] = 2.0 / h[k];
    K[k][1] = -1.0 / h[k];
    M[k][0] = 2.0 * h[k] / 3.0;
    M[k][1] = h[k] / 6.0;
  }
  for (int i = 0; i < 8; ++i) {
    const int ix = i & 1, iy = (i >> 1) & 1, iz = i >> 2;
    const double D[3] = {K[0][ix] * M[1][iy] * M[2][iz], M[0][ix] * K[1][iy] * M[2][iz],
                         M[0][ix] * M[1][iy] * K[2][iz]};
    const double L = D[0] + D[1] + D[2];
    for (int a = 0; a < 3; ++a) P.c[a][i] = (T)(mu * L + (lam + mu) * D[a]);
  }
  for (int a = 0; a < 3; ++a) {
    double r = 0.0;  // sum over dx, dy of c(dx, dy, 1): weights 1, 2, 2, 4 by class
    for (int i = 4; i < 8; ++i) {
      const int ix = i & 1, iy = (i >> 1) & 1;
      const double D[3] = {K[0][ix] * M[1][iy] * M[2][1], M[0][ix] * K[1][iy] * M[2][1],
                           M[0][ix] * M[1][iy] * K[2][1]};
      r += (ix ? 2.0 : 1.0) * (iy ? 2.0 : 1.0) * (mu * (D[0] + D[1] + D[2]) + (lam + mu) * D[a]);
    }
    P.r1[a] = (T)r;
  }
  const double q = -(lam + mu) / 4.0;
  for (int s = 0; s < 2; ++s) {
    P.qxy[s] = (T)(q * M[2][s]);
    P.qxz[s] = (T)(q * M[1][s]);
    P.qyz[s] = (T)(q * M[0][s]);
  }
  for (int st = 0; st < 2; ++st) {
    P.kxz[st] = (T)((lam - mu) / 4.0 * M[1][st]);
    P.kyz[st] = (T)((lam - mu) / 4.0 * M[0][st]);
  }
  double Ke[8][8][3][3];
  // element matrix of one cell: corners cn, cm = lx + 2 ly + 4 lz; per axis the
  // element-level 1-D integrals Kel = [[1,-1],[-1,1]]/h, Mel = h[[1/3,1/6],[1/6,1/3]],
  // Gel(A, B) = int phi_A' phi_B = s_A / 2 (s = -1 at the lower corner, +1 upper)
  for (int cn = 0; cn < 8; ++cn)
    for (int cm = 0; cm < 8; ++cm) {
      int ln[3], lm[3];
      for (int k = 0; k < 3; ++k) {
        ln[k] = (cn >> k) & 1;
        lm[k] = (cm >> k) & 1;
      }
      auto DE = [&](int i, int j) {
        double v = 1.0;
        for (int k = 0; k < 3; ++k) {
          double f;
          if (i == j && j == k) f = (ln[k] == lm[k] ? 1.0 : -1.0) / h[k];
          else if (k == i) f = (ln[k] ? 0.5 : -0.5);
          else if (k == j) f = (lm[k] ? 0.5 : -0.5);
          else f = h[k] * (ln[k] == lm[k] ? 1.0 / 3.0 : 1.0 / 6.0);
          v *= f;
        }
        return v;
      };
      const double Ls = DE(0, 0) + DE(1, 1) + DE(2, 2);
      for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b)
        {
          Ke[cn][cm][a][b] = lam * DE(a, b) + mu * DE(b, a) + (a == b ? mu * Ls : 0.0);
          P.ke[cn][cm][a][b] = (T)Ke[cn][cm][a][b];
        }
    }
  // one-sided stencils of the x and y faces: the four cells around a face node merged.  On
  // side s of axis n the node is corner bit s of its cells along n; along the other axes it
  // is bit o and the neighbour bit m, at offset m - o.
  auto face = [&](int n, T (&F)[2][2][9][3][3]) {
    const int ax = n == 0 ? 1 : 0;  // the in-plane axis beside z
    for (int s = 0; s < 2; ++s) {
      double f[2][9][3][3] = {};
      for (int o = 0; o < 4; ++o)
        for (int cm = 0; cm < 8; ++cm) {
          const int oa = o & 1, oz = o >> 1;
          const int cn = (s << n) + (oa << ax) + (oz << 2);
          const int j = 3 * ((cm >> 2) - oz + 1) + ((cm >> ax) & 1) - oa + 1;
          for (int a = 0; a < 3; ++a)
            for (int b = 0; b < 3; ++b) f[(cm >> n) & 1][j][a][b] += Ke[cn][cm][a][b];
        }
      for (int c = 0; c < 2; ++c)
        for (int j = 0; j < 9; ++j)
          for (int a = 0; a < 3; ++a)
            for (int b = 0; b < 3; ++b) F[s][c][j][a][b] = (T)f[c][j][a][b];
    }
  };
  face(0, P.fx);
  face(1, P.fy);
}

// SMs of the current device (queried once per device).
static int grid_sm_count() {
  static int cached[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 152;
  if (!cached[dev]) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
      n = 152;
    cached[dev] = n;
  }
  return cached[dev];
}

// Coefficients and tiling of a brick of nodes[0] x nodes[1] x nodes[2] nodes with
// spacings h; returns the launch's CTA count (grid_cta's order: interior tiles, x faces, y
// faces, edges), or -1 when it does not fit an int.
// deep: always GR_DEEP_TZ planes per tile (launches shared by many bricks need no spreading
// of one brick over the SMs, and deeper tiles reload fewer halo planes).
// groups > 0: the tiles and faces are shared out among that many groups at once (the
// persistent CG): the fewest planes that leave each at most one, or the rule above.
template <class T>
static int64_t grid_setup_dims(const int32_t nodes[3], const double h[3], double mu, double lam,
                               GridCoef<T>& P, bool deep = false, int64_t groups = 0) {
  const int nx = nodes[0], ny = nodes[1], nz = nodes[2];
  grid_coefficients<T>(h, mu, lam, P);
  P.nx = nx;
  P.ny = ny;
  P.nz = nz;
  const int ix = nx - 2, iy = ny - 2, iz = nz - 2;
  P.tiles_x = ix > 0 ? (ix + GR_TX - 1) / GR_TX : 0;
  P.tiles_y = iy > 0 ? (iy + GR_TY - 1) / GR_TY : 0;
  const int64_t columns = (int64_t)P.tiles_x * P.tiles_y, sms = grid_sm_count();
  auto tiles_of = [&](int64_t tz) { return (nz + tz - 1) / tz; };
  const int64_t nt = grid_threads<T>();
  P.edge_lanes = deep ? 1 : 8;
  const int64_t per_edge = nt / P.edge_lanes;
  const int64_t n_edge = (edge_nodes(nx, ny, nz) + per_edge - 1) / per_edge;
  const int64_t n_y = (2 * (int64_t)ix * iz + nt - 1) / nt;
  P.xt_y = iy > 0 ? (iy + GR_XT - 1) / GR_XT : 0;
  P.xt_z = iz > 0 ? (iz + grid_xt_z<T>() - 1) / grid_xt_z<T>() : 0;
  const int64_t n_x = 2 * (int64_t)P.xt_y * P.xt_z;
  const int64_t faces = n_edge + n_y + n_x;
  // Planes per tile: a tile sweeps its planes one after the other, at a few CTAs per SM
  // mostly waiting on itself, and reloads two halo planes.
  int64_t tz = GR_DEEP_TZ;
  if (!deep && columns > 0) {
    if (sizeof(T) == 4) {
      // two and a half tiles per SM on small grids, at most GR_MAX_TZ planes on large ones
      // (HVP at 64^3: 4 planes 6.1 us, 8 planes 6.6, 12 planes 8.2; 96^3: 10 planes 12.8, 12
      // planes 14.5; 128^3: 15 planes 22.7, 11 planes 23.4, 19 planes 25.6)
      tz = (2 * columns * nz + 5 * sms - 1) / (5 * sms);
      tz = tz < 2 ? 2 : (tz > GR_MAX_TZ ? GR_MAX_TZ : tz);
    } else {
      // Two CTAs share an SM's FP64 pipe: the fewest planes for the busiest SM, in sweep steps
      // (7.2 us each).  One tile per SM costs a step and a half more at most where face CTAs
      // and a short last layer are its neighbours, and 1.6 times its own steps where these
      // are so many that some SMs hold two tiles.  HVP with a mask: 24^3 1 plane 23.9 us, 2
      // planes 31.1; 38^3 4 planes 46.3, 2 planes 57.7; 50^3 5 planes 63.7, 3 planes 71.2;
      // 64^3 7 planes 79.8, 4 planes 85.5; 96^3 13 planes 218, 25 planes 339; 128^3 19
      // planes 451, 13 planes 497.
      double best = -1.0;
      for (int64_t c = 1; c <= 24; ++c) {
        const int64_t tiles = columns * tiles_of(c), last = nz % c;
        const int64_t full = columns * (last == 1 || last == 2 ? nz / c : tiles_of(c));
        const double steps = (double)(c + 2);
        double cost;
        if (full <= sms && 4 * (tiles + faces) <= 7 * sms) {
          cost = tiles + faces <= sms ? steps : steps + (steps < 6.0 ? steps / 4 : 1.5);
        } else {
          const int64_t r = (tiles + sms - 1) / sms;
          cost = (r <= 1 ? 1.6 : (double)r) * steps;
        }
        if (best < 0.0 || cost < best) {
          best = cost;
          tz = c;
        }
      }
    }
    tz = (nz + tiles_of(tz) - 1) / tiles_of(tz);  // the same tiles, of even depth
    if (groups > 0)
      for (int64_t c = 2; c <= GR_MAX_TZ; ++c)
        if (columns * tiles_of(c) + faces <= groups) {
          tz = c;
          break;
        }
  }
  P.tz = (int)tz;
  P.tiles_z = (int)tiles_of(tz);
  const int64_t n_int = columns * P.tiles_z;
  if (n_int + faces > 0x7fffffff) return -1;
  P.n_yface_ctas = (int)n_y;
  P.n_xface_ctas = (int)n_x;
  return n_int + faces;
}

// The same for a structured-brick plan (tg_grid_detect's nodes and spacings).
template <class T>
static int64_t grid_setup(const tg_block_plan* plan, double mu, double lam, GridCoef<T>& P,
                          int64_t groups = 0) {
  return grid_setup_dims<T>(plan->grid_nodes, plan->grid_h, mu, lam, P, false, groups);
}

}  // namespace tg
