// Trilinear (modal) form of the Hex8 cell, shared by the operator maps, the fused
// residual / HVP / energy kernels and the element tangents.
//
// A nodal field on a Hex8 cell is f(xi) = 1/8 sum_m c_m xi^m over the eight monomials m
// of {1, xi1, xi2, xi1 xi2, xi3, xi1 xi3, xi2 xi3, xi1 xi2 xi3} (bit k of m: factor
// xi_{k+1}), with c_m = sum_a (prod_{k in m} s_{a,k}) f_a for the corner signs s_{a,k} of
// tatva/element/base.py:478-491: a three-stage butterfly over the corners.  At the Gauss
// point with coordinates (sx g, sy g, sz g), g = 1/sqrt(3), and with the modes scaled
// once by c_3, c_5, c_6 *= g and c_7 *= g^2,
//   8 df/dxi1 = c_1 + sy c_3 + sz c_5 + sy sz c_7
//   8 df/dxi2 = c_2 + sx c_3 + sz c_6 + sx sz c_7
//   8 df/dxi3 = c_4 + sx c_5 + sy c_6 + sx sy c_7,
// so the two points of a z pair share everything but two additions.  The factor 8
// cancels between the Jacobian and the field (physical gradients are inv(8 J) times 8
// df/dxi) and again on the way back, so it appears only in det J = det(8 J) / 512.
//
// Why: the kernels on this path are bound by their FP64 (or issued FP32) operations.
// Per point and component the reference gradient costs 5.5 additions instead of 24
// multiply-adds over the nodes, and the way back 8.5 instead of 24.
#pragma once

#include "tg_common.cuh"

namespace tg {

// reference node a <-> binary corner (bit k: side along axis k), its own inverse
__host__ __device__ constexpr int hex_bin(int a) { return a ^ ((a >> 1) & 1); }

// corner values in reference order -> modes c_m, unscaled, in place.  The corners enter
// relative to corner 0 (mode 0 is then 8 times the offset of the cell's mean from it):
// the sums stay of the size of the differences across the cell, where sums of absolute
// coordinates would round at eps |x| and lose 3x in the gradients of a fine mesh.
template <class T, int C>
__device__ __forceinline__ void hex_modes8(T (&v)[8][C]) {
#pragma unroll
  for (int c = 0; c < C; ++c) {
    T w[8];
#pragma unroll
    for (int a = 1; a < 8; ++a) w[hex_bin(a)] = v[a][c] - v[0][c];
    w[0] = w[1];  // first stage of corners 0 (zero) and 1
#pragma unroll
    for (int b = 2; b < 8; b += 2) {
      const T x = w[b], y = w[b | 1];
      w[b] = x + y;
      w[b | 1] = y - x;
    }
#pragma unroll
    for (int k = 2; k < 8; k <<= 1)
#pragma unroll
      for (int b = 0; b < 8; ++b)
        if (!(b & k)) {
          const T x = w[b], y = w[b | k];
          w[b] = x + y;
          w[b | k] = y - x;
        }
#pragma unroll
    for (int m = 0; m < 8; ++m) v[m][c] = w[m];
  }
}

// adjoint of hex_modes8: mode weights -> corner contributions in reference order, in place
template <class T, int C>
__device__ __forceinline__ void hex_modes8_adjoint(T (&v)[8][C]) {
#pragma unroll
  for (int c = 0; c < C; ++c) {
    T w[8];
#pragma unroll
    for (int m = 0; m < 8; ++m) w[m] = v[m][c];
#pragma unroll
    for (int k = 1; k < 8; k <<= 1)
#pragma unroll
      for (int b = 0; b < 8; ++b)
        if (!(b & k)) {
          const T x = w[b], y = w[b | k];
          w[b] = x - y;
          w[b | k] = x + y;
        }
#pragma unroll
    for (int a = 0; a < 8; ++a) v[a][c] = w[hex_bin(a)];
  }
}

// the Gauss coordinate folded into the mixed modes (its own adjoint)
template <class T, int C>
__device__ __forceinline__ void hex_scale_gauss(T (&m)[8][C]) {
  const T g = T(HEX_GAUSS), g2 = T(HEX_GAUSS) * T(HEX_GAUSS);
#pragma unroll
  for (int c = 0; c < C; ++c) {
    m[3][c] *= g;
    m[5][c] *= g;
    m[6][c] *= g;
    m[7][c] *= g2;
  }
}

// Sides of the z pair p of Gauss points, p = 0..3 with (sx, sy) = (-,-), (+,-), (+,+),
// (-,+): its points are p (sz = -1) and p + 4 (sz = +1) of the reference order.
template <class T>
__device__ __forceinline__ void hex_pair_sides(int p, T& sx, T& sy) {
  sx = (p == 1 || p == 2) ? T(1) : T(-1);
  sy = (p >= 2) ? T(1) : T(-1);
}

// 8 df/dxi of the field with scaled modes m at the z pair (sx, sy): lo + sz hi
template <class T, int C>
struct HexPair {
  T e0[C], e1[C], f0[C], f1[C], d2[C];
  __device__ __forceinline__ void set(const T (&m)[8][C], T sx, T sy) {
    const T sxy = sx * sy;
#pragma unroll
    for (int c = 0; c < C; ++c) {
      e0[c] = fma(sy, m[3][c], m[1][c]);
      e1[c] = fma(sy, m[7][c], m[5][c]);
      f0[c] = fma(sx, m[3][c], m[2][c]);
      f1[c] = fma(sx, m[7][c], m[6][c]);
      d2[c] = fma(sxy, m[7][c], fma(sy, m[6][c], fma(sx, m[5][c], m[4][c])));
    }
  }
  // D[i][c] at the point with side sz (0: -, 1: +)
  __device__ __forceinline__ void at(int up, T (&D)[3][C]) const {
#pragma unroll
    for (int c = 0; c < C; ++c) {
      D[0][c] = up ? e0[c] + e1[c] : e0[c] - e1[c];
      D[1][c] = up ? f0[c] + f1[c] : f0[c] - f1[c];
      D[2][c] = d2[c];
    }
  }
};

// adjoint of HexPair: F[up][i][c] of the pair's two points added to the scaled-mode
// weights w (hex_scale_gauss, then hex_modes8_adjoint give the corner contributions)
template <class T, int C>
__device__ __forceinline__ void hex_pair_adjoint(const T (&F)[2][3][C], T sx, T sy, T (&w)[8][C]) {
  const T sxy = sx * sy;
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const T s0 = F[1][0][c] + F[0][0][c], d0 = F[1][0][c] - F[0][0][c];
    const T s1 = F[1][1][c] + F[0][1][c], d1 = F[1][1][c] - F[0][1][c];
    const T s2 = F[1][2][c] + F[0][2][c];
    w[1][c] += s0;
    w[2][c] += s1;
    w[4][c] += s2;
    w[3][c] = fma(sx, s1, fma(sy, s0, w[3][c]));
    w[5][c] = fma(sx, s2, w[5][c] + d0);
    w[6][c] = fma(sy, s2, w[6][c] + d1);
    w[7][c] = fma(sxy, s2, fma(sx, d1, fma(sy, d0, w[7][c])));
  }
}

// field value at the point (sx, sy, sz) from its scaled modes and its value at corner 0
template <class T>
__device__ __forceinline__ T hex_value(const T (&m)[8], T corner0, T sx, T sy, T sz) {
  const T g = T(HEX_GAUSS);
  const T mixed = fma(sx * sy, m[3], fma(sx * sz, m[5], fma(sy * sz, m[6], sx * sy * sz * m[7])));
  const T s = fma(g, fma(sx, m[1], fma(sy, m[2], fma(sz, m[4], mixed))), m[0]);
  return fma(T(0.125), s, corner0);
}

// true when the cell is a parallelepiped: no mixed modes, the Jacobian is constant
template <class T>
__device__ __forceinline__ bool hex_constant_jacobian(const T (&mx)[8][3]) {
  bool z = true;
#pragma unroll
  for (int c = 0; c < 3; ++c)
    z = z && mx[3][c] == T(0) && mx[5][c] == T(0) && mx[6][c] == T(0) && mx[7][c] == T(0);
  return z;
}

}  // namespace tg
