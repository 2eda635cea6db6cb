// Logarithm of a deformed cell's volume ratio.  Plain C++, so that its rounding is tested on
// the host.
#pragma once

#include <cmath>

#include "tg_sum.h"  // TG_HD

namespace tg {

// ln(det j / det J) of the Jacobians of a cell before (J, inverse R, rdet: reciprocal
// determinant) and after a displacement with reference gradient D = j - J (r, dj: inverse and
// determinant of j), from the difference of the determinants: with the rows J_k, j_k, D_k,
//   det j - det J = D_0.(j_1 x j_2) + D_1.(j_2 x J_0) + D_2.(J_0 x J_1),
// the first and last cross products being columns of the inverses.  It rounds as ln det F does
// with F = I + D R: at eps for small D.  The quotient of the two determinants rounds at eps
// times the cell's flatness whatever the strain, and lambda multiplies it.  FP32, 1 % strain,
// root mean square: ln det F 8e-8; the quotient 8e-8, 1.0e-7 and 4.8e-7 for cells flattened
// 1:1, 10:1 and 100:1; the difference 3e-8 for all three.
template <class T>
TG_HD T log_volume_ratio(const T (&J)[3][3], const T (&R)[3][3], T rdet, const T (&j)[3][3],
                         const T (&r)[3][3], T dj, const T (&D)[3][3]) {
  using std::fma;
  using std::log;
  const T d0 = fma(D[0][2], r[2][0], fma(D[0][1], r[1][0], D[0][0] * r[0][0]));
  const T d2 = fma(D[2][2], R[2][2], fma(D[2][1], R[1][2], D[2][0] * R[0][2]));
  const T c0 = fma(j[2][1], J[0][2], -(j[2][2] * J[0][1]));
  const T c1 = fma(j[2][2], J[0][0], -(j[2][0] * J[0][2]));
  const T c2 = fma(j[2][0], J[0][1], -(j[2][1] * J[0][0]));
  const T d1 = fma(D[1][2], c2, fma(D[1][1], c1, D[1][0] * c0));
  return log(T(1) + fma(dj * rdet, d0, fma(rdet, d1, d2)));
}

}  // namespace tg
