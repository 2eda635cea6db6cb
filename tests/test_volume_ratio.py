"""ln of a deformed cell's volume ratio (csrc/tg_volume.h) in FP32 on flat cells.

The tangent of the Neo-Hookean law has lambda ln J, so an error of ln J at a small strain is
multiplied by lambda.  Bound: J = det(I + G) for the strain G; with unit roundoff u the entries
of I + G round at u each, and ln J at 3 u of them plus 3 u of its products and the logarithm:
6 u in all, for any shape of the cell as long as strain times flatness stays below 1/2 (the
strain's own rounding is u times that).
"""

import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
U = 2.0**-24

SOURCE = r"""
#include "tg_volume.h"
extern "C" void ratios(const float (*J)[3][3], const float (*R)[3][3], const float* rdet,
                       const float (*j)[3][3], const float (*r)[3][3], const float* dj,
                       const float (*D)[3][3], int n, float* out) {
  for (int i = 0; i < n; ++i)
    out[i] = tg::log_volume_ratio<float>(J[i], R[i], rdet[i], j[i], r[i], dj[i], D[i]);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("volume")
    src, so = d / "volume.cpp", d / "volume.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    "-I" + os.path.join(ROOT, "tatva_gb300", "csrc"), str(src), "-o", str(so)],
                   check=True)
    return ctypes.CDLL(str(so))


def _inverse(a):
    """Cofactor inverse and determinant in the arithmetic of ``a``'s dtype."""
    c = np.stack([np.cross(a[:, (k + 1) % 3], a[:, (k + 2) % 3]) for k in range(3)], 2)
    det = (a[:, 0] * c[:, :, 0]).sum(1)
    return c / det[:, None, None], det


@pytest.mark.parametrize("flatness", [1, 10, 100])
@pytest.mark.parametrize("strain", [1e-4, 1e-3, 5e-3])
def test_small_strains_on_flat_cells(lib, flatness, strain):
    rng = np.random.default_rng(int(flatness))
    n = 4000
    q = np.linalg.qr(rng.standard_normal((n, 3, 3)))[0]
    J = (np.eye(3) + 0.2 * rng.uniform(-1, 1, (n, 3, 3))) * np.array([1, 1, 1 / flatness]) @ q
    D = (J @ (strain * rng.uniform(-1, 1, (n, 3, 3)))).astype(np.float32)
    J = J.astype(np.float32)
    j = J + D
    R, det = _inverse(J)
    r, dj = _inverse(j)
    out = np.zeros(n, np.float32)
    args = [np.ascontiguousarray(a, dtype=np.float32) for a in (J, R, 1 / det, j, r, dj, D)]
    lib.ratios(*(ctypes.c_void_p(a.ctypes.data) for a in args), n,
               ctypes.c_void_p(out.ctypes.data))
    J64, D64 = J.astype(np.float64), D.astype(np.float64)
    exact = np.log(np.linalg.det(J64 + D64) / np.linalg.det(J64))
    assert np.abs(out - exact).max() <= 6 * U
    if flatness == 100:  # what the bound is about: the quotient of the determinants breaks it
        assert np.abs(np.log(dj / det) - exact).max() > 6 * U
