"""The edge-vector Tri3 / Tet4 element and the Neo-Hookean HVP in the deformed cell's axes
against the oracle: one element, scrambled node order, cells away from the origin, large
deformation.

Tolerances (relative, max norm): FP64 1e-12, FP32 1e-4, the repository's bounds of the
fused kernels against the oracle.
"""

import numpy as np
import pytest
import torch

from oracle import elements as oe
from oracle import materials as omat
from oracle import mesh as om
from oracle import operator as oop
from tatva_gb300 import Mesh, Operator, element, materials

pytestmark = pytest.mark.gpu

LAWS = {"linear_elastic": (materials.LinearElastic, omat.LinearElastic, (0.7, 1.9)),
        "poisson": (materials.Poisson, omat.Poisson, (1.3, 0.6)),
        "neo_hookean": (materials.NeoHookean, omat.NeoHookean, (1.0, 10.0))}


def rel(a, b):
    a = a.detach().double().cpu().numpy()
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300))


def _mesh(elem, n, rng):
    if elem == "tri3":
        c, e = om.unit_square(*n[:2])
    elif elem == "tet4":
        c, e = om.kuhn_box((1, 1, 1), n, origin=(0, 0, 0))
    else:
        c, e = om.brick(*n)
    h = 1.0 / max(n)
    c = c + 0.12 * h * rng.uniform(-1, 1, c.shape) + 1.5
    p = rng.permutation(c.shape[0])
    return c[np.argsort(p)], p[e].astype(np.int32)


@pytest.mark.parametrize("elem,n,kind", [
    (el, n, k) for el in ("tri3", "tet4", "hex8") for n in ((1, 1, 1), (5, 3, 4))
    for k in LAWS if not (el == "tri3" and k == "neo_hookean")])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_elements_match_oracle(cuda, elem, n, kind, dtype):
    rng = np.random.default_rng(8)
    c, e = _mesh(elem, n, rng)
    els = {"tri3": (element.Tri3, oe.Tri3), "tet4": (element.Tetrahedron4, oe.Tetrahedron4),
           "hex8": (element.Hexahedron8, oe.Hexahedron8)}[elem]
    op = Operator(Mesh(c, e, device=cuda), els[0]())
    oo = oop.OracleOperator(c, e, els[1]())
    cls, ocls, par = LAWS[kind]
    en = cls(op, *par)
    law = ocls(*par, dim=2) if elem == "tri3" and kind == "linear_elastic" else ocls(*par)
    nv = en.n_values
    A = np.eye(c.shape[1])[:, :nv] * 0.35 + 0.1 * rng.uniform(-1, 1, (c.shape[1], nv))
    u = (c - 1.5) @ A + 0.02 / max(n) * rng.standard_normal((c.shape[0], nv))
    u, v = u.reshape(-1), rng.standard_normal(c.shape[0] * nv)
    tol = 1e-12 if dtype == torch.float64 else 1e-4
    ut, vt = (torch.as_tensor(a, dtype=dtype, device=cuda) for a in (u, v))
    assert rel(en.residual(ut), omat.residual(oo, law, u)) < tol
    assert rel(en.hvp(ut, vt), omat.hvp(oo, law, u, v)) < tol
