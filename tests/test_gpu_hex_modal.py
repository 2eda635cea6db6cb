"""The trilinear (modal) Hex8 element of the residual / HVP / energy kernels against the
oracle's per-point evaluation, where its algebra can go wrong: one element, every node
moved, cells far from the origin, every law.

Tolerances (relative, max norm).  FP64: 1e-12, the repository's bound against the oracle.
FP32: 1e-4, the repository's bound of the fused FP32 kernels.
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


@pytest.mark.parametrize("shape,origin", [((1, 1, 1), 0.0), ((3, 2, 5), 0.0), ((2, 3, 2), 4.0)])
@pytest.mark.parametrize("kind", list(LAWS))
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_modal_element_matches_oracle(cuda, shape, origin, kind, dtype):
    rng = np.random.default_rng(5)
    c, e = om.brick(*shape, lengths=tuple(float(s) for s in shape))
    c = c + 0.18 * rng.uniform(-1, 1, c.shape) + origin  # every node moved, outer ones too
    op = Operator(Mesh(c, e, device=cuda), element.Hexahedron8())
    oo = oop.OracleOperator(c, e, oe.Hexahedron8())
    cls, ocls, par = LAWS[kind]
    en, law = cls(op, *par), ocls(*par)
    n = c.shape[0] * en.n_values
    u, v = 0.04 * rng.standard_normal(n), rng.standard_normal(n)
    tol = 1e-12 if dtype == torch.float64 else 1e-4
    ut, vt = (torch.as_tensor(a, dtype=dtype, device=cuda) for a in (u, v))
    assert rel(en.residual(ut), omat.residual(oo, law, u)) < tol
    assert rel(en.hvp(ut, vt), omat.hvp(oo, law, u, v)) < tol
    assert rel(en.value(ut).reshape(1), np.array([omat.energy(oo, law, u)])) < tol
