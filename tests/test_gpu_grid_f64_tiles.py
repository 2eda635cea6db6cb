"""FP64 stencil of the structured brick at the depths its tiles take: one plane each (two to 33
node planes), several planes with a last layer of one or two, rows of columns that a tile
has and the grid does not.  Against the element-block kernels of the same plan: relative
max norm 1e-13 (27 entries of 24 products a row in other orders: about 200 roundings of
2^-53, and cancellation of the rigid part)."""

import numpy as np
import pytest
import torch

from oracle import mesh as om
from tatva_gb300 import Mesh, Operator, element, materials

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [
    (2, 2, 1), (2, 2, 2), (2, 2, 3), (33, 8, 9), (9, 10, 16), (32, 33, 32),  # one plane a tile
    (34, 33, 34), (44, 34, 44), (50, 50, 50),    # 2, 3 and 5 planes; a last layer of 1, 3 and 1
    (64, 41, 21), (4, 5, 300)])
@pytest.mark.parametrize("mask", [False, True])
def test_hvp(cuda, shape, mask):
    c, e = om.brick(*shape, lengths=(1.0, 0.9, 1.1))
    op = Operator(Mesh(c, e, device=cuda), element.Hexahedron8())
    en = materials.LinearElastic(op, 0.7, 1.9)
    plan = en.plan()
    assert plan.grid
    rng = np.random.default_rng(5)
    v = torch.as_tensor(rng.standard_normal(en.n_dofs), device=cuda)
    f = None
    if mask:
        fixed = (rng.random(en.n_dofs) < 0.1).astype(np.uint8)
        fixed.reshape(-1, 3)[c[:, 2] == c[:, 2].max()] = 1
        f = torch.as_tensor(fixed, device=cuda)
    got = en.hvp(None, v, fixed=f)
    plan.grid = False
    try:
        want = en.hvp(None, v, fixed=f)
    finally:
        plan.grid = True
    assert float((got - want).abs().max()) <= 1e-13 * float(want.abs().max())
