"""FP32 CG over the range of right-hand sides that FP32 vectors hold: |b|^2 beyond the largest
float, and small |b|.  A power of two on b scales every number of the recursion exactly as long
as nothing over- or underflows, so the solutions are the same bits but for that factor."""

import numpy as np
import pytest
import torch

from oracle import mesh as om
from tatva_gb300 import Mesh, Operator, element, materials, solvers

pytestmark = pytest.mark.gpu


# 14,739 dofs of |b_i| about 1: b.b = 2^14, 2^130 times 2^58 squared; a thread's own sums
# (at most 30 nodes) stay below 2^126
@pytest.mark.parametrize("power", [58, 40, -30])
def test_scaled_right_hand_sides(cuda, power):
    c, e = om.brick(16, 16, 16, lengths=(16.0, 16.0, 16.0))
    op = Operator(Mesh(c, e, device=cuda), element.Hexahedron8())
    en = materials.LinearElastic(op, 0.7, 1.9)
    assert en.plan().grid
    fixed = torch.as_tensor(np.repeat(c[:, 0] == 0.0, 3).astype(np.uint8), device=cuda)
    g = torch.Generator(device=cuda).manual_seed(5)
    b = torch.randn(en.n_dofs, device=cuda, generator=g)
    b = torch.where(fixed.bool(), 0.0, b)
    one = solvers.cg(en, b, fixed=fixed, rtol=1e-30, maxiter=20, raise_on_fail=False)
    far = solvers.cg(en, b * 2.0**power, fixed=fixed, rtol=1e-30, maxiter=20,
                     raise_on_fail=False)
    assert one.iterations == far.iterations == 20
    assert torch.equal(far.x, one.x * 2.0**power)
    far = solvers.cg(en, b * 2.0**power, fixed=fixed, rtol=1e-5)
    assert far.converged
