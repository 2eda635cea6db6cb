"""Persistent CG with all, some or none of its vectors kept in shared memory (by the size of
the brick): the same bits whatever the launches' lengths (each stores what it kept and the
next loads it again), and the residual asked for.

The recursion stops at |r| <= 1e-3 |b|; the true residual is formed with the FP64 HVP.  FP32
vectors and operator: the two differ by the rounding of about 100 updates of a residual that
starts at |b|, 100 * 2^-24 |b| = 6e-6 |b|, and by the rounding of A32 against A64, 2^-24 a
coefficient times a condition of a few hundred for these bricks, 2e-5 |b|; 1.05e-3 holds both.
"""

import pytest
import torch

from tatva_gb300 import solvers
from tatva_gb300.problems import clamped_brick

pytestmark = pytest.mark.gpu


# cells a side -> vectors kept (152 SMs): FP32 20, 64: four, 80: three, 96: two, 103: one;
# FP64 20: four, 64: two, 96: one, 103: none
@pytest.mark.parametrize("n", [20, 64, 80, 96, 103])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_launch_lengths_and_residual(cuda, n, dtype):
    P = clamped_brick(n, cuda)
    en, fixed = P["energy"], P["fixed"]
    b = P["b"].to(dtype)
    one = solvers.cg(en, b, fixed=fixed, rtol=1e-3, check_every=200)
    many = solvers.cg(en, b, fixed=fixed, rtol=1e-3, check_every=1)
    assert one.converged and many.iterations == one.iterations
    assert torch.equal(one.x, many.x)
    x = one.x.double().reshape(-1)
    r = P["b"].double().reshape(-1) - en.hvp(None, x, fixed=fixed).reshape(-1)
    assert float(r.norm() / P["b"].double().norm()) <= 1.05e-3
