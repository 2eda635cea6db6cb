"""Stages of the brick engine's inner solves: whatever the inner tolerance and budget, a request
reaches the FP64 residual (the oracle's operator; <= 2e-10 for the engine's 1e-10, whose own
residual equals the oracle's to about 1e-15 relative), the inner solves are counted as asked
for, and the bits do not depend on the step length."""

import numpy as np
import pytest
import torch

from oracle import elements as oe
from oracle import materials as omat
from oracle import operator as oop
from tatva_gb300 import serving
from tatva_gb300.problems import clamped_brick

pytestmark = pytest.mark.gpu


def _rel_res(req, x):
    P = clamped_brick(req.side, "cpu", traction=1.0)
    op = oop.OracleOperator(P["mesh"].coords_host(), P["mesh"].elements_host(), oe.Hexahedron8())
    law = omat.LinearElastic(*omat.lame_from_young(req.young, req.poisson))
    fixed, b = P["fixed"].numpy().astype(bool), P["b"].numpy() * req.traction
    xv = x.cpu().numpy()
    y = omat.hvp(op, law, None, np.where(fixed, 0.0, xv))
    y[fixed] = xv[fixed]
    return float(np.linalg.norm(b - y) / np.linalg.norm(b))


# (inner tolerance, inner budget, side, fewest and most inner solves that can do it): an inner
# solve gains its tolerance (the last one less), one with a budget of 9 steps any amount
@pytest.mark.parametrize("inner_rtol,max_inner,side,lo,hi", [
    (1e-11, 10000, 9, 1, 2),     # one inner solve of many stages
    (1e-4, 10000, 13, 3, 4),
    (0.04, 10000, 6, 7, 9),      # one stage each (0.04 > the largest reduction of a stage)
    (0.02, 10000, 6, 6, 8),      # two stages each
    (0.9, 10000, 4, 10, 225),    # hardly any reduction: steps one by one
    (1e-4, 9, 6, 3, 60),         # ended by the budget
])
def test_every_inner_tolerance_converges(cuda, inner_rtol, max_inner, side, lo, hi):
    req = serving.SolveRequest(0, 0.0, side, 1.7, 0.33, 1e-3)
    out = []
    for k in (3, 20, 45):
        srv = serving.Server(cuda, slots=2, inner_rtol=inner_rtol, max_inner=max_inner,
                             max_outer=300, step_iterations=k)
        srv.model(side)
        rec = srv.solve_alone(req)
        assert rec.status == 0 and rec.rel_res <= 1e-10
        assert lo <= rec.refinements <= hi, rec.refinements
        out.append(rec)
    for a in out[1:]:
        assert torch.equal(a.x, out[0].x) and a.iterations == out[0].iterations
    assert _rel_res(req, out[0].x) <= 2e-10
