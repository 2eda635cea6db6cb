"""The persistent CG of structured bricks (one cooperative launch per block of iterations)
where its sharing of tiles, faces and vector entries can go wrong: bricks of a single cell or
layer, vectors whose length is not a multiple of four, fewer pieces than CTAs, partial blocks.

Tolerances: the FP64 solution agrees with the element-block CG (same tolerance 1e-12) to 1e-9
relative; FP32 solves reach a true FP64 residual of 1e-4 |b| (rtol 1e-5 on the recursion).
"""

import numpy as np
import pytest
import torch

from oracle import mesh as om
from tatva_gb300 import Mesh, Operator, element, materials, solvers

pytestmark = pytest.mark.gpu


def _problem(shape, cuda, clamp=True):
    c, e = om.brick(*shape, lengths=tuple(0.1 * s for s in shape))
    op = Operator(Mesh(c, e, device=cuda), element.Hexahedron8())
    en = materials.LinearElastic(op, 0.7, 1.9)
    assert en.plan().grid
    g = torch.Generator(device=cuda).manual_seed(3)
    b = torch.randn(en.n_dofs, dtype=torch.float64, device=cuda, generator=g)
    fixed = np.zeros((c.shape[0], 3), np.uint8)
    fixed[c[:, 0] == 0.0] = 1
    fixed[np.argmax(c.sum(1)), 1] = 1  # a single component elsewhere
    fixed = torch.as_tensor(fixed.reshape(-1), device=cuda)
    return en, torch.where(fixed.bool(), 0.0, b) if clamp else b, fixed


@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 5, 2), (2, 3, 4), (33, 9, 17), (5, 40, 6),
                                   (37, 34, 35)])
def test_solutions(cuda, shape):
    en, b, fixed = _problem(shape, cuda)
    x = solvers.cg(en, b, fixed=fixed, rtol=1e-12)
    assert x.converged
    plan = en.plan()
    plan.grid = False
    try:
        ref = solvers.cg(en, b, fixed=fixed, rtol=1e-12)
        assert float((x.x - ref.x).norm() / ref.x.norm()) < 1e-9
    finally:
        plan.grid = True
    x32 = solvers.cg(en, b.float(), fixed=fixed, rtol=1e-5)
    r = b - en.hvp(None, x32.x.double(), fixed=fixed)
    assert float(r.norm() / b.norm()) < 1e-4


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_partial_blocks_and_repeats(cuda, dtype):
    """13 iterations in blocks of 5, of 13 and one by one: exact counts, the same bits."""
    en, b, fixed = _problem((20, 17, 19), cuda)
    runs = [solvers.cg(en, b.to(dtype), fixed=fixed, rtol=1e-30, maxiter=13, check_every=k,
                       raise_on_fail=False) for k in (5, 13, 1, 5)]
    assert all(r.iterations == 13 and not r.converged for r in runs)
    assert all(torch.equal(r.x, runs[0].x) for r in runs)


def test_without_fixed_dofs_a_rigid_body_load_breaks_down_or_converges(cuda):
    """No Dirichlet mask: singular operator, consistent right-hand side (zero mean force):
    the kernel without a mask runs and reduces the residual."""
    en, b, _ = _problem((9, 8, 7), cuda, clamp=False)
    rhs = en.hvp(None, b)  # in the operator's range
    r = solvers.cg(en, rhs, rtol=1e-8, maxiter=2000, raise_on_fail=False)
    assert r.rel_res <= 1e-8


def test_streams_and_threads(cuda):
    """Two host threads, each solving on its own: every solve gives the same bits."""
    import threading

    en, b, fixed = _problem((24, 20, 22), cuda)
    want = solvers.cg(en, b, fixed=fixed, rtol=1e-10).x
    out = {}

    def work(k):
        e2, b2, f2 = _problem((24, 20, 22), cuda)
        out[k] = [solvers.cg(e2, b2, fixed=f2, rtol=1e-10).x for _ in range(3)]

    ts = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert all(torch.equal(x, want) for k in out for x in out[k]) and len(out) == 2
