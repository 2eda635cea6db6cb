"""CG on structured bricks over both its paths: one cooperative launch for a block of iterations
(``grid_cg_kernel``), and separate launches captured in a graph (``grid_le_kernel`` with p.q,
``cg_update_kernel``, ``cg_p_kernel``), which larger bricks and a refused cooperative launch take.

Tolerances: solutions to the same tolerance 1e-12 (1e-10 mixed) agree with the element-block CG's
to 1e-9 (1e-8) relative; FP32 solves reach a true FP64 residual of 1e-4 |b| (rtol 1e-5 on the
recursion).  Above 3.5 M unknowns, 30 FP32 iterations: each rounds its vectors and scalars at
2^-24, 30 * 2^-24 = 2e-6 of x, times the growth of a difference over the iterations (below 500
for the residual's drop by 10 here): 1e-3.
"""

import ctypes
import threading

import numpy as np
import pytest
import torch

from oracle import mesh as om
from tatva_gb300 import Mesh, Operator, _lib, element, materials, solvers
from tatva_gb300._device import workspace
from tatva_gb300.problems import clamped_brick

pytestmark = pytest.mark.gpu
PATHS = pytest.mark.parametrize("persistent", [True, False])


def _problem(shape, cuda):
    c, e = om.brick(*shape, lengths=tuple(0.1 * s for s in shape))
    op = Operator(Mesh(c, e, device=cuda), element.Hexahedron8())
    en = materials.LinearElastic(op, 0.7, 1.9)
    g = torch.Generator(device=cuda).manual_seed(3)
    b = torch.randn(en.n_dofs, dtype=torch.float64, device=cuda, generator=g)
    fixed = np.zeros((c.shape[0], 3), np.uint8)
    fixed[c[:, 0] == 0.0] = 1
    fixed[np.argmax(c.sum(1)), 1] = 1  # a single component elsewhere
    fixed = torch.as_tensor(fixed.reshape(-1), device=cuda)
    return en, torch.where(fixed.bool(), 0.0, b), fixed


@PATHS
@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 5, 2), (2, 3, 4), (33, 9, 17), (5, 40, 6),
                                   (37, 34, 35)])
def test_solutions(cuda, shape, persistent):
    en, b, fixed = _problem(shape, cuda)
    plan = en.plan()
    assert plan.grid and plan.persistent_cg
    plan.grid = False
    ref = solvers.cg(en, b, fixed=fixed, rtol=1e-12).x
    plan.grid = True
    plan.persistent_cg = persistent
    x = solvers.cg(en, b, fixed=fixed, rtol=1e-12)
    assert x.converged and float((x.x - ref).norm() / ref.norm()) < 1e-9
    m = solvers.mixed_cg(en, b, fixed=fixed, rtol=1e-10)
    assert m.converged and float((m.x - ref).norm() / ref.norm()) < 1e-8
    x32 = solvers.cg(en, b.float(), fixed=fixed, rtol=1e-5)
    r = b - en.hvp(None, x32.x.double(), fixed=fixed)
    assert float(r.norm() / b.norm()) < 1e-4


@PATHS
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_blocks_checks_and_bits(cuda, dtype, persistent):
    """13 iterations in blocks of 5, of 13 and one by one: exact counts, the same bits, and the
    host's checks say which path ran (16 blocks in one cooperative launch)."""
    en, b, fixed = _problem((20, 17, 19), cuda)
    en.plan().persistent_cg = persistent
    for every, separate in ((5, 3), (13, 1), (1, 13)):
        r = solvers.cg(en, b.to(dtype), fixed=fixed, rtol=1e-30, maxiter=13, check_every=every,
                       raise_on_fail=False)
        assert r.iterations == 13 and not r.converged
        assert r.checks == (1 if persistent else separate)
        first = r.x if every == 5 else first
        assert torch.equal(r.x, first)
    runs = [solvers.mixed_cg(en, b, fixed=fixed, rtol=1e-10, check_every=k) for k in (6, 50)]
    assert runs[0].iterations == runs[1].iterations and torch.equal(runs[0].x, runs[1].x)


@PATHS
def test_checks_of_a_mixed_solve(cuda, persistent):
    """k iterations of an inner solve take ceil(k / interval) checks."""
    en, b, fixed = _problem((20, 17, 19), cuda)
    en.plan().persistent_cg = persistent
    m = solvers.mixed_cg(en, b, fixed=fixed, rtol=1e-10, check_every=20)
    interval = 16 * 20 if persistent else 20
    assert max(m.outer, m.iterations / interval) <= m.checks
    assert m.checks <= m.outer + m.iterations // interval


@PATHS
def test_prescribed_values(cuda, persistent):
    """b nonzero on fixed dofs: x = b there exactly, the rest as the element-block CG's."""
    en, b, fixed = _problem((14, 9, 11), cuda)
    b = 1e-3 * torch.randn(b.numel(), dtype=torch.float64, device=cuda,
                           generator=torch.Generator(device=cuda).manual_seed(1))
    plan = en.plan()
    plan.grid = False
    ref = solvers.cg(en, b, fixed=fixed, rtol=1e-11).x
    plan.grid = True
    plan.persistent_cg = persistent
    for r in (solvers.cg(en, b, fixed=fixed, rtol=1e-11),
              solvers.mixed_cg(en, b, fixed=fixed, rtol=1e-10)):
        assert r.converged and torch.equal(r.x[fixed.bool()], b[fixed.bool()])
        assert float((r.x - ref).norm() / ref.norm()) < 1e-8


def test_above_the_cooperative_launch(cuda):
    """3,573,048 unknowns: separate launches by size alone."""
    P = clamped_brick(105, cuda)
    en, fixed, b = P["energy"], P["fixed"], P["b"].float()
    plan = en.plan()
    assert plan.grid and plan.persistent_cg and en.n_dofs > 3_500_000
    r = solvers.cg(en, b, fixed=fixed, rtol=1e-30, maxiter=30, check_every=7,
                   raise_on_fail=False)
    assert r.iterations == 30 and r.checks == 5
    plan.grid = False
    ref = solvers.cg(en, b, fixed=fixed, rtol=1e-30, maxiter=30, raise_on_fail=False)
    plan.grid = True
    assert ref.iterations == 30
    assert float((r.x - ref.x).norm() / ref.x.norm()) < 1e-3
    x = r.x.double().reshape(-1)
    res = P["b"].double().reshape(-1) - en.hvp(None, x, fixed=fixed).reshape(-1)
    assert abs(float(res.norm() / P["b"].double().norm()) - r.rel_res) < 1e-3 * r.rel_res


@PATHS
def test_two_streams_at_once(cuda, persistent):
    """Two host threads, each with its own stream, plan, vectors and workspace, solving at the
    same time: every solve gives the bits of a solve alone."""
    L = _lib.lib()
    problems = [_problem((24, 20, 22), cuda) for _ in range(2)]
    want = None
    jobs = []
    for en, b, fixed in problems:
        en.plan().persistent_cg = persistent
        want = solvers.cg(en, b, fixed=fixed, rtol=1e-10).x
        desc, keep = en.operator_desc(None, fixed, torch.float64)
        diag = en.diagonal(torch.zeros_like(b), fixed).reshape(-1).contiguous()
        nb = L.tg_cg_workspace_bytes(ctypes.byref(desc))
        jobs.append((desc, keep, b, diag, workspace(nb, cuda), nb, torch.cuda.Stream(device=cuda)))
    torch.cuda.synchronize()
    start, out = threading.Barrier(2), {}

    def work(k):
        desc, _, b, diag, ws, nb, st = jobs[k]
        torch.cuda.set_device(cuda.index or 0)
        start.wait()
        res = []
        for _ in range(5):
            x = torch.zeros_like(b)
            torch.cuda.current_stream().synchronize()
            stats = _lib.SolveStats()
            rc = L.tg_cg_solve(ctypes.byref(desc), b.data_ptr(), x.data_ptr(), diag.data_ptr(),
                               1e-10, 10000, 50, ws.data_ptr(), nb, ctypes.byref(stats),
                               st.cuda_stream)
            st.synchronize()
            res.append((rc, x))
        out[k] = res

    ts = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert len(out) == 2
    assert all(rc == _lib.TG_OK and torch.equal(x, want) for k in out for rc, x in out[k])
