"""The element kernels of eval / grad and their transposes where they can go wrong: element
counts around a warp and a CTA, component counts with and without their own kernel, and
arrays that are not 32-byte aligned, through the C ABI.

Tolerances (relative, max norm): FP64 1e-12, FP32 2e-5, the repository's bounds of the maps
against the oracle (here in FP64 with distorted cells of size 1).
"""

import numpy as np
import pytest
import torch

from oracle import elements as oe
from oracle import mesh as om
from oracle import operator as oop
from tatva_gb300 import Mesh, Operator, _lib, element
from tatva_gb300._device import prec_of

pytestmark = pytest.mark.gpu

ELS = {"tri3": (element.Tri3, oe.Tri3), "tet4": (element.Tetrahedron4, oe.Tetrahedron4),
       "hex8": (element.Hexahedron8, oe.Hexahedron8)}


def rel(a, b):
    a = a.detach().double().cpu().numpy()
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300))


def _setup(elem, n, cuda, jitter=0.15):
    if elem == "tri3":
        c, e = om.unit_square(*n[:2])
        c = c * np.array(n[:2])
    elif elem == "tet4":
        c, e = om.kuhn_box(tuple(float(k) for k in n), n, origin=(0, 0, 0))
    else:
        c, e = om.brick(*n, lengths=tuple(float(k) for k in n))
    rng = np.random.default_rng(2)
    c = c + jitter * rng.uniform(-1, 1, c.shape)
    return Operator(Mesh(c, e, device=cuda), ELS[elem][0]()), oop.OracleOperator(c, e, ELS[elem][1]())


def _odd(t, odd):
    """A copy of t that starts one value after a 256-byte boundary (or at one)."""
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    v = buf[1:] if odd else buf[:-1]
    v.copy_(t.reshape(-1))
    return v


@pytest.mark.parametrize("elem,n", [("tri3", (1, 1, 1)), ("tri3", (8, 9, 1)), ("tet4", (1, 1, 1)),
                                    ("tet4", (3, 4, 2)), ("hex8", (1, 1, 1)), ("hex8", (4, 8, 4)),
                                    ("hex8", (3, 11, 4))])
@pytest.mark.parametrize("V", [1, 2, 3, 4, 6])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_maps_and_transposes(cuda, elem, n, V, dtype):
    op, oo = _setup(elem, n, cuda)
    rng = np.random.default_rng(V)
    E, Q, D, nn = op.n_elements, op.n_quad, op.dim, op.n_nodes
    u = rng.standard_normal((nn, V))
    q, f = rng.standard_normal((E, Q, V)), rng.standard_normal((E, Q, V, D))
    tol = 1e-12 if dtype == torch.float64 else 2e-5
    t = lambda a: torch.as_tensor(a, dtype=dtype, device=cuda)  # noqa: E731
    assert rel(op.eval(t(u)), oo.eval(u)) < tol
    assert rel(op.grad(t(u)), oo.grad(u)) < tol
    assert rel(op._eval_t_raw(t(q), (V,)), oo.eval_transpose(q)) < tol
    assert rel(op._grad_t_raw(t(f), (V,)), oo.grad_transpose(f)) < tol
    # the reverse mode is the transpose of the forward maps (FP64: to rounding)
    if dtype == torch.float64:
        a = float((op.grad(t(u)) * t(f)).sum())
        b = float((op._grad_t_raw(t(f), (V,)) * t(u)).sum())
        assert abs(a - b) <= 1e-12 * float(np.abs(f).sum())


@pytest.mark.parametrize("odd", [False, True])
@pytest.mark.parametrize("V", [1, 2, 3])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_hex8_unaligned_arrays(cuda, V, odd, dtype):
    """Arrays at an odd offset take the element kernels' narrow accesses: same bits."""
    op, _ = _setup("hex8", (3, 5, 3), cuda)
    g = torch.Generator(device=cuda).manual_seed(V)
    E, nn, P = op.n_elements, op.n_nodes, prec_of(dtype)
    rnd = lambda *s: torch.randn(*s, dtype=dtype, device=cuda, generator=g)  # noqa: E731
    u, q, f = rnd(nn, V), rnd(E, 8, V), rnd(E, 8, V, 3)
    conn, xyz = op.mesh.elements, op.coords_as(dtype)
    ip, ii = op.incidence()
    st = torch.cuda.current_stream().cuda_stream
    uo, qo, fo = _odd(u, odd), _odd(q, odd), _odd(f, odd)
    out = _odd(torch.zeros_like(q), odd)
    _lib.call("tg_eval", 2, P, uo.data_ptr(), nn, V, conn.data_ptr(), E, out.data_ptr(), st)
    assert torch.equal(out.view_as(q), op.eval(u))
    out = _odd(torch.zeros_like(f), odd)
    _lib.call("tg_grad", 2, P, uo.data_ptr(), xyz.data_ptr(), nn, V, conn.data_ptr(), E,
              out.data_ptr(), st)
    assert torch.equal(out.view_as(f), op.grad(u))
    nb = _lib.lib().tg_grad_transpose_workspace_bytes(2, P, E, V)
    ws = _odd(torch.zeros(E * 8 * V, dtype=dtype, device=cuda), odd)
    y = torch.empty_like(u)
    _lib.call("tg_grad_transpose", 2, P, fo.data_ptr(), xyz.data_ptr(), nn, V, conn.data_ptr(), E,
              ip.data_ptr(), ii.data_ptr(), y.data_ptr(), ws.data_ptr(), nb, st)
    assert torch.equal(y, op._grad_t_raw(f, (V,)))
    assert nb == _lib.lib().tg_eval_transpose_workspace_bytes(2, P, E, V)
    _lib.call("tg_eval_transpose_ws", 2, P, qo.data_ptr(), nn, V, conn.data_ptr(), E,
              ip.data_ptr(), ii.data_ptr(), y.data_ptr(), ws.data_ptr(), nb, st)
    assert torch.equal(y, op._eval_t_raw(q, (V,)))
    z = torch.empty_like(u)  # the entry point without a workspace: same sums, other rounding
    _lib.call("tg_eval_transpose", 2, P, qo.data_ptr(), nn, V, conn.data_ptr(), E, ip.data_ptr(),
              ii.data_ptr(), z.data_ptr(), st)
    assert rel(y, z.double().cpu().numpy()) < (1e-13 if dtype == torch.float64 else 1e-5)
