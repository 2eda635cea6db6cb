"""Infinite, NaN and nearly largest nodal and quadrature values through the operator maps: the
results are those of the weighted sums out[e, q] = sum_a N_a(xi_q) u[conn[e, a]] and so on, where
a positive weight keeps an infinity an infinity and a mean of large numbers is a large number.
"""

import numpy as np
import pytest
import torch

from oracle import elements as oe
from oracle import mesh as om
from oracle import operator as oop
from tatva_gb300 import Mesh, Operator, element

pytestmark = pytest.mark.gpu

HUGE = {torch.float32: 3.0e38, torch.float64: 1.7e308}  # 0.88 and 0.95 of the largest number
EPS = {torch.float32: 2.0**-24, torch.float64: 2.0**-53}


def _hex(cuda, n):
    c, e = om.brick(*n)
    c = c + 0.1 / max(n) * np.random.default_rng(2).uniform(-1, 1, c.shape)
    return (Operator(Mesh(c, e, device=cuda), element.Hexahedron8()),
            oop.OracleOperator(c, e, oe.Hexahedron8()), c, e)


def _shape(vals):
    return () if vals == 0 else (vals,)


def _same_kinds(got, want):
    """Infinities of the same sign, NaN and finite numbers in the same places."""
    got = got.detach().double().cpu().numpy()
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(np.isposinf(got), np.isposinf(want))
    assert np.array_equal(np.isneginf(got), np.isneginf(want))
    return got


def _weights():
    s = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1],
                  [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]], float)
    return (1 + s[None] * s[:, None] / np.sqrt(3.0)).prod(-1) / 8  # (q, a), all positive


@pytest.mark.parametrize("vals", [0, 2, 3, 5])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_hex_eval_of_infinite_and_nan_nodes(cuda, vals, dtype):
    op, _, c, e = _hex(cuda, (4, 3, 2))
    u = np.random.default_rng(4).standard_normal((c.shape[0],) + _shape(vals))
    flat = u.reshape(c.shape[0], -1)
    flat[e[5, 0], 0], flat[e[17, 6], -1], flat[e[9, 3], 0] = np.inf, -np.inf, np.nan
    want = np.einsum("qa,eav->eqv", _weights(), flat[e]).reshape(e.shape[0], 8, *_shape(vals))
    got = _same_kinds(op.eval(torch.as_tensor(u, dtype=dtype, device=cuda)), want)
    ok = np.isfinite(want)
    assert np.abs(got[ok] - want[ok]).max() <= 32 * EPS[dtype] * np.abs(flat[np.isfinite(flat)]).max()
    assert np.isinf(want).any() and np.isnan(want).any()


@pytest.mark.parametrize("vals", [0, 3, 4])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_hex_eval_and_transpose_of_huge_values(cuda, vals, dtype):
    """Means of values near the largest number, of both signs, in one element."""
    op, _, c, e = _hex(cuda, (1, 1, 1))
    rng = np.random.default_rng(6)
    u = HUGE[dtype] * np.where(rng.random((8,) + _shape(vals)) < 0.5, -1.0, 1.0)
    ut = torch.as_tensor(u, dtype=dtype, device=cuda).requires_grad_(True)
    big = torch.as_tensor(u, dtype=dtype).double().numpy().reshape(8, -1)
    out = op.eval(ut)
    got = out.detach().double().cpu().numpy().reshape(8, -1)
    want = np.einsum("qa,av->qv", _weights(), big[e[0]] / HUGE[dtype])
    assert np.abs(got / HUGE[dtype] - want).max() <= 32 * EPS[dtype]
    g = torch.as_tensor(u[None], dtype=dtype, device=cuda)
    (du,) = torch.autograd.grad(out, ut, g)
    want = np.zeros_like(big)
    want[e[0]] = np.einsum("qa,qv->av", _weights(), big / HUGE[dtype])
    got = du.double().cpu().numpy().reshape(8, -1) / HUGE[dtype]
    assert np.abs(got - want).max() <= 32 * EPS[dtype]


@pytest.mark.parametrize("vals", [0, 1, 3, 5])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_hex_eval_transpose_of_infinite_and_nan_points(cuda, vals, dtype):
    op, _, c, e = _hex(cuda, (4, 3, 2))
    q = np.random.default_rng(5).standard_normal((e.shape[0], 8) + _shape(vals))
    flat = q.reshape(e.shape[0], 8, -1)
    flat[3, 0, 0], flat[20, 5, -1], flat[11, 7, 0] = np.inf, -np.inf, np.nan
    u = torch.zeros((c.shape[0],) + _shape(vals), dtype=dtype, device=cuda, requires_grad=True)
    (du,) = torch.autograd.grad(op.eval(u), u, torch.as_tensor(q, dtype=dtype, device=cuda))
    want = np.zeros((c.shape[0], flat.shape[2]))
    np.add.at(want, e.ravel(), np.einsum("qa,eqv->eav", _weights(), flat).reshape(e.size, -1))
    _same_kinds(du, want.reshape(du.shape))
    assert np.isinf(want).any() and np.isnan(want).any()


def _simplex(cuda, elem):
    """A mesh whose shape gradients have no zero component, and G (e, a, d)."""
    rng = np.random.default_rng(3)
    c, e = om.unit_square(4, 3) if elem == "tri3" else om.kuhn_box((1, 1, 1), (3, 2, 2))
    c = np.asarray(c, float) + 0.08 * rng.uniform(-1, 1, np.shape(c))
    d = c.shape[1]
    X = c[e]
    R = np.linalg.inv(X[:, 1:] - X[:, :1])  # (e, d, k)
    G = np.concatenate([-R.sum(2)[:, None], R.transpose(0, 2, 1)], 1)
    assert np.abs(G).min() > 1e-4  # far above FP32's rounding of G: every sign is certain
    cls = element.Tri3 if elem == "tri3" else element.Tetrahedron4
    return Operator(Mesh(c, e, device=cuda), cls()), c, e, G, d


@pytest.mark.parametrize("elem", ["tri3", "tet4"])
@pytest.mark.parametrize("vals", [0, 3, 5])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_simplex_grad_of_infinite_and_nan_nodes(cuda, elem, vals, dtype):
    op, c, e, G, d = _simplex(cuda, elem)
    for corner in range(e.shape[1]):
        u = np.random.default_rng(4).standard_normal((c.shape[0],) + _shape(vals))
        flat = u.reshape(c.shape[0], -1)
        flat[e[4, corner], 0], flat[e[-1, corner], -1] = np.inf, -np.inf
        flat[e[9, corner], 0] = np.nan
        with np.errstate(invalid="ignore"):
            want = (flat[e][:, :, :, None] * G[:, :, None, :]).sum(1)  # (e, v, d)
        _same_kinds(op.grad(torch.as_tensor(u, dtype=dtype, device=cuda)),
                    want.reshape((e.shape[0], 1) + _shape(vals) + (d,)))
        assert np.isinf(want).any() and np.isnan(want).any()


@pytest.mark.parametrize("elem", ["tri3", "tet4"])
@pytest.mark.parametrize("vals", [0, 3, 5])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_simplex_grad_transpose_of_infinite_and_nan_points(cuda, elem, vals, dtype):
    op, c, e, G, d = _simplex(cuda, elem)
    f = np.random.default_rng(5).standard_normal((e.shape[0], 1) + _shape(vals) + (d,))
    flat = f.reshape(e.shape[0], -1, d)
    flat[3, 0, 0], flat[-2, -1, 1], flat[10, 0, 0] = np.inf, -np.inf, np.nan
    u = torch.zeros((c.shape[0],) + _shape(vals), dtype=dtype, device=cuda, requires_grad=True)
    (du,) = torch.autograd.grad(op.grad(u), u, torch.as_tensor(f, dtype=dtype, device=cuda))
    with np.errstate(invalid="ignore"):
        per = (flat[:, None] * G[:, :, None, :]).sum(-1)  # (e, a, v)
        want = np.zeros((c.shape[0], flat.shape[1]))
        np.add.at(want, e.ravel(), per.reshape(e.size, -1))
    _same_kinds(du, want.reshape(du.shape))
    assert np.isinf(want).any() and np.isnan(want).any()
