"""Backward passes of the operator maps: the plain backward (no autograd node of its own),
the differentiable one (create_graph), and what takes neither: batched and forward-mode
cotangents are refused, as an autograd.Function without those rules refuses them."""

import pytest
import torch
from torch.autograd import forward_ad

from oracle import mesh as om
from tatva_gb300 import Mesh, Operator, element

pytestmark = pytest.mark.gpu


def _op(cuda):
    c, e = om.kuhn_box((1, 1, 1), (2, 3, 2), origin=(0, 0, 0))
    return Operator(Mesh(c, e, device=cuda), element.Tetrahedron4())


MAPS = {"eval": lambda op, u: op.eval(u), "grad": lambda op, u: op.grad(u),
        "integrate": lambda op, u: op._integrate_quad_array(op.eval(u)),
        "gather": lambda op, u: op._gather(u)}


@pytest.mark.parametrize("name", list(MAPS))
def test_plain_and_differentiable_backward_agree(cuda, name):
    op = _op(cuda)
    g = torch.Generator(device=cuda).manual_seed(0)
    u = torch.randn(op.n_nodes, 3, dtype=torch.float64, device=cuda, generator=g,
                    requires_grad=True)
    y = MAPS[name](op, u)
    w = torch.randn(y.shape, dtype=y.dtype, device=cuda, generator=g, requires_grad=True)
    (a,) = torch.autograd.grad(y, u, w, retain_graph=True)
    assert not a.requires_grad
    (b,) = torch.autograd.grad(y, u, w, create_graph=True)
    assert b.requires_grad and torch.equal(a, b)
    v = torch.randn(u.shape, dtype=u.dtype, device=cuda, generator=g)
    (c,) = torch.autograd.grad(b, w, v)  # the transpose of the transpose: the map itself
    assert torch.equal(c, MAPS[name](op, v))


@pytest.mark.parametrize("name", list(MAPS))
def test_transformed_cotangents_are_refused(cuda, name):
    op = _op(cuda)
    u = torch.ones(op.n_nodes, 3, dtype=torch.float64, device=cuda, requires_grad=True)
    y = MAPS[name](op, u)
    w = torch.ones_like(y)
    with pytest.raises(RuntimeError):
        torch.autograd.grad(y, u, torch.stack([w, w]), retain_graph=True, is_grads_batched=True)
    with forward_ad.dual_level():
        dual = forward_ad.make_dual(w, torch.ones_like(w))
        with pytest.raises((RuntimeError, NotImplementedError)):
            torch.autograd.grad(y, u, dual, retain_graph=True)


def test_backward_on_a_side_stream(cuda):
    op = _op(cuda)
    u = torch.ones(op.n_nodes, dtype=torch.float64, device=cuda, requires_grad=True)
    want = torch.autograd.grad(op.grad(u * 2).square().sum(), u)[0]
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        got = torch.autograd.grad(op.grad(u * 2).square().sum(), u)[0]
    torch.cuda.current_stream().wait_stream(s)
    assert torch.equal(got, want)
