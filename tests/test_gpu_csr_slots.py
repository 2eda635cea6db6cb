"""The tables of the CSR tangent (``tg_csr_slots``): the position of every corner among the
columns of its row and the longest row, exactly, against a search on the host; colours at
and above the kernel's limit take the compressed route."""

import dataclasses

import numpy as np
import pytest
import torch

from oracle import mesh as om
from tatva_gb300 import Mesh, Operator, element, materials, sparse

pytestmark = pytest.mark.gpu


def _mesh(case):
    if case == "fan":  # one node in every element, the others in two
        m = 37
        th = np.linspace(0, 2 * np.pi, m, endpoint=False)
        c = np.concatenate([[[0.0, 0.0]], np.stack([np.cos(th), np.sin(th)], 1)])
        i = np.arange(m)
        return c, np.stack([0 * i, 1 + i, 1 + (i + 1) % m], 1).astype(np.int32), element.Tri3()
    if case.startswith("tri3"):
        return *om.unit_square(*((1, 1) if case == "tri3_small" else (23, 9))), element.Tri3()
    if case == "tet4":
        return *om.kuhn_box((1, 1, 1), (4, 3, 5), origin=(0, 0, 0)), element.Tetrahedron4()
    return *om.brick(*((1, 1, 1) if case == "hex8_small" else (3, 4, 5))), element.Hexahedron8()


def _energy(op, law):
    return (materials.Poisson(op, 1.0, 0.0) if law == "poisson"
            else materials.LinearElastic(op, 0.7, 1.9))


@pytest.mark.parametrize("case", ["fan", "tri3_small", "tri3", "tet4", "hex8_small", "hex8"])
@pytest.mark.parametrize("law", ["poisson", "linear_elastic"])
def test_slots(cuda, case, law):
    c, e, el = _mesh(case)
    op = Operator(Mesh(c, e, device=cuda), el)
    en = _energy(op, law)
    V, NN = en.n_values, e.shape[1]
    csr = sparse.pattern_from_mesh(op.mesh, V)
    cm = sparse.ColoredMatrix.from_csr(csr, device=cuda)
    slots, max_deg = en.csr_slots(cm, cm.n_colors)
    assert max_deg == np.max(np.diff(csr.indptr)) // V
    inc = op.incidence()[1].cpu().numpy()
    got = slots.cpu().numpy().view(np.uint16).reshape(len(inc), -1)
    for j, ea in enumerate(inc):
        conn = e[ea // NN]
        n = conn[ea % NN]
        cols = csr.indices[csr.indptr[V * n]:csr.indptr[V * n + 1]:V] // V
        assert np.array_equal(got[j, :NN], np.searchsorted(cols, conn))
        assert not got[j, NN:].any()


@pytest.mark.parametrize("top", [1023, 1024])
def test_largest_colour(cuda, top):
    c, e, el = _mesh("tet4")
    op = Operator(Mesh(c, e, device=cuda), el)
    en = _energy(op, "linear_elastic")
    cm = sparse.ColoredMatrix.from_csr(sparse.pattern_from_mesh(op.mesh, 3), device=cuda)
    colors = cm.colors.clone()
    colors[colors == 0] = top
    cm = dataclasses.replace(cm, colors=colors)
    assert (en.csr_slots(cm, cm.n_colors) is None) == (top == 1024)
    assert (en.csr_slots(cm, en.MAX_COLORS) is None) == (top == 1024)
    u = torch.zeros(en.n_dofs, dtype=torch.float64, device=cuda)
    want = sparse.decompress(en.compressed_hessian(u, cm.colors, cm.n_colors),
                             *sparse.compute_rows_cols(cm))
    got = sparse.jacfwd(en.residual, cm)(u).data
    if top == 1024:  # the compressed route: the same bits
        assert torch.equal(got, want)
    else:  # up to 24 summed tets of about 20 roundings a product
        assert float((got - want).abs().max()) <= 512 * 2.0 ** -53 * float(want.abs().max())
