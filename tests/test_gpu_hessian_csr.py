"""Tangent values straight into CSR (``tg_csr_slots`` / ``tg_hessian_csr``): against the
oracle's assembled tangent and against the compressed Hessian with decompression, which
patterns and colourings that the direct route refuses still take.

Tolerances (relative, max norm): against the oracle FP64 1e-12, FP32 1e-4; where both
routes run, FP64 1e-13 and FP32 1e-5 (the same element formula, other rounding).
"""

import dataclasses

import numpy as np
import pytest
import scipy.sparse as sps
import torch

from oracle import elements as oe
from oracle import materials as omat
from oracle import mesh as om
from oracle import operator as oop
from tatva_gb300 import Mesh, Operator, element, materials, sparse

pytestmark = pytest.mark.gpu

LAWS = {"linear_elastic": (materials.LinearElastic, omat.LinearElastic, (0.7, 1.9)),
        "poisson": (materials.Poisson, omat.Poisson, (1.3, 0.6)),
        "neo_hookean": (materials.NeoHookean, omat.NeoHookean, (1.0, 10.0))}
ELS = {"tri3": (element.Tri3, oe.Tri3), "tet4": (element.Tetrahedron4, oe.Tetrahedron4),
       "hex8": (element.Hexahedron8, oe.Hexahedron8)}


def rel(a, b):
    a, b = (x.detach().double().cpu().numpy() if isinstance(x, torch.Tensor) else x
            for x in (a, b))
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300))


def _setup(elem, n, kind, cuda, seed=0):
    if elem == "tri3":
        c, e = om.unit_square(*n[:2])
    elif elem == "tet4":
        c, e = om.kuhn_box((1, 1, 1), n, origin=(0, 0, 0))
    else:
        c, e = om.brick(*n)
    rng = np.random.default_rng(seed)
    c = c + 0.1 / max(n) * rng.uniform(-1, 1, c.shape)
    op = Operator(Mesh(c, e, device=cuda), ELS[elem][0]())
    cls, ocls, par = LAWS[kind]
    en = cls(op, *par)
    law = ocls(*par, dim=2) if elem == "tri3" and kind == "linear_elastic" else ocls(*par)
    u = 0.03 / max(n) * rng.standard_normal(en.n_dofs)
    csr = sparse.pattern_from_mesh(op.mesh, en.n_values)
    return op, oop.OracleOperator(c, e, ELS[elem][1]()), en, law, u, csr


def _compressed(en, cm, u):
    Jc = en.compressed_hessian(u, cm.colors, cm.n_colors)
    return sparse.decompress(Jc, *sparse.compute_rows_cols(cm))


# node counts below, at and above one warp's 32 nodes and one CTA's 64
@pytest.mark.parametrize("elem,n", [("tri3", (1, 1, 1)), ("tri3", (3, 7, 1)), ("tri3", (20, 13, 1)),
                                    ("tet4", (1, 1, 1)), ("tet4", (3, 3, 3)), ("tet4", (4, 5, 3)),
                                    ("hex8", (1, 1, 1)), ("hex8", (3, 3, 3)), ("hex8", (5, 3, 4))])
@pytest.mark.parametrize("kind", list(LAWS))
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_direct_values(cuda, elem, n, kind, dtype):
    if elem == "tri3" and kind == "neo_hookean":
        pytest.skip("3D law")
    op, oo, en, law, u, csr = _setup(elem, n, kind, cuda)
    cm = sparse.ColoredMatrix.from_csr(csr, device=cuda)
    assert en.csr_slots(cm, cm.n_colors) is not None
    ut = torch.as_tensor(u, dtype=dtype, device=cuda)
    K = sparse.jacfwd(en.residual, cm)(ut)
    want = omat.assemble_csr_data(oo, omat.element_tangents(oo, law, u), en.n_values, csr.indptr,
                                  csr.indices)
    f64 = dtype == torch.float64
    assert K.data.dtype == dtype
    assert rel(K.data, want) < (1e-12 if f64 else 1e-4)
    assert rel(K.data, _compressed(en, cm, ut)) < (1e-13 if f64 else 1e-5)


def test_extra_entries_and_nodes_without_elements(cuda):
    """A pattern with more couplings than the mesh has: the extra entries are zero."""
    c, e = om.kuhn_box((1, 1, 1), (3, 2, 3), origin=(0, 0, 0))
    c = np.concatenate([c, [[2.0, 2.0, 2.0]]])
    op = Operator(Mesh(c, e, device=cuda), element.Tetrahedron4())
    en = materials.NeoHookean(op, 1.0, 10.0)
    node = sparse.pattern_from_mesh(op.mesh, 1).tolil()
    nn = c.shape[0]
    node[0, nn - 2] = node[nn - 2, 0] = 1
    csr = sps.kron(node.tocsr(), np.ones((3, 3)), format="csr").astype(np.int8)
    csr.sort_indices()
    cm = sparse.ColoredMatrix.from_csr(csr, device=cuda)
    assert en.csr_slots(cm, cm.n_colors) is not None
    u = torch.as_tensor(0.01 * np.random.default_rng(1).standard_normal(en.n_dofs), device=cuda)
    K = sparse.jacfwd(en, cm)(u)
    assert rel(K.data, _compressed(en, cm, u)) < 1e-13
    assert K.to_csr()[0, 3 * (nn - 2)] == 0.0


@pytest.mark.parametrize("case", ["unsorted", "missing", "colours", "scalar_rows", "short"])
def test_refused_patterns_keep_the_compressed_route(cuda, case):
    op, oo, en, law, u, csr = _setup("tet4", (3, 2, 2), "neo_hookean", cuda)
    cm = sparse.ColoredMatrix.from_csr(csr, device=cuda)
    if case == "unsorted":  # two node blocks of every row swapped
        ix = csr.indices.copy()
        for r in range(csr.shape[0]):
            k = csr.indptr[r]
            ix[k:k + 6] = np.r_[csr.indices[k + 3:k + 6], csr.indices[k:k + 3]]
        cm = dataclasses.replace(cm, indices=torch.as_tensor(ix, device=cuda))
    elif case == "colours":  # not a distance-2 colouring: the entries of a colour add up
        cm = dataclasses.replace(cm, colors=(cm.colors % 5).contiguous())
    else:
        a = csr.tolil()
        if case == "missing":      # a coupling of the mesh left out, as a whole node block
            a[0:3, 3:6] = 0
        elif case == "scalar_rows":  # one entry left out: rows of a node differ
            a[0, 3] = 0
        else:
            a[csr.shape[0] - 3:, :] = 0
        csr2 = a.tocsr()
        csr2.eliminate_zeros()
        csr2.sort_indices()
        cm = sparse.ColoredMatrix.from_csr(csr2, colors=cm.colors.cpu().numpy(), device=cuda)
    assert en.csr_slots(cm, cm.n_colors) is None
    ut = torch.as_tensor(u, device=cuda)
    assert torch.equal(sparse.jacfwd(en.residual, cm)(ut).data, _compressed(en, cm, ut))


def test_long_rows_and_many_colours_are_refused(cuda):
    """A fan of tets around one node: its row block outgrows shared memory."""
    m = 160
    th = np.linspace(0, 2 * np.pi, m, endpoint=False)
    c = np.concatenate([[[0, 0, 0], [0, 0, 1]], np.stack([np.cos(th), np.sin(th), 0 * th], 1)])
    i = np.arange(m)
    e = np.stack([0 * i, 2 + i, 2 + (i + 1) % m, 0 * i + 1], 1).astype(np.int32)
    op = Operator(Mesh(c, e, device=cuda), element.Tetrahedron4())
    en = materials.LinearElastic(op, 0.7, 1.9)
    cm = sparse.ColoredMatrix.from_csr(sparse.pattern_from_mesh(op.mesh, 3), device=cuda)
    assert cm.n_colors <= 1024 and en.csr_slots(cm, cm.n_colors) is None
    u = torch.zeros(en.n_dofs, dtype=torch.float64, device=cuda)
    assert torch.equal(sparse.jacfwd(en.residual, cm)(u).data, _compressed(en, cm, u))
    po = materials.Poisson(op, 1.0, 0.0)  # one value per node: the same fan fits
    cm1 = sparse.ColoredMatrix.from_csr(sparse.pattern_from_mesh(op.mesh, 1), device=cuda)
    assert po.csr_slots(cm1, cm1.n_colors) is not None
    u1 = torch.zeros(po.n_dofs, dtype=torch.float64, device=cuda)
    assert rel(sparse.jacfwd(po, cm1)(u1).data, _compressed(po, cm1, u1)) < 1e-13
