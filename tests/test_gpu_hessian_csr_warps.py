"""CSR tangent at node counts around the 32 nodes of a warp and the 64 of two, for the types and
row lengths that take CTAs of one warp (FP64 Hex8) and of two (the others): against the
compressed Hessian with decompression (the same element formula, other rounding)).

Tolerance, relative to the largest entry: an entry sums up to eight elements of up to eight
points, with about eight roundings a product: 512 roundings of 2^-53 (FP64) or 2^-24 (FP32)."""

import numpy as np
import pytest
import torch

from oracle import mesh as om
from tatva_gb300 import Mesh, Operator, element, materials, sparse

pytestmark = pytest.mark.gpu

LAWS = {"poisson": (materials.Poisson, 1.3, 0.6),
        "linear_elastic": (materials.LinearElastic, 0.7, 1.9)}


# 2 x 2 x k nodes: 28, 32, 36, 60, 64, 68; 63; 195 with rows of eight to 27 columns
@pytest.mark.parametrize("shape", [(1, 1, 6), (1, 1, 7), (1, 1, 8), (1, 1, 14), (1, 1, 15),
                                   (1, 1, 16), (2, 2, 6), (2, 4, 12)])
@pytest.mark.parametrize("kind", list(LAWS))
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("elem", ["hex8", "tet4"])
def test_node_counts(cuda, elem, shape, kind, dtype):
    c, e = om.brick(*shape) if elem == "hex8" else om.kuhn_box((1, 1, 1), shape, origin=(0, 0, 0))
    c = c + 0.1 / max(shape) * np.random.default_rng(3).uniform(-1, 1, c.shape)
    op = Operator(Mesh(c, e, device=cuda),
                  element.Hexahedron8() if elem == "hex8" else element.Tetrahedron4())
    cls, *par = LAWS[kind]
    en = cls(op, *par)
    cm = sparse.ColoredMatrix.from_csr(sparse.pattern_from_mesh(op.mesh, en.n_values), device=cuda)
    slots = en.csr_slots(cm, cm.n_colors)
    assert slots is not None
    u = torch.zeros(en.n_dofs, dtype=dtype, device=cuda)
    want = sparse.decompress(en.compressed_hessian(u, cm.colors, cm.n_colors),
                             *sparse.compute_rows_cols(cm)).double()
    got = en.tangent_csr(u, cm, slots).double()
    eps = 2.0 ** -53 if dtype == torch.float64 else 2.0 ** -24
    assert float((got - want).abs().max()) <= 512 * eps * float(want.abs().max())
