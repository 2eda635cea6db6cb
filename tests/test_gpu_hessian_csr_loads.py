"""CSR tangent with connectivity rows that do and do not start on 16-byte boundaries (rows
loaded whole or entry by entry), on meshes whose nodes have one to many elements (the loads
run ahead of the element work): the same bits."""

import ctypes

import numpy as np
import pytest
import torch

from oracle import mesh as om
from tatva_gb300 import Mesh, Operator, _lib, element, materials, sparse
from tatva_gb300._device import prec_of, ptr, stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 1, 3), (5, 4, 3)])
@pytest.mark.parametrize("elem", ["tet4", "hex8"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_unaligned_connectivity(cuda, shape, elem, dtype):
    c, e = (om.kuhn_box((1, 1, 1), shape, origin=(0, 0, 0)) if elem == "tet4"
            else om.brick(*shape))
    op = Operator(Mesh(c, e, device=cuda),
                  element.Tetrahedron4() if elem == "tet4" else element.Hexahedron8())
    en = materials.NeoHookean(op, 1.0, 1.5)
    cm = sparse.ColoredMatrix.from_csr(sparse.pattern_from_mesh(op.mesh, 3), device=cuda)
    u = torch.as_tensor(np.random.default_rng(1).standard_normal(c.size) * 1e-2, dtype=dtype,
                        device=cuda)
    slots = en.csr_slots(cm, cm.n_colors)
    assert slots is not None
    want = en.tangent_csr(u, cm, slots)
    ip, ii = op.incidence()
    row = op.mesh.elements.reshape(-1)
    m = en.material(dtype)
    for shift in (1, 2, 3):
        conn = torch.zeros(row.numel() + shift, dtype=torch.int32, device=cuda)[shift:]
        conn.copy_(row)
        assert conn.data_ptr() % 16 != 0
        got = torch.full_like(want, float("nan"))
        _lib.call("tg_hessian_csr", op.element.tg_id, prec_of(dtype), ctypes.byref(m),
                  ptr(op.coords_as(dtype)), op.n_nodes, ptr(conn), op.n_elements, ptr(u), ptr(ip),
                  ptr(ii), ptr(slots[0]), ptr(cm.indptr), slots[1], ptr(got), stream())
        assert torch.equal(got, want)
