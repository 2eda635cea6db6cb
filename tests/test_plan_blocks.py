"""The default block size of an element-block plan: small meshes are cut into enough
blocks to fill the GPU, and no default plan outgrows the fixed scratch of
``tg_apply_noalloc`` because of it (host only)."""

import numpy as np
import pytest

from oracle import mesh as om
from tatva_gb300 import Mesh, Operator, element
from tatva_gb300.plan import (DEFAULT_BLOCK_ELEMS, SMALL_MESH_BLOCKS, SMALL_PLAN_PARTIALS,
                              small_mesh_blocks)


@pytest.mark.parametrize("n", [1, 63, 64, 76_799, 76_800, 307_199, 307_200, 614_399])
def test_small_meshes_get_enough_blocks(n):
    be, threads = small_mesh_blocks(1, n)
    assert 64 <= be <= 512 and threads in (64, 128)
    assert be == 64 or n // be >= SMALL_MESH_BLOCKS


def test_large_meshes_keep_the_default_blocks():
    assert small_mesh_blocks(1, 614_400) is None and small_mesh_blocks(2, 2_097_152) is None


def test_default_plans_by_mesh_and_law():
    c, e = om.kuhn_box((1, 1, 1), (5, 4, 6), origin=(0, 0, 0))
    op = Operator(Mesh(c, e, device="cpu"), element.Tetrahedron4())
    assert op.plan().block_elems == 64 and op.plan() is op.plan(box_kernels=False)
    c, e = om.brick(16, 8, 8)
    op = Operator(Mesh(c, e, device="cpu"), element.Hexahedron8())
    assert op.plan().sizes["n_lattice_blocks"] == 2          # linear elasticity: box kernels
    assert op.plan(box_kernels=False).block_elems == 64      # the other laws
    op = Operator(Mesh(om.jitter_interior(c, 1 / 16, 0.2, seed=0), e, device="cpu"),
                  element.Hexahedron8())
    assert op.plan().block_elems == 64


def test_scattered_connectivity_keeps_the_default_plan():
    """Elements that share almost every node with elements elsewhere: the small blocks
    would need more partial slots than the fixed scratch holds."""
    rng = np.random.default_rng(0)
    n_nodes, n_elems = 100_000, 400_000
    e = np.stack([rng.integers(0, n_nodes // 4, n_elems) + k * (n_nodes // 4) for k in range(4)], 1)
    op = Operator(Mesh(rng.random((n_nodes, 3)), e.astype(np.int32), device="cpu"),
                  element.Tetrahedron4())
    small = op.plan(512, 4096, 128)
    assert small.sizes["n_partials"] > SMALL_PLAN_PARTIALS
    assert op.plan().block_elems == DEFAULT_BLOCK_ELEMS[1]
