"""Hex8 energies of displacements that are not finite: the infinity that the sums over the nodes
give (a trial step far out compares as larger than any state), NaN where they give NaN."""

import numpy as np
import pytest
import torch

from oracle import mesh as om
from tatva_gb300 import Mesh, Operator, element, materials

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("law", ["linear_elastic", "poisson"])
@pytest.mark.parametrize("corner", [0, 3, 6])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_infinite_displacements(cuda, law, corner, dtype):
    c, e = om.brick(4, 3, 3)
    rng = np.random.default_rng(1)
    c = c + 0.05 * rng.uniform(-1, 1, c.shape)  # no shape gradient with a zero component
    op = Operator(Mesh(c, e, device=cuda), element.Hexahedron8())
    en = (materials.LinearElastic(op, 0.7, 1.9) if law == "linear_elastic"
          else materials.Poisson(op, 1.3, 0.6))
    u = 0.1 * rng.standard_normal((c.shape[0], en.n_values))
    ok = en.energy_per_element(torch.as_tensor(u, dtype=dtype, device=cuda))
    node = e[17, corner]
    u[node, -1] = -np.inf  # Poisson: 1/2 kappa |grad u|^2 - f u is +infinity too
    got = en.energy_per_element(torch.as_tensor(u, dtype=dtype, device=cuda))
    touched = torch.as_tensor((e == node).any(1), device=cuda)
    assert torch.isposinf(got[touched]).all()
    assert torch.equal(got[~touched], ok[~touched])
    assert torch.isposinf(en.value(torch.as_tensor(u, dtype=dtype, device=cuda)))
    u[node, -1] = np.nan
    got = en.energy_per_element(torch.as_tensor(u, dtype=dtype, device=cuda))
    assert torch.isnan(got[touched]).all() and torch.equal(got[~touched], ok[~touched])
