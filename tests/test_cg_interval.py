"""Length of the CG's launches (a host query): what a solve may ask for in one launch stays far
from where the 32-bit arrival counter of the cooperative launch wraps (2^32 arrivals, four a CTA
and iteration, 152 CTAs: seven million iterations)."""

import ctypes

import pytest

from tatva_gb300 import _lib


def _desc(nodes, kind=_lib.TG_LINEAR_ELASTIC):
    plan = _lib.BlockPlan()
    plan.grid_nodes[:] = nodes
    plan.grid_h[:] = (1.0, 1.0, 1.0)
    op = _lib.OperatorDesc()
    op.elem, op.prec = _lib.TG_HEX8, _lib.TG_F32
    op.mat.kind = kind
    op.plan = ctypes.addressof(plan)
    op.n_nodes = max(nodes[0] * nodes[1] * nodes[2], 8)
    return op, plan


def _interval(op, k):
    return _lib.lib().tg_cg_check_interval(ctypes.byref(op), k)


@pytest.mark.parametrize("every,want", [(-3, 16), (0, 16), (1, 16), (50, 800), (4096, 65536),
                                        (4097, 65536), (600_000, 65536), (2**31 - 1, 65536)])
def test_a_cooperative_launch_is_bounded(every, want):
    op, keep = _desc((65, 65, 65))
    assert _interval(op, every) == want
    assert 4 * 512 * want < 2**31  # 512 CTAs at most


@pytest.mark.parametrize("every,want", [(0, 1), (1, 1), (50, 50), (600_000, 600_000)])
def test_separate_launches_keep_the_interval(every, want):
    for op, keep in (_desc((130, 129, 129)), _desc((0, 0, 0)),
                     _desc((65, 65, 65), _lib.TG_NEO_HOOKEAN)):
        assert _interval(op, every) == want
