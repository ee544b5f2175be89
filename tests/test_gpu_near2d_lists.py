"""The near field and M2P of a leaf with more than 64 cells in list 1 (more than
one staged segment) and more than the 32 fixed slots in lists 1 and 3 (the
captured evaluation's spill pass): a coarse leaf whose right neighbour is refined
six levels along their common edge. Field and potential against the oracle, the
captured field against the eager one."""
import numpy as np
import pytest

from lsmps_vpm_v2_b200 import PREC_MIXED, default_params
from lsmps_vpm_v2_b200.workloads import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-10   # FP64 sums of a few thousand terms in another order
ROOT, LOW = 2.02, -1.01   # the box of particles from -1 to 1, one per cent wider
DEEP = 6


def cell(rng, level, ix, iy, n):
    """n particles inside a cell, clear of its edges."""
    h = ROOT / 2**level
    return np.stack([LOW + (ix + rng.uniform(0.1, 0.9, n)) * h, LOW + (iy + rng.uniform(0.1, 0.9, n)) * h])


def refined_edge(cap):
    """Leaf (3, 4) of level 3 holds `cap` particles; cell (4, 4) is refined along
    x = its left edge, a few particles in the column beside it on every level."""
    rng = np.random.default_rng(cap)
    parts = [np.array([[-1.0, 1.0], [-1.0, 1.0]]), cell(rng, 3, 3, 4, cap)]
    for ix in range(8):
        for iy in range(8):
            if (ix, iy) not in ((3, 4), (4, 4), (0, 0), (7, 7)):
                parts.append(cell(rng, 3, ix, iy, 3))
    for d in range(1, DEEP + 1):
        for row in range(2**d):
            parts.append(cell(rng, 3 + d, 4 * 2**d + 1, 4 * 2**d + row, 1))
    for row in range(2**DEEP):
        parts.append(cell(rng, 3 + DEEP, 4 * 2**DEEP, 4 * 2**DEEP + row, cap * 5 // 8))
    x, y = np.concatenate(parts, axis=1)
    return x.copy(), y.copy(), rng.normal(size=x.size), np.ones(x.size, np.uint8)


@pytest.mark.parametrize("cap", [8, 40, 200])
def test_long_lists(ctx, port, cap):
    x, y, q, a = refined_edge(cap)
    kw = dict(max_src=cap, max_par=cap)
    eager = ctx.field2d(x, y, q, a, default_params(**kw))
    lists = ctx.dump_tree2d()["lists"]
    n1, n3 = (np.diff(lists[which][1]) for which in (1, 3))
    assert n1.max() > 64 and n3[n1.argmax()] > 32
    ref = port.fmm2d_field(x, y, q, a, **kw)
    assert rel_l2(eager, ref) <= TOL
    assert rel_l2([ctx.potential2d(x, y, q, a, default_params(**kw))], [port.fmm2d_potential(x, y, q, a, **kw)]) <= TOL
    graph = ctx.field2d(x, y, q, a, default_params(use_graph=1, **kw))
    assert np.array_equal(eager[0], graph[0]) and np.array_equal(eager[1], graph[1])
    mixed = ctx.field2d(x, y, q, a, default_params(precision=PREC_MIXED, **kw))
    graph = ctx.field2d(x, y, q, a, default_params(precision=PREC_MIXED, use_graph=1, **kw))
    assert np.array_equal(mixed[0], graph[0]) and np.array_equal(mixed[1], graph[1])
