"""The FP64 list-2 M2L on both sides of the line between a warp per target cell
and the kernel per parent, whose line is at 1,200 expected leaves up to p = 14
and at 4,000 above: field and potential against the oracle, and the captured
field against the eager one, bit for bit."""
import numpy as np
import pytest

from lsmps_vpm_v2_b200 import default_params
from lsmps_vpm_v2_b200.workloads import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-10   # FP64 in another order of operations
CAP = 5


@pytest.mark.parametrize("p,leaves", [(14, 1200), (15, 4000), (16, 4000)])
@pytest.mark.parametrize("above", [0, 1])
def test_both_sides(ctx, port, p, leaves, above):
    n = CAP * leaves - 1 + above
    rng = np.random.default_rng(n + p)
    xy = rng.uniform(-1.0, 1.0, (2, n))
    xy[:, : n // 3] = 0.3 + 0.05 * rng.normal(size=(2, n // 3))
    q, a = rng.normal(size=n), (rng.uniform(size=n) >= 0.1).astype(np.uint8)
    kw = dict(p=p, max_src=CAP, max_par=CAP)
    out = ctx.field2d(*xy, q, a, default_params(**kw))
    assert rel_l2(out, port.fmm2d_field(*xy, q, a, **kw)) <= TOL
    assert rel_l2([ctx.potential2d(*xy, q, a, default_params(**kw))], [port.fmm2d_potential(*xy, q, a, **kw)]) <= TOL
    graph = ctx.field2d(*xy, q, a, default_params(use_graph=1, **kw))
    assert np.array_equal(out[0], graph[0]) and np.array_equal(out[1], graph[1])
