"""Leaf caps up to the largest integer, as a caller gives them who wants no
limit: the tree and the values of caps of n, on every form of the particle sort
(one block, a cluster, the grid, the full keys of 31 levels)."""
import numpy as np
import pytest

from lsmps_vpm_v2_b200 import PREC_MIXED, default_params

pytestmark = pytest.mark.gpu
MOST = 2**31 - 1


@pytest.mark.parametrize("n", [2, 900, 5000, 40_000])
@pytest.mark.parametrize("caps", [(MOST, MOST), (MOST - 1, 60), (60, MOST)])
@pytest.mark.parametrize("form", [dict(), dict(max_depth=31), dict(precision=PREC_MIXED, use_graph=1)])
def test_no_limit(ctx, n, caps, form):
    rng = np.random.default_rng(n)
    x, y = rng.uniform(-1.0, 1.0, (2, n))
    q, a = rng.normal(size=n), (rng.uniform(size=n) >= 0.2).astype(np.uint8)
    a[0] = 1
    least = [min(c, n) for c in caps]
    out = ctx.field2d(x, y, q, a, default_params(max_src=caps[0], max_par=caps[1], **form))
    ref = ctx.field2d(x, y, q, a, default_params(max_src=least[0], max_par=least[1], **form))
    assert np.array_equal(out[0], ref[0]) and np.array_equal(out[1], ref[1])


@pytest.mark.parametrize("cap", [MOST, MOST - 5])
def test_no_limit_3d(ctx, cap):
    rng = np.random.default_rng(3)
    v = [*rng.uniform(-1.0, 1.0, (3, 700)), *rng.normal(size=(3, 700)), np.ones(700, np.uint8)]
    out = ctx.velocity3d_alpha(*v, default_params(leaf_cap_3d=cap))
    ref = ctx.velocity3d_alpha(*v, default_params(leaf_cap_3d=701))
    assert np.array_equal(out, ref)
