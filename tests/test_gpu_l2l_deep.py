"""Local expansions of leaves far below the dense grid of cells, whose ancestors
come from the parent chain: nested blobs, every tenth the size of the last,
against the oracle."""
import numpy as np
import pytest

from lsmps_vpm_v2_b200 import BINOM_EXACT, default_params
from lsmps_vpm_v2_b200.workloads import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-10   # FP64 in another order of operations


def nested(blobs, per, seed):
    rng = np.random.default_rng(seed)
    xy = np.concatenate([rng.normal(size=(2, per)) * 0.1**i for i in range(blobs)], axis=1)
    return xy[0].copy(), xy[1].copy(), rng.normal(size=blobs * per), np.ones(blobs * per, np.uint8)


@pytest.mark.parametrize("p,exact", [(1, False), (5, False), (16, False), (18, True), (24, True)])
@pytest.mark.parametrize("blobs,per", [(2, 900), (7, 400)])
def test_deep_leaves(ctx, port, p, exact, blobs, per):
    d = nested(blobs, per, p)
    kw = dict(p=p, max_src=20, max_par=30)
    *out, stats = ctx.field2d(*d, default_params(binom=BINOM_EXACT if exact else 0, **kw), stats=True)
    assert blobs == 2 or stats.max_level >= 20
    assert rel_l2(out, port.fmm2d_field(*d, exact_binom=exact, **kw)) <= TOL
