"""Lists 1 and 3 from the one-launch CSR: leaf counts on both sides of its
64-leaf tiles, and lists longer than the fixed slots beside short ones (a dense
blob against the edge of a coarse leaf). Every list against the oracle."""
import numpy as np
import pytest

from lsmps_vpm_v2_b200 import VpmError, default_params

pytestmark = pytest.mark.gpu


def grid(side, drop):
    """One particle in the middle of each cell of a side x side grid, the last
    `drop` left out; leaves of at most one."""
    k = (np.arange(side) + 0.5) / side
    x, y = (g.ravel() for g in np.meshgrid(k, k))
    return x[: x.size - drop], y[: y.size - drop]


def blob(n, seed, rest=60):
    rng = np.random.default_rng(seed)
    x, y = rng.uniform(-1, 1, (2, n))
    k = n - rest
    x[:k], y[:k] = 0.01 * rng.uniform(size=k) - 0.01, rng.uniform(-1, 1, k)
    return x, y


CASES = {"leaves_1x": (grid(8, 0), 1), "leaves_4x": (grid(16, 0), 1), "leaves_less": (grid(16, 9), 1),
         "leaves_16x": (grid(32, 3), 1), "long": (blob(4000, 1), 8), "long_many": (blob(40000, 2), 8), "long_200": (blob(4000, 1, 200), 8),
         "long_600": (blob(4000, 1, 600), 8)}
REFUSED = ("long", "long_many")   # the walk of a leaf outgrows its queue of 160 cells


def oracle_lists(port, name):
    (x, y), cap = CASES[name]
    a = np.ones(x.size, np.uint8)
    kw = dict(max_src=cap, max_par=cap)
    return x, y, a, kw


@pytest.mark.parametrize("name", list(CASES))
def test_lists(ctx, port, name):
    x, y, a, kw = oracle_lists(port, name)
    if name in REFUSED:
        with pytest.raises(VpmError, match="queue overflow"):
            ctx.build_tree2d(x, y, a, default_params(**kw))
        return
    ctx.build_tree2d(x, y, a, default_params(**kw))
    lists = ctx.dump_tree2d()["lists"]
    for which in (1, 2, 3, 4):
        cid, offs, out = lists[which]
        po, pv = port.lists2d(x, y, a, which, cid, **kw)
        assert np.array_equal(offs, po), which
        for k in range(cid.size):
            assert sorted(out[offs[k]:offs[k + 1]]) == sorted(pv[po[k]:po[k + 1]]), (which, cid[k])
