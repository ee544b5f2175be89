"""The particle sort at the edges of its forms: one block, clusters of 2 to 16
blocks and the first size of the grid form; keys that share their upper levels
(sorted again with all passes); few active particles and source caps above the
particle caps, where the leaf's source limit is what the records look for.
Trees cell for cell against the oracle."""
import numpy as np
import pytest

from lsmps_vpm_v2_b200 import VpmError, default_params
from test_gpu_parity2d import _tree_equal

pytestmark = pytest.mark.gpu


def check(ctx, port, x, y, act, **kw):
    ctx.build_tree2d(x, y, act, default_params(**kw))
    _tree_equal(ctx.dump_tree2d(), port.tree2d(x, y, act, **kw))


@pytest.mark.parametrize("n", [1, 2, 33, 1023, 1024, 1025, 2049, 4097, 8193, 16384, 16385, 32767, 32768, 32769])
def test_sizes(ctx, port, n):
    rng = np.random.default_rng(n)
    x, y = rng.uniform(-1, 1, (2, n))
    act = (rng.uniform(size=n) < 0.5).astype(np.uint8)
    if n == 1:   # a single particle has no root cell: refused
        with pytest.raises(VpmError):
            check(ctx, port, x, y, act)
        return
    check(ctx, port, x, y, act)


@pytest.mark.parametrize("n", [1500, 20000, 40000])
@pytest.mark.parametrize("scale", [1e-2, 1e-4])
def test_deep(ctx, port, n, scale):
    rng = np.random.default_rng(n)
    x, y = rng.uniform(-1, 1, (2, n))
    x[: n // 2], y[: n // 2] = 0.3 + scale * rng.uniform(-1, 1, (2, n // 2))
    check(ctx, port, x, y, np.ones(n, np.uint8))


@pytest.mark.parametrize("n", [3000, 40000])
@pytest.mark.parametrize("share", [0.0, 0.01, 0.9])
@pytest.mark.parametrize("max_src,max_par", [(5, 200), (100, 40), (0, 30), (50, 75)])
def test_active_limit(ctx, port, n, share, max_src, max_par):
    rng = np.random.default_rng(n)
    x, y = rng.uniform(-1, 1, (2, n))
    act = (rng.uniform(size=n) < share).astype(np.uint8)
    if max_src == 0 and act.any():   # a cell with an active particle never becomes a leaf: refused
        with pytest.raises(VpmError, match="deeper than the key resolution"):
            check(ctx, port, x, y, act, max_src=max_src, max_par=max_par)
        return
    check(ctx, port, x, y, act, max_src=max_src, max_par=max_par)
