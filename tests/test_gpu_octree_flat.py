"""The octree's two constructions: the flat one from ten-level keys (leaves of
at most 64 particles) and the level-by-level one that takes over in the same
call when the tree is deeper than the keys, or from the start when leaves are
larger. Trees cell for cell and velocities against the oracle."""
import numpy as np
import pytest

from test_gpu_parity3d import TOL, assert_same_tree, params, rel_l2

pytestmark = pytest.mark.gpu


def blob(n, scale, seed):
    """Half the particles in a blob of the given size, a fifth inactive:
    depth grows with log2(1 / scale)."""
    rng = np.random.default_rng(seed)
    p = rng.uniform(-1.0, 1.0, (n, 3))
    p[: n // 2] = 0.3 + scale * rng.normal(size=(n // 2, 3))
    p = p[rng.permutation(n)]
    return (*np.ascontiguousarray(p.T), *rng.normal(0.0, 1e-3, (3, n))), (rng.uniform(size=n) >= 0.2).astype(np.uint8)


@pytest.mark.parametrize("scale,deep", [(0.1, False), (1e-3, True), (1e-6, True)])
@pytest.mark.parametrize("leaf_cap", [4, 33, 65, 66])
def test_tree_and_velocity(ctx, port, scale, deep, leaf_cap):
    args, act = blob(5000, scale, 7)
    ints, geom = port.tree3d(*args[:3], act, leaf_cap=leaf_cap)
    if leaf_cap == 4:
        assert (int(ints[0, 5]) > 10) == deep
    ctx.build_tree3d(*args[:3], act, params(leaf_cap))
    dump = ctx.dump_tree3d()
    assert_same_tree(dump, ints, geom)
    offs, pids = dump["leaf_offs"], dump["leaf_pids"]
    assert np.array_equal(np.sort(pids), np.arange(5000))
    for k in np.flatnonzero(np.diff(offs) > 1):
        assert np.all(np.diff(pids[offs[k]:offs[k + 1]]) > 0)
    ref = port.fmm3d_velocity(*args, act, leaf_cap=leaf_cap)
    assert rel_l2(ctx.velocity3d_alpha(*args, act, params(leaf_cap)), ref) <= TOL


@pytest.mark.parametrize("n", [1, 2, 31, 1023, 1024, 1025])
def test_small_sets(ctx, port, n):
    args, act = blob(n, 0.2, n)
    ints, geom = port.tree3d(*args[:3], act, leaf_cap=8)
    ctx.build_tree3d(*args[:3], act, params(8))
    assert_same_tree(ctx.dump_tree3d(), ints, geom)
