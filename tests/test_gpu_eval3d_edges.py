"""The 3D evaluation at the edges of its blocks (64 targets, two per lane) and
of its rule for the warps per block (eight up to 296 blocks, 18,944 particles):
both tree paths against the oracle, target flags that empty one half of a
block or a whole block, and the mixed form against the plain one."""
import numpy as np
import pytest

from lsmps_vpm_v2_b200._lib import PREC_MIXED, default_params, treecell3d_params

pytestmark = pytest.mark.gpu

TOL = 1e-10          # FP64: both sum a few thousand terms, in another order (eps times their number)
TOL_MIXED = 1e-5     # FP32 terms (6e-8 each), FP64 sums


def rel_l2(a, b):
    a, b = np.concatenate([np.ravel(v) for v in a]), np.concatenate([np.ravel(v) for v in b])
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def cloud(n, seed):
    """Two thirds in a cube, one third in a dense blob (leaves on several
    levels), a tenth inactive."""
    rng = np.random.default_rng(seed)
    p = rng.uniform(-1.0, 1.0, (n, 3))
    p[: n // 3] = 0.2 + 0.1 * rng.normal(size=(n // 3, 3))
    p = p[rng.permutation(n)]
    a = rng.normal(0.0, 1e-3, (3, n))
    return (*np.ascontiguousarray(p.T), *a), (rng.uniform(size=n) >= 0.1).astype(np.uint8)


@pytest.mark.parametrize("n", [511, 512, 513, 544, 545, 577, 18944, 18945])
def test_octree_velocity_at_block_edges(ctx, port, n):
    args, act = cloud(n, n)
    ref = port.fmm3d_velocity(*args, act)
    plain = ctx.velocity3d_alpha(*args, act, default_params())
    assert rel_l2(plain, ref) <= TOL
    assert rel_l2(ctx.velocity3d_alpha(*args, act, default_params(precision=PREC_MIXED)), plain) <= TOL_MIXED


@pytest.mark.parametrize("n", [1600, 1601, 18945])
@pytest.mark.parametrize("pick", ["left", "few", "none"])
def test_treecell_targets(ctx, port, n, pick):
    args, act = cloud(n, n + 1)
    tgt = {"left": args[0] < 0.0, "few": np.arange(n) % 97 == 5, "none": np.zeros(n, bool)}[pick].astype(np.uint8)
    ref = port.treecell3d_velocity(*args, act)
    for form, tol in ((0, TOL), (PREC_MIXED, TOL_MIXED)):
        out = ctx.velocity3d_treecell(*args, act, tgt, treecell3d_params(precision=form))
        assert all(np.all(v[tgt == 0] == 0.0) for v in out)
        if tgt.any():
            assert rel_l2([v[tgt == 1] for v in out], [v[tgt == 1] for v in ref]) <= tol
