"""The 2D translations: M2M of the large cells and L2L of the leaves (one lane
per expansion, every order has its own instantiation) and the FP64 list-2 M2L
per parent (orders 1..16, trees above its size rule), against the oracle, with
the reference's and with exact binomials, on trees with leaves on many levels."""
import numpy as np
import pytest

from lsmps_vpm_v2_b200 import BINOM_EXACT, default_params
from lsmps_vpm_v2_b200.workloads import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-10   # FP64 in another order of operations


def scatter(n, seed, blob):
    """A lattice-free set, half of it in a blob: cells above 1,024 particles on
    several levels, an empty corner (missing children), a tenth inactive."""
    rng = np.random.default_rng(seed)
    p = rng.uniform(-1.0, 1.0, (n, 2))
    p[: n // 2] = -0.3 + blob * rng.normal(size=(n // 2, 2))
    p = p[~((p[:, 0] > 0.4) & (p[:, 1] > 0.1))]
    q = rng.normal(0.0, 1.0, len(p))
    return p[:, 0].copy(), p[:, 1].copy(), q, (rng.uniform(size=len(p)) >= 0.1).astype(np.uint8)


@pytest.mark.parametrize("p", [1, 2, 3, 5, 7, 8, 9, 11, 13, 14, 15, 16, 17, 18])
def test_per_parent_m2l_and_shifts(ctx, port, p):
    """Leaf cap 5: about 10,000 / 5 leaves, above the per-parent rule (p <= 16)."""
    x, y, q, a = scatter(10_000, p, 0.05)
    kw = dict(p=p, max_src=5, max_par=5)
    assert rel_l2(ctx.field2d(x, y, q, a, default_params(**kw)), port.fmm2d_field(x, y, q, a, **kw)) <= TOL
    assert rel_l2(ctx.potential2d(x, y, q, a, default_params(**kw)), port.fmm2d_potential(x, y, q, a, **kw)) <= TOL


@pytest.mark.parametrize("p", [6, 12, 17, 19, 22, 26, 30])
def test_exact_binomials(ctx, port, p):
    x, y, q, a = scatter(6_000, p, 0.2)
    kw = dict(p=p, max_src=20, max_par=30)
    ref = port.fmm2d_field(x, y, q, a, exact_binom=True, **kw)
    assert rel_l2(ctx.field2d(x, y, q, a, default_params(binom=BINOM_EXACT, **kw)), ref) <= TOL
