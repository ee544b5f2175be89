"""Strengths that are not finite, in the potential: they reach every other
particle, and leave the one that carries them as it is without its own."""
import numpy as np
import pytest

from lsmps_vpm_v2_b200 import default_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("n,cap", [(40, 50), (700, 5), (3000, 50), (3000, 250)])
def test_own_strength(ctx, n, cap, value):
    rng = np.random.default_rng(n + cap)
    x, y = rng.uniform(-1.0, 1.0, (2, n))
    q, a = rng.normal(size=n), np.ones(n, np.uint8)
    prm = default_params(max_src=cap, max_par=cap)
    for i in rng.integers(0, n, 4):
        without, with_ = q.copy(), q.copy()
        without[i], with_[i] = 0.0, value
        phi, ref = ctx.potential2d(x, y, with_, a, prm), ctx.potential2d(x, y, without, a, prm)
        assert phi[i] == ref[i]
        assert not np.isfinite(np.delete(phi, i)).any()
