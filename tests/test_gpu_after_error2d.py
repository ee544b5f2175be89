"""A context after an evaluation that ended in a fatal error (non-finite
positions, a tree deeper than the keys, too few cells): every kernel behind the
tree build returns, and the next evaluation on the same arena gives the bits of
the one before."""
import numpy as np
import pytest

from lsmps_vpm_v2_b200 import PREC_MIXED, Context, VpmError, default_params

pytestmark = pytest.mark.gpu


def scatter(n, seed):
    rng = np.random.default_rng(seed)
    return (*rng.uniform(-1.0, 1.0, (2, n)), rng.normal(size=n), np.ones(n, np.uint8))


def not_finite(n):
    x, y, q, a = scatter(n, 2)
    x[n // 2] = np.nan
    return x, y, q, a


def coincident(n):
    """A third of the particles in one point: deeper than any key."""
    x, y, q, a = scatter(n, 3)
    x[: n // 3], y[: n // 3] = 0.25, 0.125
    return x, y, q, a


def deep(n):
    """A blob that needs more than 16 levels: evaluated again with 31."""
    x, y, q, a = scatter(n, 4)
    x[: n // 3] = 0.25 + 1e-6 * x[: n // 3]
    y[: n // 3] = 0.125 + 1e-6 * y[: n // 3]
    return x, y, q, a


def many_cells(n):
    """Pairs of near particles, caps of one: more than eight cells a particle."""
    x, y, q, a = scatter(n, 5)
    x[1::2], y[1::2] = x[::2][: n // 2] + 2e-7, y[::2][: n // 2]
    return x, y, q, a


@pytest.mark.parametrize("bad,caps,error", [(not_finite, (50, 75), "non-finite"), (coincident, (50, 75), "deeper"),
                                            (deep, (50, 75), None), (many_cells, (1, 1), None)])
@pytest.mark.parametrize("op", ["field", "field_graph", "mixed_graph", "potential"])
def test_next_evaluation_is_whole(op, bad, caps, error):
    ctx = Context(0)
    form = dict(use_graph=int("graph" in op), precision=PREC_MIXED if "mixed" in op else 0, p=12)
    call = ctx.potential2d if op == "potential" else ctx.field2d
    good = scatter(20_000, 1)
    prm = default_params(max_src=50, max_par=75, **form)
    before = np.array(call(*good, prm))
    args = (*bad(20_000), default_params(max_src=caps[0], max_par=caps[1], **form))
    if error:
        with pytest.raises(VpmError, match=error):
            call(*args)
    else:
        assert np.isfinite(np.array(call(*args))).all()
    assert np.array_equal(before, np.array(call(*good, prm)))
    ctx.close()
