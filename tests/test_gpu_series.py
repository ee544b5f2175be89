"""The logarithm of the FP64 potential and the reciprocal root of the FP64 3D
evaluation, each seen alone: one source of strength one, all other particles at
chosen distances with strength zero."""
import numpy as np
import pytest

from lsmps_vpm_v2_b200 import default_params

pytestmark = pytest.mark.gpu
EPS = 2.0**-53


def log_half(r2):
    """log(r2) / 2 in extended precision."""
    return np.log(r2.astype(np.longdouble)) / 2


def potential(ctx, dx, apart):
    """Potential at (dx, 0) of a source at the origin, no cell below level 1; one
    call for all dx, or (apart) one for each, where the square of the distance of
    two of them could vanish."""
    if apart:
        return np.concatenate([potential(ctx, dx[i:i + 1], False) for i in range(dx.size)])
    x = np.concatenate([[0.0], dx])
    q = np.zeros(x.size)
    q[0] = 1.0
    prm = default_params(max_src=x.size, max_par=x.size)
    return ctx.potential2d(x, np.zeros(x.size), q, np.ones(x.size, np.uint8), prm)[1:]


SQRT_HALF = np.sqrt(0.5)


@pytest.mark.parametrize("name", ["one", "root_half", "mantissas", "small", "large", "ends"])
def test_log_of_the_potential(ctx, name):
    """r^2 next to 1 (where the logarithm vanishes), next to sqrt(1/2) and its
    double (the two ends of the reduced argument), over all mantissas and
    exponents, and on both sides of 2^-1007 and 2^1009, where CUDA's log takes
    over. Stated: at most 3.3e-16 of the logarithm, taken of the rounded r^2; one
    rounding is allowed on top."""
    rng = np.random.default_rng(len(name))
    if name == "one":
        dx = 1.0 + np.concatenate([np.arange(-400, 400) * 2.0**-52, rng.uniform(-1, 1, 1000) * 2.0 ** -rng.uniform(4, 50, 1000)])
    elif name == "root_half":
        dx = 2.0 ** rng.integers(-3, 4, 2000) * SQRT_HALF**0.5 * (1 + rng.integers(-300, 300, 2000) * 2.0**-52)
    elif name == "mantissas":
        dx = 2.0 ** rng.uniform(-30, 30, 4000)
    elif name == "small":
        dx = 2.0 ** rng.uniform(-503, -30, 700)
    elif name == "large":
        dx = 2.0 ** rng.uniform(30, 504, 2000)
    else:
        e = np.concatenate([np.full(350, -503.5), np.full(350, 504.5)])
        dx = 2.0**e * (1 + rng.uniform(-1, 1, 700) * 2.0 ** -rng.uniform(1, 40, 700))
    dx = np.unique(dx)
    dx *= rng.choice([-1.0, 1.0], dx.size)
    ref = log_half(dx * dx)
    assert (np.abs(potential(ctx, dx, name in ("small", "ends")) - ref) <= (3.3e-16 + EPS) * np.abs(ref)).all()


@pytest.mark.parametrize("scale", [1.0, 2.0**-40, 2.0**41, 2.0**-101, 2.0**100])
def test_reciprocal_root_of_the_3d_form(ctx, scale):
    """u = alpha x r / r^3 of one source, alone, at the particles of its near
    leaves. The root's step leaves an error of order e^3 with e below 2^-19, far
    under a unit; r^2 (three roundings), the third power of the root, the cross
    product and the sum come to ten units at most."""
    rng = np.random.default_rng(7)
    n = 400
    p = rng.uniform(-1.0, 1.0, (3, n))
    p[:, 0] = 0.1
    near = slice(1, 28)   # in the source's own leaf
    p[:, near] = p[:, :1] + rng.uniform(-1.0, 1.0, (3, 27)) * 10.0 ** rng.uniform(-5, -2.2, 27)
    a = np.zeros((3, n))
    a[:, 0] = (0.3, -0.7, 0.5)
    u = np.array(ctx.velocity3d_alpha(*(p * scale), *a, np.ones(n, np.uint8), default_params(leaf_cap_3d=30)))
    tree = ctx.dump_tree3d()
    own = [set(tree["leaf_pids"][b:e]) for b, e in zip(tree["leaf_offs"][:-1], tree["leaf_offs"][1:])]
    assert any({0, *range(1, 28)} <= leaf for leaf in own)   # or the sums below would hold far cells
    r = (p * scale).astype(np.longdouble)[:, near] - (p * scale).astype(np.longdouble)[:, :1]
    ref = np.cross(a[:, 0].astype(np.longdouble), r.T).T / np.sqrt((r * r).sum(axis=0)) ** 3
    size = np.linalg.norm(a[:, 0]) * np.sqrt((r * r).sum(axis=0)) / np.sqrt((r * r).sum(axis=0)) ** 3
    assert (np.abs(u[:, near] - ref) <= 10 * 2 * EPS * size).all()
