"""The FP64 near field (field and potential) where its tiling can go wrong:
leaves of 1 to some hundreds of particles around the chunk of 192 targets and
around each number of targets per lane, lists longer than one segment of 64
cells, coincident particles, and the captured graph (lists from the slots and,
for leaves that outgrew them, from the CSR) against the eager call."""
import numpy as np
import pytest

from lsmps_vpm_v2_b200 import default_params
from lsmps_vpm_v2_b200.workloads import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-10   # FP64 sums of a few thousand terms in another order


def points(n, seed, blob=0.0):
    rng = np.random.default_rng(seed)
    p = rng.uniform(-1.0, 1.0, (n, 2))
    if blob:
        p[: n // 2] = 0.1 + blob * rng.normal(size=(n // 2, 2))
    q = rng.normal(0.0, 1.0, n)
    return p[:, 0].copy(), p[:, 1].copy(), q, (rng.uniform(size=n) >= 0.1).astype(np.uint8)


def same(out, ref):
    fin = [np.isfinite(r) for r in ref]
    for o, r, f in zip(out, ref, fin):
        assert np.array_equal(f, np.isfinite(o)) and np.array_equal(np.isnan(r), np.isnan(o))
    assert rel_l2([o[f] for o, f in zip(out, fin)], [r[f] for r, f in zip(ref, fin)]) <= TOL


@pytest.mark.parametrize("cap", [1, 2, 7, 31, 33, 63, 65, 191, 192, 193, 400])
@pytest.mark.parametrize("blob", [0.0, 0.01])
def test_leaf_sizes(ctx, port, cap, blob):
    x, y, q, a = points(6001, cap, blob)
    kw = dict(max_src=cap, max_par=cap)
    same(ctx.field2d(x, y, q, a, default_params(**kw)), port.fmm2d_field(x, y, q, a, **kw))
    same([ctx.potential2d(x, y, q, a, default_params(**kw))], [port.fmm2d_potential(x, y, q, a, **kw)])


def test_coincident_particles(ctx, port):
    x, y, q, a = points(3000, 5)
    x[100:103] = x[700:703]
    y[100:103] = y[700:703]
    same(ctx.field2d(x, y, q, a), port.fmm2d_field(x, y, q, a))


@pytest.mark.parametrize("n,blob", [(5000, 0.0), (20011, 0.003)])
def test_graph_equals_eager(ctx, n, blob):
    import torch
    d = [torch.from_numpy(v).cuda() for v in points(n, n, blob)]
    out = [[torch.zeros_like(d[0]) for _ in range(2)] for _ in range(2)]
    ctx.set_stream(torch.cuda.current_stream().cuda_stream or None)
    try:
        for graph in (0, 1):
            ctx.field2d_device(*d, *out[graph], default_params(max_src=10, max_par=15, use_graph=graph))
        ctx.sync()
    finally:
        ctx.set_stream(None)
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
