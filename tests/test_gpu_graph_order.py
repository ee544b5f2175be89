"""A captured evaluation replayed after the context has evaluated at another
order or with the other binomials: the translation tables of the arena are then
those of that call, and the replay needs its own again."""
import numpy as np
import pytest

from lsmps_vpm_v2_b200 import BINOM_EXACT, PREC_MIXED, Context, default_params

pytestmark = pytest.mark.gpu


def blob(n, seed):
    """Leaves on many levels: lists 2, 3 and 4 all in use."""
    rng = np.random.default_rng(seed)
    p = rng.uniform(-1.0, 1.0, (n, 2))
    p[: n // 2] = 0.2 + 0.02 * rng.normal(size=(n // 2, 2))
    return p[:, 0].copy(), p[:, 1].copy(), rng.normal(size=n), np.ones(n, np.uint8)


@pytest.mark.parametrize("graph", [1, 2])
@pytest.mark.parametrize("first,other", [
    (dict(p=12), dict(p=8)), (dict(p=8), dict(p=16)), (dict(p=17), dict(p=17, binom=BINOM_EXACT)),
    (dict(p=12, precision=PREC_MIXED), dict(p=7)), (dict(p=18, precision=PREC_MIXED, binom=BINOM_EXACT), dict(p=9))])
def test_replay_after_another_order(first, other, graph):
    d = blob(8000, 3)
    fresh = Context(0)
    ref = fresh.field2d(*d, default_params(use_graph=graph, **first))
    fresh.close()
    ctx = Context(0)
    for _ in range(2):
        assert np.array_equal(ref, ctx.field2d(*d, default_params(use_graph=graph, **first)))
        ctx.field2d(*d, default_params(**other))
    ctx.close()


@pytest.mark.parametrize("form", [dict(p=12), dict(p=12, precision=PREC_MIXED)])
def test_batch_replay_after_another_order(form):
    import torch
    solves = [blob(n, n) for n in (3000, 4000, 2000)]
    offs = np.concatenate([[0], np.cumsum([s[0].size for s in solves])]).astype(np.int64)
    dev = [torch.from_numpy(np.concatenate([s[k] for s in solves])).cuda() for k in range(4)]
    out = [torch.zeros_like(dev[0]) for _ in range(2)]
    ctx = Context(0)
    ctx.set_stream(torch.cuda.current_stream().cuda_stream or None)

    def call(**kw):
        ctx.field2d_batched_device(offs, *[v.data_ptr() for v in dev], *[v.data_ptr() for v in out],
                                   default_params(**kw))
        ctx.sync()
        return [v.clone() for v in out]

    ref = call(use_graph=1, **form)
    call(p=7)
    again = call(use_graph=1, **form)
    ctx.set_stream(None)
    ctx.close()
    assert all(torch.equal(a, b) for a, b in zip(ref, again))
