"""A captured batch after an eager batch of larger solves on the same context,
for which the sub-contexts had to enlarge their arenas: the graph is made again
and gives the bits it gave before."""
import numpy as np
import pytest

from lsmps_vpm_v2_b200 import PREC_MIXED, Context, default_params, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [dict(p=10), dict(p=12, precision=PREC_MIXED)])
@pytest.mark.parametrize("solves", [1, 3, 9])
def test_graph_after_larger_batch(form, solves):
    import torch

    def upload(side, seed):
        ds = [workloads.multi_vortex_2d(side * side, seed + i) for i in range(solves)]
        offs = np.concatenate([[0], np.cumsum([d["x"].size for d in ds])]).astype(np.int64)
        dev = [torch.from_numpy(np.concatenate([d[k] for d in ds])).cuda() for k in ("x", "y", "q", "active")]
        return offs, dev, [torch.zeros_like(dev[0]) for _ in range(2)]

    ctx = Context(0)
    ctx.set_stream(torch.cuda.current_stream().cuda_stream or None)

    def call(data, **kw):
        offs, dev, out = data
        ctx.field2d_batched_device(offs, *[v.data_ptr() for v in dev], *[v.data_ptr() for v in out],
                                   default_params(**kw))
        ctx.sync()
        return [v.clone() for v in out]

    small, large = upload(60, 1), upload(200, 50)
    ref = call(small, use_graph=1, **form)
    grown = call(large, **form)
    again = call(small, use_graph=1, **form)
    last = call(large, **form)
    ctx.set_stream(None)
    ctx.close()
    assert all(torch.equal(a, b) for a, b in zip(ref, again))
    assert all(torch.equal(a, b) for a, b in zip(grown, last))
