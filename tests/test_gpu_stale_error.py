"""An error that a call has reported is not reported again by a later one: a batch
after a single call, a single call after a batch."""
import numpy as np
import pytest

from lsmps_vpm_v2_b200 import Context, VpmError, default_params, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("use_graph", [0, 1])
@pytest.mark.parametrize("first", ["single", "batch"])
def test_reported_error_is_not_reported_again(first, use_graph):
    import torch
    ctx = Context(0)
    d = workloads.multi_vortex_2d(1600, 1)
    x, y, q, a = (d[k] for k in ("x", "y", "q", "active"))
    bad = x.copy()
    bad[3] = np.inf
    prm = default_params(use_graph=use_graph)
    with pytest.raises(VpmError, match="non-finite"):
        if first == "single":
            ctx.field2d(bad, y, q, a, prm)
        else:
            ctx.field2d_batched([(x, y, q, a), (bad, y, q, a)], prm)
    dev = [torch.from_numpy(v).cuda() for v in (x, y, q, a)]
    out = [torch.zeros_like(dev[0]) for _ in range(2)]
    torch.cuda.synchronize()
    if first == "single":
        ctx.field2d_batched_device(np.array([0, x.size]), *[v.data_ptr() for v in dev], *[v.data_ptr() for v in out], prm)
    else:
        ctx.field2d_device(*dev, *out, prm)
    ctx.sync()
    ref = ctx.field2d(x, y, q, a)
    assert all(np.array_equal(o.cpu().numpy(), r) for o, r in zip(out, ref))
    ctx.close()
