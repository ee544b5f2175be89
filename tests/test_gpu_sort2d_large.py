"""Particle sets on both sides of the one-launch sort's limit of 148 x 16,384
particles and well above it, where the multi-kernel sort takes over: every
particle in one leaf, and the field against the FP64 direct sum."""
import numpy as np
import pytest

from lsmps_vpm_v2_b200 import default_params, workloads
from lsmps_vpm_v2_b200._lib import lib
from lsmps_vpm_v2_b200.workloads import rel_l2, sample_targets

pytestmark = pytest.mark.gpu
LIMIT = 148 * 16384
TOL_DIRECT = 1e-4   # p = 12, the caps of the reference


@pytest.fixture(scope="module")
def vortices():
    return workloads.multi_vortex_2d(1733 * 1733, 2)


@pytest.mark.parametrize("n", [LIMIT, LIMIT + 1, 1733 * 1733])
def test_large_set(ctx, vortices, n):
    import torch
    d = [np.ascontiguousarray(vortices[k][:n]) for k in ("x", "y", "q", "active")]
    dev = [torch.from_numpy(v).cuda() for v in d]
    out = [torch.zeros_like(dev[0]) for _ in range(2)]
    tg = torch.from_numpy(np.asarray(sample_targets(n, 512), np.int64)).cuda()
    ref = [torch.zeros(tg.numel(), dtype=torch.float64, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    for use_graph in (0, 1):
        ctx.field2d_device(*dev, *out, default_params(p=12, use_graph=use_graph))
        ctx.sync()
        ctx._check(lib().vpm_direct2d_field_device(ctx._h, *[v.data_ptr() for v in dev], n, tg.data_ptr(), tg.numel(),
                                                   *[v.data_ptr() for v in ref]))
        ctx.sync()
        assert rel_l2([o[tg].cpu().numpy() for o in out], [r.cpu().numpy() for r in ref]) <= TOL_DIRECT
    assert np.array_equal(np.sort(ctx.dump_tree2d()["leaf_pids"]), np.arange(n))
