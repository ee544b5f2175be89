"""Captured batches on one thread while another works on the legacy stream: a
capture of a stream that blocks with it would fail on both."""
import threading

import numpy as np
import pytest

from lsmps_vpm_v2_b200 import Context, default_params, workloads

pytestmark = pytest.mark.gpu


def test_capture_beside_the_legacy_stream():
    import torch
    ctx = Context(0)
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    d = workloads.multi_vortex_2d(900, 1)
    dev = [torch.from_numpy(np.concatenate([d[k]] * 9)).cuda() for k in ("x", "y", "q", "active")]
    out = [torch.zeros_like(dev[0]) for _ in range(2)]
    torch.cuda.synchronize()
    stop, failed = threading.Event(), []

    def legacy():
        host, there = torch.ones(1000), torch.zeros(1000, device="cuda")
        try:
            while not stop.is_set():
                there.copy_(host)
        except RuntimeError as e:
            failed.append(e)

    other = threading.Thread(target=legacy)
    other.start()
    try:
        for solves in list(range(1, 10)) * 2:   # every layout is captured anew
            offs = np.arange(solves + 1) * 900
            ctx.field2d_batched_device(offs, *[v.data_ptr() for v in dev], *[v.data_ptr() for v in out],
                                       default_params(use_graph=1))
            ctx.sync()
    finally:
        stop.set()
        other.join()
    assert not failed
    ctx.set_stream(None)
    ctx.close()
