"""A captured batch after an eager one, which runs on fewer streams: the graph is
replayed on its own streams, and the errors of all its solves are seen."""
import time

import numpy as np
import pytest

from lsmps_vpm_v2_b200 import Context, VpmError, default_params, workloads

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ctx():
    c = Context(0)
    yield c
    c.close()


def solves(n_solves, side):
    ds = [workloads.multi_vortex_2d(side * side, i) for i in range(n_solves)]
    return [(d["x"].copy(), d["y"], d["q"], d["active"]) for d in ds]


def test_replay_after_eager_batch(ctx):
    graph, eager = default_params(use_graph=1), default_params()
    batch = solves(48, 60)
    ref = ctx.field2d_batched(batch, graph)
    streams = ctx.batch_streams()

    def timed(before):
        times = []
        for _ in range(4):
            if before:
                ctx.field2d_batched(batch, eager)
            start = time.perf_counter()
            out = ctx.field2d_batched(batch, graph)
            times.append(time.perf_counter() - start)
        return min(times), out

    plain, _ = timed(False)
    after, again = timed(True)
    # capturing and timing the choices anew takes ten times as long as a replay with its copies
    assert after < 3 * plain
    assert ctx.batch_streams() == streams
    assert all(np.array_equal(a, b) for r, s in zip(ref, again) for a, b in zip(r, s))
    for k in range(len(batch)):   # largest first, each on a stream of its own as long as there are some
        ctx.field2d_batched(batch, eager)
        x = batch[k][0]
        kept, x[7] = x[7], np.nan
        with pytest.raises(VpmError, match="non-finite"):
            ctx.field2d_batched(batch, graph)
        x[7] = kept
    ctx.field2d_batched(batch, graph)
