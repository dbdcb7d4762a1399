"""Admission by memory under contention: many calls at once in a budget that holds the buffers of one.

Every call waits for the workspace that has them and none is refused, whatever the others try meanwhile
(a call that prepares a workspace in vain must neither be refused when the right one came free in that time
nor leave others waiting for it).
"""
import numpy as np
import pytest

from conftest import small_setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("trial", range(6))
def test_many_calls_in_memory_for_one(trial):
    from s2l_b200 import capi
    w, st = small_setup("bubbles3d")
    probe = capi.Context(0)
    g = capi.GpuSetup(probe, st)
    empty = g.device_bytes()
    bs = np.random.default_rng(31 + trial).uniform(-1.0, 1.0, (24, st.n))
    alone = [g.gmres(b, restart=w.restart, rtol=1e-8)[0] for b in bs]
    one = g.device_bytes()
    g.close()
    probe.close()
    ctx = capi.Context(0, hbm_budget=one + (one - empty) // 2)
    ctx.serve_start(8, batching=0)
    g = capi.GpuSetup(ctx, st)
    tickets = [g.submit(b, restart=w.restart, rtol=1e-8) for b in bs]
    for t, xa in zip(tickets, alone):
        x, _, status = t.wait(60.0)
        assert status == 0, t.info()["error"]
        assert np.array_equal(x, xa)
        t.free()
    g.close()
    ctx.close()
