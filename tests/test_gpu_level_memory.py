"""Memory of setups with level sweeps: the second layout (for blocks of columns) is optional memory.

Within an HBM budget that holds the setup without it, everything that fits must go on to work: the upload
itself, the first solve's Krylov basis, another setup of the context, a refactorization afterwards; results
against the oracle (1e-12 an apply), solves against a context without a budget.
"""
import numpy as np
import pytest
import scipy.sparse as sp

from conftest import small_setup
from oracle.oracle import OracleSetup, refactor_setup

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def case():
    """(workload, host setup, oracle, device bytes with both layouts, with the refactorization plan)"""
    from s2l_b200 import capi
    w, st = small_setup("poisson2d", nx=120, nsub=4)
    ctx = capi.Context(0)
    sizes = []
    for options in ({}, {"refactor": 1}):
        g = capi.GpuSetup(ctx, st, options=options)
        assert g.stat("level_layouts") == 2
        sizes.append(g.device_bytes())
        g.close()
    ctx.close()
    o = OracleSetup(st)
    yield w, st, o, *sizes
    o.close()


def check(g, st, o, widths=(1, 2, 4)):
    R = np.random.default_rng(3).standard_normal((max(widths), st.n))
    for k in widths:
        X = g.apply_block(R[:k]) if k > 1 else g.apply(R[0])[None]
        for j in range(k):
            z = o.apply(R[j])
            assert np.linalg.norm(X[j] - z) <= 1e-12 * np.linalg.norm(z), (k, j)


def test_the_upload_fits_without_the_second_layout(case):
    from s2l_b200 import capi
    _, st, o, full, _ = case
    ctx = capi.Context(0, hbm_budget=full - 4096)
    g = capi.GpuSetup(ctx, st)
    assert g.stat("level_layouts") == 1 and g.device_bytes() <= full - 4096
    check(g, st, o, widths=(1,))
    g.close()
    ctx.close()


def test_the_first_solve_takes_its_place(case):
    from s2l_b200 import capi
    w, st, o, full, _ = case
    probe = capi.Context(0)
    g = capi.GpuSetup(probe, st)
    x0, r0 = g.gmres(st.b, restart=w.restart, rtol=1e-8)
    assert g.stat("level_layouts") == 2  # no budget: kept
    g.close()
    probe.close()
    ctx = capi.Context(0, hbm_budget=full + 4096)
    g = capi.GpuSetup(ctx, st)
    assert g.stat("level_layouts") == 2
    x, r = g.gmres(st.b, restart=w.restart, rtol=1e-8)
    assert g.stat("level_layouts") == 1
    assert r["iterations"] == r0["iterations"] and np.array_equal(x, x0)  # one column: layout 0 in both
    check(g, st, o, widths=(1,))
    g.close()
    ctx.close()


def test_the_block_buffers_take_its_place(case):
    from s2l_b200 import capi
    _, st, o, full, _ = case
    probe = capi.Context(0)
    g = capi.GpuSetup(probe, st)
    check(g, st, o)
    need = g.device_bytes()
    g.close()
    probe.close()
    ctx = capi.Context(0, hbm_budget=need - 4096)
    g = capi.GpuSetup(ctx, st)
    assert g.stat("level_layouts") == 2
    check(g, st, o)
    assert g.stat("level_layouts") == 1
    g.close()
    ctx.close()


def test_another_setup_takes_its_place_and_refactorization_goes_on(case):
    from s2l_b200 import capi
    _, st, _, _, full = case
    _, st2 = small_setup("bubbles3d")
    probe = capi.Context(0)
    g2 = capi.GpuSetup(probe, st2)
    other = g2.device_bytes()
    g2.close()
    probe.close()
    ctx = capi.Context(0, hbm_budget=full + other - 4096)
    g = capi.GpuSetup(ctx, st, options={"refactor": 1})
    assert g.stat("level_layouts") == 2
    g2 = capi.GpuSetup(ctx, st2)
    assert g.stat("level_layouts") == 1
    d = 1.0 + 0.1 * np.random.default_rng(5).uniform(-1.0, 1.0, st.n)
    rows = np.repeat(np.arange(st.n), np.diff(st.A.indptr))
    A2 = sp.csr_matrix((st.A.data * d[rows] * d[st.A.indices], st.A.indices, st.A.indptr), shape=st.A.shape)
    g.refactor(A2.data)
    o = OracleSetup(refactor_setup(st, A2))
    check(g, st, o, widths=(1, 2))
    o.close()
    g2.close()
    g.close()
    ctx.close()


@pytest.mark.parametrize("requests", [6, 100])
def test_a_layout_in_use_is_waited_for(case, requests):
    """Requests run on the setup, one right after the other, while another setup is uploaded into the memory of
    its second layout."""
    from s2l_b200 import capi
    w, st, o, full, _ = case
    _, st2 = small_setup("bubbles3d")
    probe = capi.Context(0)
    g = capi.GpuSetup(probe, st)
    g.gmres(st.b, restart=w.restart, rtol=1e-8)
    solve = g.device_bytes() - full
    g2 = capi.GpuSetup(probe, st2)
    other = g2.device_bytes()
    g2.close()
    g.close()
    probe.close()
    ctx = capi.Context(0, hbm_budget=full + solve + other - 4096)
    ctx.serve_start(1, batching=0)
    g = capi.GpuSetup(ctx, st)
    tickets = [g.submit(st.b, restart=w.restart, rtol=1e-8) for _ in range(requests)]
    g2 = capi.GpuSetup(ctx, st2)
    xs = []
    for t in tickets:
        x, _, status = t.wait(120.0)
        assert status == 0, t.info()["error"]
        xs.append(x)
        t.free()
    assert all(np.array_equal(x, xs[0]) for x in xs)
    assert np.linalg.norm(st.b - st.A @ xs[0]) <= 1e-7 * np.linalg.norm(st.b)
    g2.close()
    check(g, st, o, widths=(1, 2))
    g.close()
    ctx.close()


def test_budgets_between_one_layout_and_two(case):
    """The second layout's own allocations fail at any of their steps; down to the setup with one layout."""
    from s2l_b200 import capi
    _, st, o, full, _ = case
    ctx = capi.Context(0, hbm_budget=full - 4096)
    g = capi.GpuSetup(ctx, st)
    one = g.device_bytes()
    assert g.stat("level_layouts") == 1
    g.close()
    ctx.close()
    for part in (0.9, 0.7, 0.5, 0.3, 0.1, 0.0):
        ctx = capi.Context(0, hbm_budget=one + int(part * (full - one)))
        g = capi.GpuSetup(ctx, st)
        assert g.stat("level_layouts") == 1 and g.device_bytes() == one
        check(g, st, o, widths=(1,))
        g.close()
        ctx.close()


def test_a_waiting_call_takes_no_further_workspaces(case):
    """A call whose Krylov basis misses the budget by a little waits for the second layout in use of another
    setup; while it waits it must not pile up workspaces (each fits, none helps)."""
    from s2l_b200 import capi
    w, st, _, full, _ = case
    w2, st2 = small_setup("bubbles3d")
    kw2 = {"restart": 50, "rtol": 1e-8}
    probe = capi.Context(0)
    g = capi.GpuSetup(probe, st)
    g.gmres(st.b, restart=w.restart, rtol=1e-8)
    solve = g.device_bytes() - full
    g2 = capi.GpuSetup(probe, st2)
    upload = g2.device_bytes()
    x0, _ = g2.gmres(st2.b, **kw2)
    alone = g2.device_bytes()
    g2.close()
    g.close()
    probe.close()
    ctx = capi.Context(0, hbm_budget=full + solve + alone - 4096)
    ctx.serve_start(1, batching=0)
    g = capi.GpuSetup(ctx, st)
    g2 = capi.GpuSetup(ctx, st2)
    assert g.stat("level_layouts") == 2
    tickets = [g.submit(st.b, restart=w.restart, rtol=1e-8) for _ in range(60)]
    x, _ = g2.gmres(st2.b, **kw2)
    assert np.array_equal(x, x0)
    assert g.stat("level_layouts") == 1
    assert g2.device_bytes() <= alone + (alone - upload)
    for t in tickets:
        assert t.wait(120.0)[2] == 0
        t.free()
    g2.close()
    g.close()
    ctx.close()
