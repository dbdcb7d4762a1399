"""A setup whose fastest layouts do not fit the HBM budget is uploaded with the smallest ones.

Level sweeps may take more memory than dataflow sweeps (longer dense tails), and small setups pad their
couplings for speed.  Budgets that hold the dataflow sweeps and the narrowest couplings must do, with the
refactorization plan too; below those the upload still fails with S2L_ERR_OOM.  Results against the oracle:
1e-12 (FP32 factors 1e-5).
"""
import numpy as np
import pytest
import scipy.sparse as sp

from conftest import small_setup
from oracle.oracle import OracleSetup, refactor_setup

pytestmark = pytest.mark.gpu


def size_of(st, options):
    from s2l_b200 import capi
    ctx = capi.Context(0)
    g = capi.GpuSetup(ctx, st, options=options)
    out = g.device_bytes(), g.stat("level_sweeps")
    g.close()
    ctx.close()
    return out


@pytest.mark.parametrize("refactor", [0, 1])
def test_dataflow_sweeps_where_level_sweeps_do_not_fit(refactor):
    from s2l_b200 import capi
    _, st = small_setup("poisson2d", nx=150, nsub=6, precision="single")
    base = {"refactor": refactor}
    full, level = size_of(st, dict(base, tail_max=4096))
    flow, none = size_of(st, dict(base, level_sweeps=0))
    assert level > 0 and none == 0
    if refactor:  # (the plan keeps the dataflow split: level sweeps are the smaller ones)
        flow = min(flow, full - 4096)
    assert flow < full
    ctx = capi.Context(0, hbm_budget=flow + 4096)
    g = capi.GpuSetup(ctx, st, options=base)
    assert g.device_bytes() <= flow + 4096
    if not refactor:
        assert g.stat("level_sweeps") == 0
    o = OracleSetup(st)
    r = np.random.default_rng(2).standard_normal(st.n)
    if refactor:
        d = 1.0 + 0.1 * np.random.default_rng(5).uniform(-1.0, 1.0, st.n)
        rows = np.repeat(np.arange(st.n), np.diff(st.A.indptr))
        A2 = sp.csr_matrix((st.A.data * d[rows] * d[st.A.indices], st.A.indices, st.A.indptr), shape=st.A.shape)
        g.refactor(A2.data)
        o.close()
        o = OracleSetup(refactor_setup(st, A2))
    z = o.apply(r)
    assert np.linalg.norm(g.apply(r) - z) <= 1e-5 * np.linalg.norm(z)
    o.close()
    g.close()
    ctx.close()


def test_narrow_couplings_where_padded_ones_do_not_fit():
    from s2l_b200 import capi
    _, st = small_setup("bubbles3d", nx=24, nsub=8, overlap=1)
    full, level = size_of(st, {})
    assert level == 0
    ctx = capi.Context(0, hbm_budget=int(full * 0.987))  # what its layouts took with rows of 12-byte entries
    g = capi.GpuSetup(ctx, st)
    o = OracleSetup(st)
    r = np.random.default_rng(2).standard_normal(st.n)
    z = o.apply(r)
    assert np.linalg.norm(g.apply(r) - z) <= 1e-12 * np.linalg.norm(z)
    o.close()
    g.close()
    ctx.close()
    tight = capi.Context(0, hbm_budget=int(full * 0.8))
    with pytest.raises(capi.S2LError) as e:
        capi.GpuSetup(tight, st)
    assert e.value.code == 2 and "budget" in str(e.value)
    tight.close()
