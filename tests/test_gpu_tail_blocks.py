"""Couplings in warp units and the dense tails' block products against the oracle's substitution.

Edges: tails of 1 row, one below, at and above the 16, 32 and 128 of the block products' tiles, rows of all
lengths in a unit (1 to 32 lanes a row), every block width (1 to 16 columns, FP64 and FP32), a
subdomain of more than 65536 rows (32-bit coupling columns), refactorized values.  Tolerances: the sums
differ from the oracle's by their order only, n eps cond-free growth of well-scaled Poisson factors,
1e-12 (FP32 factors 1e-5; 1e-11 for 68,000 rows).
"""
import numpy as np
import pytest
import scipy.sparse as sp

from conftest import small_setup
from oracle.oracle import OracleSetup, refactor_setup

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from s2l_b200 import capi
    c = capi.Context(0)
    yield c
    c.close()


def check(g, o, n, tol, widths=(1, 2, 4, 8, 16), seed=5):
    rng = np.random.default_rng(seed)
    for k in widths:
        R = rng.standard_normal((k, n))
        Z = g.apply_block(R)
        for j in range(k):
            z = o.apply(R[j])
            assert np.linalg.norm(Z[j] - z) <= tol * np.linalg.norm(z), (k, j)
    z = o.apply(R[0])
    assert np.linalg.norm(g.apply(R[0]) - z) <= tol * np.linalg.norm(z)


@pytest.mark.parametrize("precision", ["double", "single"])
@pytest.mark.parametrize("tail", [1, 15, 16, 17, 31, 33, 64, 127, 128, 129, 200])
def test_tail_blocks(ctx, tail, precision):
    from s2l_b200.capi import GpuSetup
    _, st = small_setup("bubbles3d", precision=precision)
    g = GpuSetup(ctx, st, options={"tail_rows": tail, "tail_min": 1})
    assert g.stat("tail_rows") > 0
    o = OracleSetup(st)
    check(g, o, st.n, 1e-5 if precision == "single" else 1e-12)
    for i, s in enumerate(st.subdomains):  # one subdomain's units alone
        b = np.random.default_rng(i).standard_normal(s.n_local)
        x = o.local_solve(i, b)
        assert np.linalg.norm(g.local_solve(i, b) - x) <= (1e-5 if precision == "single" else 1e-12) * np.linalg.norm(x)
    o.close()
    g.close()


@pytest.mark.parametrize("level", [0, 1])
@pytest.mark.parametrize("name", ["bubbles3d", "convdiff3d"])
def test_refactorized_couplings(ctx, name, level):
    from s2l_b200.capi import GpuSetup
    _, st = small_setup(name)
    g = GpuSetup(ctx, st, options={"tail_rows": 90, "refactor": 1, "level_sweeps": level})
    rng = np.random.default_rng(8)
    d = 1.0 + 0.1 * rng.uniform(-1.0, 1.0, st.n)
    rows = np.repeat(np.arange(st.n), np.diff(st.A.indptr))
    A2 = sp.csr_matrix((st.A.data * d[rows] * d[st.A.indices], st.A.indices, st.A.indptr), shape=st.A.shape)
    g.refactor(A2.data)
    o = OracleSetup(refactor_setup(st, A2))
    check(g, o, st.n, 1e-12, widths=(1, 4, 16))
    o.close()
    g.close()


def test_wide_columns(ctx):
    from s2l_b200.capi import GpuSetup
    _, st = small_setup("poisson2d", nx=370, nsub=2)
    assert max(s.n_local for s in st.subdomains) > 65536
    g = GpuSetup(ctx, st, options={"tail_rows": 300})
    o = OracleSetup(st)
    check(g, o, st.n, 1e-11, widths=(1, 4, 16))
    o.close()
    g.close()
