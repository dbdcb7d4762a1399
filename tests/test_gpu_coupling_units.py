"""The couplings between the sparse part and the dense tail with one, two and more columns.

One and two columns load a unit's first step ahead of its rows; units have 0 steps (tail rows without sparse
entries: a sparse part of one row), 1, 2 and odd numbers of them, and lanes get 2, 4 or 16 entries by the
number of entries of the whole setup.  Against the oracle's substitution (1e-12; FP32 factors 1e-5: the sums
differ by their order only).
"""
import numpy as np
import pytest

from conftest import small_setup
from oracle.oracle import OracleSetup

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from s2l_b200 import capi
    c = capi.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("name,kw,options", [
    ("bubbles3d", {}, {"tail_rows": 1 << 20}),                              # a sparse part of one row
    ("bubbles3d", {}, {"tail_rows": 300}),
    ("convdiff3d", {"precision": "single"}, {"tail_rows": 1 << 20}),
    ("convdiff3d", {}, {"tail_rows": 150, "tail_min": 1}),
    ("bubbles3d", {"nx": 30, "nsub": 8, "overlap": 1}, {"tail_rows": 780, "level_sweeps": 0}),  # four entries a lane
    ("bubbles3d", {"nx": 30, "nsub": 8, "overlap": 1}, {"tail_rows": 780, "level_sweeps": 1}),
])
def test_first_steps(ctx, name, kw, options):
    from s2l_b200.capi import GpuSetup
    _, st = small_setup(name, **kw)
    tol = 1e-5 if kw.get("precision") == "single" else 1e-12
    g = GpuSetup(ctx, st, options=options)
    assert g.stat("coupling_nnz") > (2 * 0.75 * 128 * 32 * 148 if "nx" in kw else 0)
    o = OracleSetup(st)
    R = np.random.default_rng(17).standard_normal((4, st.n))
    Z = [o.apply(r) for r in R]
    for k in (1, 2, 4):
        X = g.apply_block(R[:k]) if k > 1 else g.apply(R[0])[None]
        for j in range(k):
            assert np.linalg.norm(X[j] - Z[j]) <= tol * np.linalg.norm(Z[j]), (k, j)
    for i in range(0, len(st.subdomains), 3):
        b = np.random.default_rng(i).standard_normal(st.subdomains[i].n_local)
        x = o.local_solve(i, b)
        assert np.linalg.norm(g.local_solve(i, b) - x) <= tol * np.linalg.norm(x)
    o.close()
    g.close()
