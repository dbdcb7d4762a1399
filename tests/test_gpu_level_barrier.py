"""Level sweeps whose warps reach the cluster barrier from ragged loops.

The lanes of a warp take different numbers of right-hand sides (rows without entries, and the warp's own)
before the first barrier of a sweep, and only some lanes copy the last part of a step before every other
one.  Odd sizes, so that neither count is a multiple of 32, on clusters of 8, 4 and 2 CTAs, one and more
columns: the oracle's substitution (1e-12; FP32 factors 1e-5), and the same bits every time.
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
    ("poisson2d", {"nx": 53, "nsub": 5}, {}),
    ("poisson2d", {"nx": 67, "nsub": 20}, {"tail_rows": 7}),
    ("poisson2d", {"nx": 71, "nsub": 37}, {"tail_max": 0}),
    ("convdiff3d", {"nx": 13, "nsub": 3, "precision": "single"}, {"tail_max": 0, "chain_block": 3}),
])
def test_ragged_right_hand_sides(ctx, name, kw, options):
    from s2l_b200.capi import GpuSetup
    _, st = small_setup(name, **kw)
    tol = 1e-5 if kw.get("precision") == "single" else 1e-12
    g = GpuSetup(ctx, st, options=dict(options, level_sweeps=1))
    assert g.stat("level_sweeps") >= 2  # a cluster
    o = OracleSetup(st)
    R = np.random.default_rng(11).standard_normal((4, st.n))
    Z = [o.apply(r) for r in R]
    first = {}
    for _ in range(10):
        for k in (1, 2, 4):
            X = g.apply_block(R[:k]) if k > 1 else g.apply(R[0])[None]
            for j in range(k):
                assert np.linalg.norm(X[j] - Z[j]) <= tol * np.linalg.norm(Z[j]), (k, j)
            assert np.array_equal(X, first.setdefault(k, X)), k
    o.close()
    g.close()
