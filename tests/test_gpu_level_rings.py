"""Level sweeps over the range of their shared memory: rings of 8 to 2 steps, 1 to 4 columns a CTA.

The depth of the cp.async rings and the columns a CTA holds follow from the slots of x and s, so large
sparse parts (no dense tail) reach each of them: FP64 from 4,500 to 19,600 rows a subdomain, FP32 from 10,000
to 40,900; above, s no longer fits and the setup falls back to dataflow sweeps.  The test computes what a
launch takes from the slots and asks for it.  Against the oracle's substitution, 1, 2, 4 and 16 columns:
forward errors of a backward stable solve, cond eps with cond <= 8e3 for these grids: 1e-11 (FP64), 5e-4
(FP32, worst case of both sides); and the same bits twice.
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


def ring(real_bytes, values):
    """Steps of a ring beside `values` of x and s: 16 warps, 128 values and 16-bit columns a step."""
    for depth in (8, 4, 3):
        if 16 * depth * 128 * (real_bytes + 2) + values * real_bytes <= 227 * 1024 - 64:
            return depth
    return 2


@pytest.mark.parametrize("precision,nx,kc,rings", [  # rings: of 1, 2 and 4 columns a CTA
    ("double", 95, 4, (8, 4, 2)),
    ("double", 106, 2, (8, 4)),
    ("double", 130, 2, (4, 3)),
    ("double", 137, 2, (4, 2)),
    ("double", 148, 1, (4,)),
    ("double", 186, 1, (3,)),
    ("double", 197, 1, (2,)),
    ("double", 203, 0, ()),
    ("single", 143, 4, (8, 8, 2)),
    ("single", 155, 2, (8, 8)),
    ("single", 203, 2, (8, 2)),
    ("single", 245, 1, (4,)),
    ("single", 277, 1, (3,)),
    ("single", 285, 1, (2,)),
    ("single", 298, 0, ()),
])
def test_rings_and_columns(ctx, precision, nx, kc, rings):
    from s2l_b200.capi import GpuSetup
    _, st = small_setup("poisson2d", nx=nx, nsub=2, precision=precision)
    g = GpuSetup(ctx, st, options={"tail_max": 0, "level_sweeps": 1})
    slots, rb = int(g.stat("level_slots")), 4 if precision == "single" else 8
    if kc == 0:
        assert g.stat("level_sweeps") == 0
    else:
        assert slots > max(s.n_local for s in st.subdomains)
        assert g.stat("kc_max") == kc
        assert tuple(ring(rb, slots * 2**q) for q in range(len(rings))) == rings
    o = OracleSetup(st)
    tol = 5e-4 if precision == "single" else 1e-11
    R = np.random.default_rng(nx).standard_normal((16, st.n))
    Z = [o.apply(r) for r in R[:4]]
    for k in (1, 2, 4, 16):
        X = g.apply_block(R[:k]) if k > 1 else g.apply(R[0])[None]
        for j in range(min(k, 4)):
            assert np.linalg.norm(X[j] - Z[j]) <= tol * np.linalg.norm(Z[j]), (k, j)
        assert np.array_equal(X, g.apply_block(R[:k]) if k > 1 else g.apply(R[0])[None]), k
    o.close()
    g.close()


@pytest.mark.parametrize("nx,nsub,layout,cs", [(40, 40, {"tail_rows": 5}, 2), (48, 90, {"tail_max": 0}, 1)])
def test_refactorized_on_small_clusters(ctx, nx, nsub, layout, cs):
    from s2l_b200.capi import GpuSetup
    _, st = small_setup("poisson2d", nx=nx, nsub=nsub)
    g = GpuSetup(ctx, st, options=dict(layout, level_sweeps=1, refactor=1))
    assert g.stat("level_sweeps") == cs
    rng = np.random.default_rng(nx)
    d = 1.0 + 0.1 * rng.uniform(-1.0, 1.0, st.n)
    rows = np.repeat(np.arange(st.n), np.diff(st.A.indptr))
    A2 = sp.csr_matrix((st.A.data * d[rows] * d[st.A.indices], st.A.indices, st.A.indptr), shape=st.A.shape)
    g.refactor(A2.data)
    o = OracleSetup(refactor_setup(st, A2))
    R = rng.standard_normal((4, st.n))
    X = g.apply_block(R)
    for j in range(4):
        z = o.apply(R[j])
        assert np.linalg.norm(X[j] - z) <= 1e-12 * np.linalg.norm(z)
        assert np.linalg.norm(g.apply(R[j]) - z) <= 1e-12 * np.linalg.norm(z)
    o.close()
    g.close()
