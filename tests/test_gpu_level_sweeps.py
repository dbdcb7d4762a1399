"""Level-synchronous sparse sweeps (a thread-block cluster per subdomain, barriers instead of ready flags).

The setup option "level_sweeps" forces them (1) or the dataflow sweeps (0); by default a setup takes
whichever has the shorter chain of hand-overs.  Forced on, every layout must give the oracle's
substitution: the local solves and the two-level apply (1e-12 with FP64 factors, 1e-5 with FP32),
blocks of 1 to 16 columns column by column, and the refactorized setup.  Sizes: few and many
subdomains (clusters of 8 CTAs down to 1), subdomains of a few rows, tails of any size, blocks of 16 to
64 rows.
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


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


CASES = [
    ("poisson2d", {"nx": 40, "nsub": 4}, {}),
    ("poisson2d", {"nx": 9, "nsub": 2}, {"tail_max": 0}),                     # a few rows
    ("poisson2d", {"nx": 61, "nsub": 3}, {"tail_max": 0}),                    # long chains, no tail
    ("poisson2d", {"nx": 40, "nsub": 40}, {"tail_rows": 5}),                  # clusters of 2
    ("poisson2d", {"nx": 48, "nsub": 90}, {"tail_max": 0}),                   # one CTA per subdomain
    ("bubbles3d", {}, {}),
    ("bubbles3d", {}, {"tail_max": 0, "chain_block": 2}),
    ("bubbles3d", {"precision": "single"}, {"tail_max": 0}),
    ("bubbles3d", {"pou": "multiplicity", "one_level": "asm"}, {"tail_rows": 64, "chain_block": 16}),
    ("convdiff3d", {}, {"tail_max": 0, "sweep_group": 8}),
    ("convdiff3d", {"precision": "single"}, {"tail_rows": 40, "chain_block": 4}),
]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_level_sweeps_match_the_oracle(ctx, case):
    from s2l_b200.capi import GpuSetup
    name, kw, layout = CASES[case]
    _, st = small_setup(name, **kw)
    single = kw.get("precision") == "single"
    tol = 1e-5 if single else 1e-12
    g = GpuSetup(ctx, st, options=dict(layout, level_sweeps=1))
    assert g.stat("level_sweeps") >= 1
    o = OracleSetup(st)
    rng = np.random.default_rng(40 + case)
    for i, s in enumerate(st.subdomains):
        b = rng.standard_normal(s.n_local)
        assert rel(g.local_solve(i, b), o.local_solve(i, b)) <= tol
    r = rng.standard_normal(st.n)
    z = g.apply(r)
    assert rel(z, o.apply(r)) <= tol
    assert np.array_equal(g.apply(r), z)  # no order depends on timing
    for k in (1, 2, 3, 4, 7, 16):
        R = rng.standard_normal((k, st.n))
        Z = g.apply_block(R)
        for j in range(k):
            assert rel(Z[j], o.apply(R[j])) <= tol
    o.close()
    g.close()


@pytest.mark.parametrize("case", [0, 2, 5, 6, 7, 9, 10])
def test_level_sweeps_refactorized(ctx, case):
    from s2l_b200.capi import GpuSetup
    name, kw, layout = CASES[case]
    _, st = small_setup(name, **kw)
    tol = 1e-5 if kw.get("precision") == "single" else 1e-12
    g = GpuSetup(ctx, st, options=dict(layout, level_sweeps=1, refactor=1))
    rng = np.random.default_rng(70 + case)
    d = 1.0 + 0.1 * rng.uniform(-1.0, 1.0, st.n)
    rows = np.repeat(np.arange(st.n), np.diff(st.A.indptr))
    A2 = sp.csr_matrix((st.A.data * d[rows] * d[st.A.indices], st.A.indices, st.A.indptr), shape=st.A.shape)
    g.refactor(A2.data)
    o2 = OracleSetup(refactor_setup(st, A2))
    R = rng.standard_normal((4, st.n))
    Z = g.apply_block(R)
    for j in range(4):
        assert rel(g.apply(R[j]), o2.apply(R[j])) <= tol
        assert rel(Z[j], o2.apply(R[j])) <= tol
    o2.close()
    g.close()


def test_a_large_sparse_part_falls_back(ctx):
    """x of 8-byte values of a subdomain of more than 29,000 rows does not fit a CTA: dataflow sweeps."""
    from s2l_b200.capi import GpuSetup
    _, st = small_setup("poisson2d", nx=250, nsub=2)
    g = GpuSetup(ctx, st, options={"level_sweeps": 1, "tail_max": 0})
    assert g.stat("level_sweeps") == 0
    r = np.random.default_rng(3).standard_normal(st.n)
    o = OracleSetup(st)
    assert rel(g.apply(r), o.apply(r)) <= 1e-12
    o.close()
    g.close()


def test_the_default_takes_the_shorter_chain(ctx):
    """Deep factors get level sweeps, shallow ones and setups without chain blocks dataflow sweeps."""
    from s2l_b200 import capi
    _, st = small_setup("poisson2d", nx=120, nsub=4)
    for options, on in (({}, True), ({"chain_block": 1}, False), ({"level_sweeps": 0}, False)):
        g = capi.GpuSetup(ctx, st, options=options)
        assert (g.stat("level_sweeps") > 0) == on, options
        g.close()
    with pytest.raises(capi.S2LError) as e:
        capi.GpuSetup(ctx, st, options={"level_sweeps": 2})
    assert e.value.code == 1
