"""Whole solves on setups with level sweeps: GMRES, BiCGStab, blocks, served requests, concurrent callers.

The small workloads have few levels and would run dataflow sweeps, so level sweeps are forced.  Solves
reach their tolerance in FP64 with the iterations of the dataflow sweeps (one more or less: the local solves
differ by their rounding), served and concurrent ones are bitwise those alone.
"""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from conftest import small_setup

pytestmark = pytest.mark.gpu

CASES = [("bubbles3d", {}), ("convdiff3d", {}), ("bubbles3d", {"precision": "single"}),
         ("poisson2d", {"nx": 61, "nsub": 3})]


@pytest.fixture(scope="module", params=range(len(CASES)))
def case(request):
    from s2l_b200 import capi
    name, kw = CASES[request.param]
    w, st = small_setup(name, **kw)
    ctx = capi.Context(0)
    g = capi.GpuSetup(ctx, st, options={"level_sweeps": 1})
    flow = capi.GpuSetup(ctx, st, options={"level_sweeps": 0})
    assert g.stat("level_sweeps") > 0 and flow.stat("level_sweeps") == 0
    flexible = kw.get("precision") == "single"
    yield ctx, w, st, g, flow, {"restart": w.restart, "rtol": 1e-8, "flexible": flexible, "strict": flexible}
    flow.close()
    g.close()
    ctx.close()


def rhs(st, k, seed):
    return np.random.default_rng(seed).uniform(-1.0, 1.0, (k, st.n))


def solved(st, b, x):
    return np.linalg.norm(b - st.A @ x) <= 1.1e-8 * np.linalg.norm(b)


def test_gmres_and_bicgstab(case):
    _, _, st, g, flow, kw = case
    for b in rhs(st, 2, 1):
        x, r = g.gmres(b, **kw)
        _, rf = flow.gmres(b, **kw)
        assert solved(st, b, x) and abs(r["iterations"] - rf["iterations"]) <= 1
        if not kw["flexible"]:
            x, r = g.bicgstab(b, rtol=1e-8)
            assert r["converged"] and np.linalg.norm(b - st.A @ x) <= 1e-7 * np.linalg.norm(b)


@pytest.mark.parametrize("k", [2, 5, 16])
def test_gmres_block(case, k):
    _, _, st, g, _, kw = case
    B = rhs(st, k, 2)
    X, info = g.gmres_block(B, **kw)
    for j in range(k):
        assert solved(st, B[j], X[j])
        assert abs(info[j]["iterations"] - g.gmres(B[j], **kw)[1]["iterations"]) <= 1


def test_served_requests(case):
    from s2l_b200 import capi
    ctx, _, st, g, _, kw = case
    ctx.serve_start(3)
    B = rhs(st, 7, 3)

    def serve(bs):
        out = []
        for t in [g.submit(b, **kw) for b in bs]:
            x, _, status = t.wait(120.0)
            assert status == capi.S2L_OK, t.info()["error"]
            out.append(x)
            t.free()
        return out

    alone = [serve([b])[0] for b in B]
    for b, x, xa in zip(B, serve(B), alone):
        assert solved(st, b, x) and np.array_equal(x, xa)


def test_concurrent_callers(case):
    _, _, st, g, _, kw = case
    B = rhs(st, 8, 4)
    alone = [(g.apply(b), g.gmres(b, **kw)[0], g.apply_block(B[:4])) for b in B]
    with ThreadPoolExecutor(4) as pool:
        for _ in range(2):
            got = list(pool.map(lambda b: (g.apply(b), g.gmres(b, **kw)[0], g.apply_block(B[:4])), B))
            for a, q in zip(alone, got):
                assert all(np.array_equal(u, v) for u, v in zip(a, q))


def test_time_loop():
    """A sequence with refactorizations: levels and iterations (one more or less) of the dataflow sweeps."""
    from s2l_b200 import capi
    from s2l_b200 import workloads as W
    from s2l_b200.time_loop import TimeLoopConfig, levels, run_time_loop
    w = W.bubbles3d(12, 8, nbubbles=6, overlap=1)
    w.opts.nev = 8
    ctx = capi.Context(0)
    cfg = TimeLoopConfig(steps=3, correctors=2, reuse="refactor")
    on, off = (run_time_loop(w, cfg, ctx=ctx, workers=1, options={"level_sweeps": v}) for v in (1, 0))
    assert levels(on) == levels(off) == "201010"
    for a, b in zip(on, off):
        assert a.converged and a.true_rel_residual <= 1.1 * w.rtol and abs(a.iterations - b.iterations) <= 1
    ctx.close()
