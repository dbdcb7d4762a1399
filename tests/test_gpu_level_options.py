"""Layout options and statistics of setups with level sweeps."""
import pytest

from conftest import small_setup

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from s2l_b200 import capi
    c = capi.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("level", [-1, 0, 1])
def test_hop_us_zero_splits_by_bytes_alone(ctx, level):
    """hop_us 0 is a value like any other (the limit of small ones), not the default."""
    from s2l_b200.capi import GpuSetup
    _, st = small_setup("bubbles3d", nx=24, nsub=4)
    got = []
    for options in ({"hop_us": 0.0}, {"hop_us": 1e-12}, {}):
        g = GpuSetup(ctx, st, options=dict(options, level_sweeps=level))
        got.append((g.stat("tail_rows"), g.stat("dense_entries"), g.stat("level_sweeps")))
        g.close()
    assert got[0] == got[1]
    assert got[0][0] < got[2][0]  # levels that cost nothing need no tail


def test_sweep_group_statistic(ctx):
    """The widest lane group of the sweeps that run: 16 (dataflow) or 32 (level) unless set."""
    from s2l_b200.capi import GpuSetup
    _, st = small_setup("poisson2d", nx=61, nsub=3)
    for options, group in (({"level_sweeps": 1}, 32), ({"level_sweeps": 0}, 16), ({"level_sweeps": 1, "sweep_group": 8}, 8)):
        g = GpuSetup(ctx, st, options=options)
        assert g.stat("sweep_group") == group, options
        g.close()
