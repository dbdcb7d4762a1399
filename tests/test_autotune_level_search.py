"""The autotuner's search on setups with level sweeps, on the CPU with a stand-in for the device setup:
values around their own defaults (hop_us 2, groups of 32 lanes), the dataflow sweeps among the
candidates, no value that gives the default's layout again; a caller's own list is searched as it is."""
import pytest

from s2l_b200 import autotune


class FakeSetup:
    n = 4

    def __init__(self, ctx, st, options=None):
        self.options = dict(options or {})
        FakeSetup.built.append(dict(self.options))

    def close(self):
        pass

    def set_option(self, name, value):
        self.options[name] = value


def fake_measure(level):
    def measure(g, k, reps, rng):
        o = g.options
        on = level if o.get("level_sweeps", -1) < 0 else o["level_sweeps"]
        t = 10.0 - {1.0: 1.0}.get(o.get("hop_us"), 0.0) - (0.0 if on == level else 0.5)
        return {"local_solve_ms": t, "spmv_ms": 0.5, "level_sweeps": 8 if on else 0}
    return measure


@pytest.mark.parametrize("level", [0, 1])
def test_the_search_suits_the_sweeps(monkeypatch, level):
    monkeypatch.setattr(autotune.capi, "GpuSetup", FakeSetup)
    monkeypatch.setattr(autotune, "measure", fake_measure(level))
    FakeSetup.built = []
    _, rep = autotune.tune(None, None)
    tried = {q: [b[q] for b in FakeSetup.built if q in b] for q in ("hop_us", "chain_block", "sweep_group")}
    if level:
        assert 4.0 in tried["hop_us"] and 1.0 in tried["hop_us"] and not {0.1, 0.25, 0.5, 2.0} & set(tried["hop_us"])
        assert 16 not in tried["chain_block"] and tried["sweep_group"][0] == 16
    else:
        assert 0.1 in tried["hop_us"] and 16 in tried["chain_block"] and 32 in tried["sweep_group"]
    assert rep["chosen"]["level_sweeps"] == 1 - level  # the other kind is tried
    assert rep["chosen"]["hop_us"] == 1.0


def test_a_list_given_is_searched_as_it_is(monkeypatch):
    monkeypatch.setattr(autotune.capi, "GpuSetup", FakeSetup)
    monkeypatch.setattr(autotune, "measure", fake_measure(1))
    search = (("hop_us", (0.25, 0.5)),)
    FakeSetup.built = []
    autotune.tune(None, None, search=search)
    assert FakeSetup.built == [{}, {"hop_us": 0.5}]
    FakeSetup.built = []
    autotune.tune(None, None, search=search, level_search=(("hop_us", (2.0, 3.0)),))
    assert FakeSetup.built == [{}, {"hop_us": 3.0}]
