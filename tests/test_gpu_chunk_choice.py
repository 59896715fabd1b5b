"""The hydro stages' chunk depth is the library's choice until another one is set: what the autotuner reads
and puts back (after a failed candidate, or because the library's depth won) pins nothing."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture
def sim():
    from nebulaviewer_gb300 import build, ics
    from nebulaviewer_gb300.sim import Sim
    build.build(verbose=False)
    ic = ics.sheet(res=64, seed=4, nstars=64, device="cuda")
    s = Sim.from_state(ic["shape"], ic["dx"], ic["rho"], ic["stars"], ic["kinds"], ic["jets"], ic["jkinds"], ic["P"],
                       mom=ic["mom"], rays=(16, 32), fuv_grid=(8, 8, 16))
    s.step(1)
    yield s
    s.close()


def depths(s):
    """the depth in use with the stars' winds and without"""
    from nebulaviewer_gb300 import autotune as at
    out = []
    for wind in (0.5, 0.0):
        s.P["wind"] = wind
        s.step(1)
        out.append(at.get(s, "chunk_i"))
    s.P["wind"] = 0.5
    s.step(1)
    return out


def test_the_chosen_depth_is_not_pinned(sim, monkeypatch):
    from nebulaviewer_gb300 import autotune as at
    chosen = depths(sim)
    assert chosen[0] < chosen[1]                      # many winds: shallower chunks
    at.put(sim, "chunk_i", chosen[0])
    assert depths(sim) == chosen
    other = chosen[0] + 7
    at.put(sim, "chunk_i", other)
    assert depths(sim) == [other, other]
    at.put(sim, "chunk_i", chosen[0])
    assert depths(sim) == chosen
    # a failed candidate
    measure, calls = at._measure, []

    def failing(s, knob, steps):
        calls.append(knob)
        if len(calls) == 3:
            raise RuntimeError("injected failure")
        return measure(s, knob, steps)
    monkeypatch.setattr(at, "_measure", failing)
    with pytest.raises(RuntimeError, match="injected"):
        at.autotune(sim, knobs=["chunk_i"], use_cache=False)
    assert depths(sim) == chosen
    # the library's depth wins
    monkeypatch.setattr(at, "_measure", lambda s, knob, steps: 1.0 + abs(at.get(s, knob) - chosen[0]))
    assert at.autotune(sim, knobs=["chunk_i"], use_cache=False)["chunk_i"][0] == chosen[0]
    assert depths(sim) == chosen
    # another depth wins and stays
    monkeypatch.setattr(at, "_measure", lambda s, knob, steps: 1.0 + abs(at.get(s, knob) - 24))
    at.autotune(sim, knobs=["chunk_i"], use_cache=False)
    assert depths(sim) == [24, 24]


def test_the_chosen_depth_counts_jets(sim):
    """stars with jets alone make some tiles slower too; jets of no strength and stars without one do not"""
    from nebulaviewer_gb300 import autotune as at
    chosen = depths(sim)
    sim.P["wind"] = 0.0
    sim.step(1)
    assert at.get(sim, "chunk_i") == chosen[1]
    sim.P["jet"] = 300.0
    sim.step(1)
    assert at.get(sim, "chunk_i") == chosen[1]        # no star has a jet
    sim.jkinds = ["jet"] * 64
    sim.step(1)
    assert at.get(sim, "chunk_i") == chosen[0]
    sim.P["jet"] = 0.0
    sim.step(1)
    assert at.get(sim, "chunk_i") == chosen[1]
    sim.jkinds = ["proto"] * 64
    sim.P["jet_proto"] = 300.0
    sim.step(1)
    assert at.get(sim, "chunk_i") == chosen[0]
    sim.jkinds = ["none"] * 64
    sim.step(1)
    assert at.get(sim, "chunk_i") == chosen[1]
