"""That small grids' steps are in fact replayed as a graph (the replay counter), and that
a graph whose forcing buffer is replaced by a larger one is made anew."""
import numpy as np
import pytest

from _helpers import configs, initial

pytestmark = pytest.mark.gpu


def make(n, precision, forcing="3d3c"):
    import gturbo3d_gb300 as g
    gp, _ = configs(n, precision=precision, forcing=forcing, dt=1e-3)
    gp.famp = g.forcing_amplitude(0.1, gp) if forcing != "none" else 0.0
    sim = g.Simulation(gp)
    sim.set_state(initial(n))
    return sim


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("forcing", ["3d3c", "2d2c", "none"])
def test_steps_are_replayed(lib, precision, forcing):
    seed = 8299396 if forcing != "none" else None
    with make((16, 32, 16), precision, forcing) as sim:
        assert sim.get_tuning("graph_replays") == 0
        seed = sim.step(1, seed)
        assert sim.get_tuning("graph_replays") == 0      # the first step runs directly
        seed = sim.step(32, seed)
        assert sim.get_tuning("graph_replays") == 32
        seed = sim.step(1, seed)
        assert sim.get_tuning("graph_replays") == 33
        sim.set_tuning("x_fused", 1)                     # other passes: direct until theirs is made
        seed = sim.step(32, seed)
        assert sim.get_tuning("graph_replays") == 33 + 31
        sim.profile(True)
        seed = sim.step(8, seed)
        assert sim.get_tuning("graph_replays") == 33 + 31
    with make((256, 256, 128), precision, forcing) as sim:   # beyond 2^22 points
        sim.step(20, seed)
        assert sim.get_tuning("graph_replays") == 0
    with pytest.raises(Exception):
        with make((8, 8, 8), precision, forcing) as sim:
            sim.set_tuning("graph_replays", 0)               # a counter, not a knob


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_forcing_buffer_grows_under_a_live_graph(lib, precision):
    out = []
    for direct in (False, True):
        with make((32, 32, 32), precision) as sim:
            sim.profile(direct)
            seed = 8299396
            for _ in range(20):                # a graph over the smallest buffer, one step's entries
                seed = sim.step(1, seed)
            alive = sim.get_tuning("graph_replays")
            seed = sim.step(32, seed)          # 32 steps' entries do not fit it
            seed = sim.step(3, seed)
            assert direct or (alive > 0 and sim.get_tuning("graph_replays") > alive)
            out.append((seed, sim.get_state()))
    assert out[0][0] == out[1][0]
    for a, b in zip(out[0][1], out[1][1]):
        assert np.array_equal(a, b)
