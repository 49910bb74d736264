"""Steps replayed as one graph (small grids) against the same steps launched
directly (profiling keeps the direct launches): equal bit for bit, also when
the passes, the forcing or the call pattern change between the replays."""
import numpy as np
import pytest

from _helpers import configs, initial

pytestmark = pytest.mark.gpu


def drive(sim, direct, forced):
    seed = 8299396 if forced else None
    if direct:
        sim.profile(True)
    seed = sim.step(70, seed)            # 32-step chunks: direct first step, then replays
    for _ in range(3):
        seed = sim.step(1, seed)
    sim.set_tuning("x_fused", 1)         # other passes: a new graph
    seed = sim.step(40, seed)
    sim.set_tuning("x_fused", 2)
    ix, iy, iz = np.array([1, 1, 2]), np.array([2, 2, 1]), np.array([0, 0, 1])
    sim.step_coeffs(ix, iy, iz, np.full((3, 6), 1e-4))   # a repeated mode: added in order
    sim.step_coeffs(ix[1:], iy[1:], iz[1:], np.full((2, 6), 1e-4))
    sim.set_pruning(False)
    seed = sim.step(33, seed)
    sim.set_pruning(True)
    seed = sim.step(2, seed)
    if direct:
        sim.profile(False)
    return seed, sim.get_state(), sim.launch_count()


@pytest.mark.parametrize("n", [(8, 8, 8), (32, 16, 64), (128, 64, 16)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("forcing", ["3d3c", "2d2c", "none"])
def test_graph_steps_equal_direct_steps(lib, n, precision, forcing):
    import gturbo3d_gb300 as g
    gp, _ = configs(n, precision=precision, forcing=forcing, dt=1e-3)
    gp.famp = g.forcing_amplitude(0.1, gp)
    out = []
    for direct in (False, True):
        with g.Simulation(gp) as sim:
            sim.set_state(initial(n))
            out.append(drive(sim, direct, forcing != "none"))
    assert out[0][0] == out[1][0]
    assert out[0][2] == out[1][2]
    for a, b in zip(out[0][1], out[1][1]):
        assert np.array_equal(a, b)
