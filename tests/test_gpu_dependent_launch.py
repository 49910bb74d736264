"""Passes set up while their predecessor ends (up to 4096 blocks, single fields)
against the plain launches of a batch of two members: the smallest grid, grids
whose passes fall on both sides of the limit, and one beyond it."""
import numpy as np
import pytest

from _helpers import configs, initial

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(8, 8, 8), (16, 128, 64), (64, 64, 64), (128, 128, 128), (64, 256, 128)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_single_steps_equal_batched_steps(lib, n, precision):
    import gturbo3d_gb300 as g
    gp, _ = configs(n, precision=precision, forcing="3d3c", dt=1e-3)
    gp.famp = g.forcing_amplitude(0.1, gp)
    b0, steps = initial(n), 6
    with g.Simulation(gp) as sim:
        sim.set_state(b0)
        seed = sim.step(steps, 8299396)
        single = sim.get_state()
    with g.api.Ensemble([gp, gp]) as ens:
        for m in range(2):
            ens.set_state(m, b0)
        seeds = ens.step(steps, np.full(2, 8299396, dtype=np.int32))
        batched = [ens.get_state(m) for m in range(2)]
    assert list(seeds) == [seed, seed]
    # the same sums: at most one rounding per transform stage and step apart
    eps = np.finfo(np.float64 if precision == "fp64" else np.float32).eps
    tol = eps * steps * np.log2(np.prod(n))
    for other in batched:
        for x, y in zip(single, other):
            assert np.linalg.norm(x - y) <= tol * np.linalg.norm(y)
