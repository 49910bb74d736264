"""Device memory that a handle keeps after tangent-linear, adjoint and gradient calls:
inside the memory budget, reused and grown without a trace in the results, and a
request that cannot be met refused."""
import ctypes as C

import numpy as np
import pytest

from _helpers import configs, initial

pytestmark = pytest.mark.gpu
N = (64, 64, 64)


def simulation(precision, forcing="3d3c"):
    import gturbo3d_gb300 as g
    gp, _ = configs(N, precision=precision, forcing=forcing, dt=1e-3)
    gp.famp = g.forcing_amplitude(0.1, gp) if forcing != "none" else 0.0
    sim = g.Simulation(gp)
    sim.set_state(initial(N, seed=4))
    return gp, sim


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_kept_workspace_stays_inside_the_budget(lib, precision):
    import gturbo3d_gb300 as g
    torch = pytest.importorskip("torch")
    free = lambda: torch.cuda.mem_get_info()[0]
    x = initial(N, seed=5)
    gp, sim = simulation(precision)
    with sim:
        want = sim.tl_step(x)      # loads the kernels, without a budget
    spare = 8 << 20                # less than the call's workspace (58 MB mixed, 102 MB FP64)
    g.set_memory_budget(g.memory_estimate(gp) + spare)
    try:
        gp, sim = simulation(precision)
        with sim:
            before = free()
            got = sim.tl_step(x)
            assert before - free() <= spare + (2 << 20)   # the allocator's granule
            again = sim.tl_step(x)
    finally:
        g.set_memory_budget(0)
    for a, b, c in zip(want, got, again):
        assert np.array_equal(a, b) and np.array_equal(a, c)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_grown_and_reused_workspace(lib, precision):
    x = initial(N, seed=5)
    calls = [lambda s: s.tl_step(x), lambda s: s.gradient(6, 77, 2, 4.0)[1], lambda s: s.adj_step(x),
             lambda s: s.tl_step(x)]
    _, sim = simulation(precision)
    with sim:
        got = [f(sim) for f in calls]
    for f, one in zip(calls, got):
        _, sim = simulation(precision)
        with sim:
            for a, b in zip(f(sim), one):
                assert np.array_equal(a, b)


def test_workspace_beyond_the_device_is_refused(lib):
    from gturbo3d_gb300 import _lib
    x = initial(N, seed=5)
    _, sim = simulation("fp64")
    with sim:
        want = sim.tl_step(x)
        J, out = C.c_double(), [np.empty(sim.shape, np.complex128) for _ in range(3)]
        rc = sim.lib.gt_gradient(sim.h, 200000, 3, 1, C.c_double(4.0), C.byref(J),
                                 *(a.ctypes.data_as(C.POINTER(C.c_double)) for a in out))   # 1.6 TB of checkpoints
        assert rc == _lib.GT_ENOMEM
        for a, b in zip(want, sim.tl_step(x)):
            assert np.array_equal(a, b)
