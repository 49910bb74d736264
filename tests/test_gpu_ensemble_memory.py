"""A class of FP64 members keeps its line exponents in the members' staging fields: it takes
no device memory beyond theirs, and transfers between its steps leave the steps alone."""
import numpy as np
import pytest

from _helpers import configs, initial

pytestmark = pytest.mark.gpu


def test_class_takes_its_members_memory(lib):
    import gturbo3d_gb300 as g
    torch = pytest.importorskip("torch")
    n, m = (8, 256, 256), 20      # exponents of 1.7 MB a member; the class's own tables take 5 MB in all
    gp, _ = configs(n, precision="fp64", forcing="none")
    free = lambda: torch.cuda.mem_get_info()[0]
    with g.api.Ensemble([gp] * 2) as ens:
        ens.step(1, np.zeros(2, np.int32))         # loads the kernels
    before = free()
    sims = [g.Simulation(gp) for _ in range(m)]
    alone = before - free()
    for s in sims:
        s.close()
    before = free()
    with g.api.Ensemble([gp] * m):
        together = before - free()
    assert together <= alone + (16 << 20), (alone, together)   # 35 MB more with a block of exponents


@pytest.mark.parametrize("n", [(8, 8, 8), (8, 8, 64), (32, 16, 64)])
def test_transfers_between_steps(lib, n):
    import gturbo3d_gb300 as g
    gp, _ = configs(n, precision="fp64", forcing="none", dt=1e-3)
    out = []
    for rounds in (1, 4):
        with g.api.Ensemble([gp] * 3) as ens:
            for m in range(3):
                ens.set_state(m, initial(n, seed=m))
            for _ in range(rounds):
                ens.step(4 // rounds, np.zeros(3, np.int32))
                if rounds > 1:     # every member's staging field is overwritten both ways
                    for m in range(3):
                        ens.set_state(m, ens.get_state(m))
            out.append([ens.get_state(m) for m in range(3)])
    for a, b in zip(*out):
        for x, y in zip(a, b):
            assert np.array_equal(x, y)
