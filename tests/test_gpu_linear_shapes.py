"""The linear steps' batched passes on the shapes that select a kernel of their own:
z lines of 256 and 512 points (TMA-loaded in the mixed form), long x and y lines, an
uneven box, and the kept-column z passes of the plain inverse transforms."""
import numpy as np
import pytest

from _helpers import configs, initial, relerr
from test_gpu_adjoint import inner, real_field_spectrum

pytestmark = pytest.mark.gpu

SHAPES = [((16, 8, 256), 1.0), ((8, 16, 512), 1.0), ((64, 32, 16), 2.0), ((256, 8, 32), 1.0), ((32, 128, 64), 0.5)]


def setup(n, lz, precision):
    import gturbo3d_gb300 as g
    gp, op = configs(n, precision=precision, forcing="none", dt=1e-3, omega=3.0, xlz=2 * np.pi * lz)
    b0 = initial((n[0], n[1], n[2]), seed=3)
    if lz != 1.0:   # solenoidal in the box at hand
        from oracle.gturbo_oracle import defk, trunc, trunc_mask
        wk = defk(op)
        k = (wk.fkx[None, None, :], wk.fky[None, :, None], wk.fkz[:, None, None])
        div = sum(kc * bc for kc, bc in zip(k, b0)) / np.where(wk.k2 > 0, wk.k2, 1.0)
        b0 = [trunc(bc - kc * div, trunc_mask(wk)) for kc, bc in zip(k, b0)]
    sim = g.Simulation(gp)
    sim.set_state(b0)
    return sim, op, b0


@pytest.mark.parametrize("n,lz", SHAPES)
def test_fp64_linear_steps(lib, n, lz):
    sim, op, b0 = setup(n, lz, "fp64")
    with sim:
        x = real_field_spectrum(sim.shape, 1, op)
        y = real_field_spectrum(sim.shape, 2, op)
        tl = sim.tl_step(x)
        lhs, rhs = inner(y, tl), inner(sim.adj_step(y), x)
        assert abs(lhs - rhs) <= 1e-12 * np.sqrt(inner(y, y) * inner(tl, tl))
        # central differences: the step is quartic in the state, so the error is h^2 of it
        s = np.sqrt(inner(b0, b0) / inner(x, x))
        fd = []
        for sgn in (1, -1):
            sim.set_state([b + sgn * 1e-5 * s * v for b, v in zip(b0, x)])
            sim.step(1)
            fd.append(sim.get_state())
        fd = [(p - m) / (2e-5 * s) for p, m in zip(*fd)]
        assert relerr(tl, fd) < 1e-8


@pytest.mark.parametrize("n,lz", SHAPES)
def test_mixed_linear_steps_against_fp64(lib, n, lz):
    out = {}
    for precision in ("fp64", "mixed"):
        sim, op, _ = setup(n, lz, precision)
        with sim:
            x = real_field_spectrum(sim.shape, 1, op)
            out[precision] = [sim.tl_step(x), sim.adj_step(x), sim.velocity()]
            J, grad = sim.gradient(3, 0, 2, 2.0)
            out[precision] += [grad]
    # an FP32 rounding per transform stage (log2 of the points), for the step's transform pairs
    tol = 8 * np.finfo(np.float32).eps * np.log2(np.prod(n))
    for a, b in zip(out["mixed"], out["fp64"]):
        assert relerr(a, b) < tol
