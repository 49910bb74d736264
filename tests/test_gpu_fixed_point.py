"""The FP64 form's block fixed-point passes at the edges of their range: every
line length, inputs whose lines hold one value, one mode, equal values or many
orders of magnitude, scales near the ends of FP64, zero and non-finite lines."""
import numpy as np
import pytest

from _helpers import configs, relerr

pytestmark = pytest.mark.gpu

# 8 and 16 points (no / one warp-level reduction), 32-64 (radix-4 and radix-8 tails),
# 128-1024 (several warps a line), on each axis
SHAPES = [(8, 16, 32), (64, 128, 8), (256, 8, 64), (32, 256, 16), (512, 16, 8), (16, 512, 128), (8, 8, 1024), (1024, 32, 8)]


def fields(kind, shape):
    rng = np.random.default_rng(5)
    x = rng.standard_normal(shape)
    if kind == "constant":
        return np.full(shape, 0.75)
    if kind == "impulse":
        x = np.zeros(shape)
        x[3, 2, 1] = -1.0
    elif kind == "decades":
        x *= 10.0 ** rng.uniform(-30, 0, shape)
    elif kind == "tiny":
        x *= 1e-290
    elif kind == "huge":
        x *= 1e290
    elif kind == "zero rows":
        x[::2] = 0.0
        x[:, ::3] = 0.0
    return x


@pytest.mark.parametrize("n", SHAPES)
@pytest.mark.parametrize("kind", ["white", "constant", "impulse", "decades", "tiny", "huge", "zero rows"])
def test_fixed_point_transforms(lib, n, kind):
    import gturbo3d_gb300 as g
    from oracle.gturbo_oracle import fft_dir, fft_inv
    gp, op = configs(n, precision="fp64", forcing="none")
    x = fields(kind, (op.nz, op.ny, op.nx))
    tol = 2e-15 * np.log2(x.size)   # the FP64 bound of the other transform tests
    top = np.max(np.abs(x))
    with g.Simulation(gp) as sim:
        X = sim.fft_dir(x)
        Xr = fft_dir(x, op)
        assert relerr([X / top], [Xr / top]) < tol
        y = sim.fft_inv(Xr)
        yr = fft_inv(Xr, op)
        assert relerr([y / top], [yr / top]) < tol


def test_fixed_point_zero_and_nonfinite(lib):
    import gturbo3d_gb300 as g
    gp, op = configs((32, 16, 64), precision="fp64", forcing="none")
    x = np.zeros((op.nz, op.ny, op.nx))
    with g.Simulation(gp) as sim:
        assert not np.any(sim.fft_dir(x))
        assert not np.any(sim.fft_inv(np.zeros(sim.shape, complex)))
        for bad in (np.nan, np.inf, -np.inf):
            x[5, 6, 7] = bad
            assert np.all(np.isnan(sim.fft_dir(x)))
        x[5, 6, 7] = 0.0
        assert not np.any(sim.fft_dir(x))   # nothing of it stays behind


@pytest.mark.parametrize("n", [(8, 8, 8), (16, 8, 32), (32, 64, 16), (128, 16, 8), (8, 256, 16), (16, 16, 512), (1024, 8, 8)])
@pytest.mark.parametrize("scale", [1.0, 1e-60, 1e60])
def test_fixed_point_nonlinear_term(lib, n, scale):
    """nlt is quadratic in its argument: N(s a) = s^2 N(a) without rotation, so
    the product's exponents are checked far from 1 as well."""
    import gturbo3d_gb300 as g
    from oracle.gturbo_oracle import Oracle
    from gturbo3d_gb300.synth import initial_potential
    gp, op = configs(n, precision="fp64", forcing="none", omega=0.0)
    a = initial_potential(op.nx, op.ny, op.nz, 11)
    ref = Oracle(op).nlt(a, a)
    with g.Simulation(gp) as sim:
        got = sim.nlt([scale * v for v in a])
    assert relerr([v / scale / scale for v in got], ref) < 1e-12
