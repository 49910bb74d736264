"""The FP64 form's transforms and nonlinear term held to their stated error (below
that of FP64 arithmetic) on every line length, and non-finite values in each of the
places that carry a line's exponent."""
import numpy as np
import pytest

from _helpers import configs, initial, relerr

pytestmark = pytest.mark.gpu

# lines of 8 to 1024 points on each axis
SHAPES = [(8, 16, 32), (64, 128, 8), (256, 8, 64), (32, 256, 16), (512, 16, 8), (16, 512, 128), (8, 8, 1024),
          (1024, 32, 8), (8, 1024, 16), (16, 64, 256), (8, 32, 512), (128, 8, 16)]
# Relative L2.  The last rounding to FP64 is 0.5e-16 of a field; a pass's fixed-point roundings
# are 2^-61 of a line's L1 norm each, below 2e-17 of the field at 1024 points.  FP64 arithmetic
# is at 1.8e-16 to 3.8e-16 on such fields, and at 3.0e-16 to 3.5e-16 in the nonlinear term, where
# the pointwise FP64 work (curl, k^2, product's factors, inverse curl) adds 1e-16 to the transforms'.
BOUND, BOUND_NLT = 2.0 ** -52, 3.0e-16


def field(kind, shape):
    rng = np.random.default_rng(11)
    x = rng.standard_normal(shape)
    if kind == "white":
        return x
    if kind == "mode over noise":
        i, j, k = np.indices(shape)
        return 1e-3 * x + np.cos(2 * np.pi * (2 * i / shape[0] + j / shape[1] + 3 * k / shape[2]) + 0.3)
    f = np.fft.rfftn(x)
    k = [np.fft.fftfreq(n, 1.0 / n) for n in shape[:2]] + [np.arange(shape[2] // 2 + 1)]
    k2 = k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + k[2][None, None, :] ** 2
    f *= np.where(k2 > 0, np.where(k2 > 0, k2, 1.0) ** (-11.0 / 12.0), 0.0)   # E(k) ~ k^-5/3
    return np.fft.irfftn(f, s=shape, axes=(0, 1, 2))


def wide_rfftn(x):
    """The forward transform (1/N) in extended precision."""
    f = np.fft.rfft(x.astype(np.longdouble), axis=2)
    f = np.fft.fft(np.fft.fft(f, axis=1), axis=0)
    assert f.dtype == np.clongdouble
    return f / x.size


def wide_irfftn(z, nx):
    f = z.astype(np.clongdouble)
    f = np.fft.ifft(np.fft.ifft(f, axis=0, norm="forward"), axis=1, norm="forward")
    return np.fft.irfft(f, n=nx, axis=2, norm="forward")


def l2(a, b):
    return float(np.sqrt(np.sum(np.abs(a - b) ** 2) / np.sum(np.abs(b) ** 2)))


@pytest.mark.parametrize("n", SHAPES)
@pytest.mark.parametrize("kind", ["white", "mode over noise", "k^-5/3"])
def test_transforms_below_fp64_error(lib, n, kind):
    import gturbo3d_gb300 as g
    gp, op = configs(n, precision="fp64", forcing="none")
    x = field(kind, (op.nz, op.ny, op.nx))
    spec = wide_rfftn(x)
    z = spec.astype(np.complex128)
    with g.Simulation(gp) as sim:
        assert l2(sim.fft_dir(x).astype(np.clongdouble), spec) < BOUND
        assert l2(sim.fft_inv(z).astype(np.longdouble), wide_irfftn(z, op.nx)) < BOUND


@pytest.mark.parametrize("n", [(8, 8, 8), (32, 64, 16), (128, 16, 8), (8, 256, 16), (16, 16, 512), (1024, 8, 8)])
def test_nonlinear_term_below_fp64_error(lib, n):
    import gturbo3d_gb300 as g
    from oracle.gturbo_oracle import defk, trunc_mask
    gp, op = configs(n, precision="fp64", forcing="none", omega=3.0)
    wk = defk(op)
    a = initial(n, seed=11)
    wide = [v.astype(np.clongdouble) for v in a]
    kx, ky, kz = (k.astype(np.longdouble) for k in (wk.fkx[None, None, :], wk.fky[None, :, None], wk.fkz[:, None, None]))
    k2 = kx * kx + ky * ky + kz * kz

    def curl(v):
        return [1j * (ky * v[2] - kz * v[1]), 1j * (kz * v[0] - kx * v[2]), 1j * (kx * v[1] - ky * v[0])]

    u = [wide_irfftn(v, op.nx) for v in curl(wide)]
    w = [wide_irfftn(k2 * v, op.nx) for v in wide]
    uw = [u[1] * w[2] - u[2] * w[1], u[2] * w[0] - u[0] * w[2], u[0] * w[1] - u[1] * w[0]]
    ref = [wide_rfftn(v) + 1j * np.longdouble(op.omega) * kz * b for v, b in zip(uw, wide)]
    ref = [v / np.where(k2 > 0, k2, 1) for v in curl(ref)]
    mask = trunc_mask(wk)
    with g.Simulation(gp) as sim:
        sim.set_state(a)             # the Coriolis source
        got = sim.nlt(a)
    num = sum(np.sum(np.abs(x - np.where(mask, 0, r)) ** 2) for x, r in zip(got, ref))
    den = sum(np.sum(np.abs(np.where(mask, 0, r)) ** 2) for r in ref)
    assert float(np.sqrt(num / den)) < BOUND_NLT


def kept(op):
    from oracle.gturbo_oracle import defk, trunc_mask
    return ~trunc_mask(defk(op))


@pytest.mark.parametrize("n", [(8, 8, 8), (32, 16, 64), (64, 128, 16)])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_nonfinite_mode_reaches_every_value(lib, n, bad):
    import gturbo3d_gb300 as g
    gp, op = configs(n, precision="fp64", forcing="none")
    a = initial(n, seed=2)
    a[1][1, 2, 1] = bad
    ok = kept(op)
    with g.Simulation(gp) as sim:
        assert all(np.isnan(v[ok]).all() for v in sim.nlt(a))
        assert np.isnan(sim.fft_inv(a[1])).all()
        sim.set_state(a)
        sim.step(1)
        assert all(np.isnan(v[ok]).all() for v in sim.get_state())
        sim.set_state(initial(n, seed=2))     # nothing of it stays behind
        sim.step(1)
        got = sim.get_state()
    with g.Simulation(gp) as sim:
        sim.set_state(initial(n, seed=2))
        sim.step(1)
        for x, y in zip(got, sim.get_state()):
            assert np.array_equal(x, y)


def test_nonfinite_member_leaves_the_batch_alone(lib):
    import gturbo3d_gb300 as g
    n = (32, 16, 16)
    gp, op = configs(n, precision="fp64", forcing="none")
    ok, out = kept(op), []
    for bad in (False, True):
        with g.api.Ensemble([gp] * 3) as ens:
            for m in range(3):
                b = initial(n, seed=m)
                if bad and m == 1:
                    b[0][1, 2, 1] = np.nan
                ens.set_state(m, b)
            ens.step(3, np.zeros(3, np.int32))
            out.append([ens.get_state(m) for m in range(3)])
    for m in (0, 2):
        for x, y in zip(out[0][m], out[1][m]):
            assert np.array_equal(x, y)
    assert all(np.isnan(v[ok]).all() for v in out[1][1])
