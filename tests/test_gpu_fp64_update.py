"""The FP64 form's update b + dt N as one rounding: without viscosity and rotation
(emk = 1) a step's result is the sum of the state and an increment about 1e-4 of it,
so nearly every component is the correctly rounded one."""
import numpy as np
import pytest

from _helpers import configs

pytestmark = pytest.mark.gpu


def flat_state(op, seed):
    """A solenoidal potential of a real field, all kept modes of like size."""
    from oracle.gturbo_oracle import defk, fft_dir, trunc_mask
    wk = defk(op)
    rng = np.random.default_rng(seed)
    mask = trunc_mask(wk)
    b = [np.where(mask, 0.0, fft_dir(rng.standard_normal((op.nz, op.ny, op.nx)), op)) for _ in range(3)]
    k = (wk.fkx[None, None, :], wk.fky[None, :, None], wk.fkz[:, None, None])
    div = sum(kc * bc for kc, bc in zip(k, b)) / np.where(wk.k2 > 0, wk.k2, 1.0)
    b = [bc - kc * div for kc, bc in zip(k, b)]
    for c in b:
        c[0, 0, 0] = 0.0
    return b


@pytest.mark.parametrize("n", [(8, 8, 8), (32, 16, 16), (16, 32, 64), (16, 8, 512)])
def test_update_is_rounded_once(lib, n):
    import gturbo3d_gb300 as g
    from oracle.gturbo_oracle import Oracle, Params
    phys = dict(nu=0.0, omega=0.0)
    op = Params(nx=n[0], ny=n[1], nz=n[2], forcing="none", dt2_mode="rk2", **phys)
    ora, b0 = Oracle(op), flat_state(op, 7)
    rms = lambda f: np.sqrt(sum(float(np.sum(np.abs(v) ** 2)) for v in f))
    dt = 1e-4 * rms(b0) / rms(ora.nlt(b0, b0))   # the increment is 1e-4 of the state
    gp, _ = configs(n, precision="fp64", forcing="none", dt=dt, **phys)
    c = [x + 0.5 * dt * y for x, y in zip(b0, ora.nlt(b0, b0))]
    inc = [dt * y for y in ora.nlt(c, b0)]
    with g.Simulation(gp) as sim:
        sim.set_state(b0)
        sim.step(1)
        got = sim.get_state()
    floor = 0.05 * rms(b0) / np.sqrt(sum(np.count_nonzero(x) for x in b0))
    differ = total = 0
    for x, d, y in zip(b0, inc, got):
        for part in (np.real, np.imag):
            want = (part(x).astype(np.longdouble) + part(d).astype(np.longdouble)).astype(np.float64)
            seen = np.abs(part(x)) > floor
            differ += np.count_nonzero(seen & (want != part(y)))
            total += np.count_nonzero(seen)
    # an increment off by 1e-15 of the typical one moves the sum by 1e-19 of the typical component:
    # 2 % of a unit in the last place of the smallest component counted here, 0.1 % of the
    # typical one's; a second rounding changes 13 to 22 % of the sums
    assert total > 100 and differ <= 0.03 * total, (differ, total)
