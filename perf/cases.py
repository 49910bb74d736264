"""The work that a user of this framework has it do, as measurable cases.

Every case goes through the public entry points of ``gturbo3d_gb300``, as a
program that steps a field, writes frames, reads diagnostics or differentiates
a run calls them:

* ``run``: a number of RK2 steps from the state in the handle, then the state
  (a checkpoint) or the velocity (a frame; main.f90:188-201);
* ``ensemble``: many small fields advanced together, then their states;
* ``diagnostics``: glob, spectra and flux of the current state;
* ``transforms``: one field to spectral space and back;
* ``start``: a velocity field into the handle (main.f90:91-106), steps, the state;
* ``gradient``: the checkpointed gradient of a run's final shell energy;
* ``linear``: a tangent-linear and an adjoint step.

The forms are the plain FP64 one and the mixed one (FP32 transforms); what the
mixed form computes is returned in 32 bits, the format its frames are written
in (write.f90 writes real*4).  Fields are random-phase solenoidal velocities
with a k^4 rise, a k^(-5/3) range and a viscous tail, at total energy 0.5, as
the framework's benchmark and tests normalise theirs.
"""
import math

import numpy as np
import torch

import gturbo3d_gb300 as g

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"
RTRUNC2 = 0.6666666666666666667 ** 2
INJECTION = 0.1          # forcing power of every forced case
SHELL = (1.999, 3.0)     # forced shells k1 < |k| <= k2 (params.dat)
NU, OMEGA, DT = 2e-3, 5.0, 1e-3


def listed():
    def run(name, n, precision, forcing, steps, out):
        return {"name": name, "kind": "run", "nx": n[0], "ny": n[1], "nz": n[2], "precision": precision,
                "forcing": forcing, "steps": steps, "out": out, "lz": 1.0}

    return [
        # a host program that drives single steps on a toy grid: the smallest call
        run("step_16_fp64", (16, 16, 16), "fp64", "3d3c", 1, "state"),
        # the CPU-sized validation run: 100 plain steps at 64^3, then a checkpoint
        run("steps_64_fp64", (64, 64, 64), "fp64", "3d3c", 100, "state"),
        # the same length of run in the mixed form on a thin-layer grid
        run("steps_128x128x32_mixed", (128, 128, 32), "mixed", "3d3c", 100, "state"),
        # the 2D2C-forced precision comparison at 256^3, both forms
        run("frame_256_mixed", (256, 256, 256), "mixed", "2d2c", 50, "velocity"),
        run("steps_256_fp64", (256, 256, 256), "fp64", "2d2c", 10, "state"),
        # production grids: steps between two frames at 512^3, both forms
        run("frame_512_mixed", (512, 512, 512), "mixed", "3d3c", 25, "velocity"),
        run("frame_512_fp64", (512, 512, 512), "fp64", "3d3c", 5, "velocity"),
        # parameter sweep over seeds and rotation rates: small members batched by grid
        {"name": "ensemble_64_128_mixed", "kind": "ensemble", "precision": "mixed", "classes": "12x64,4x128",
         "steps": 64, "forcing": "3d3c"},
        # the observables of a running simulation, with the flux (one more nonlinear term)
        {"name": "diagnostics_256_mixed", "kind": "diagnostics", "nx": 256, "ny": 256, "nz": 256,
         "precision": "mixed", "forcing": "3d3c", "lz": 1.0},
        # post-processing of single fields on an uneven grid
        {"name": "transforms_256x64x128_fp64", "kind": "transforms", "nx": 256, "ny": 64, "nz": 128,
         "precision": "fp64", "forcing": "none", "lz": 1.0},
        # optimal-perturbation / assimilation work: gradient of a run, and single linear steps
        {"name": "gradient_128_fp64", "kind": "gradient", "nx": 128, "ny": 128, "nz": 128, "precision": "fp64",
         "forcing": "3d3c", "steps": 10, "every": 5, "lz": 1.0},
        {"name": "linear_64x128x64_mixed", "kind": "linear", "nx": 64, "ny": 128, "nz": 64, "precision": "mixed",
         "forcing": "3d3c", "lz": 1.0},
    ]


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "ensemble", "diagnostics", "transforms", "start", "gradient",
                       "linear"])
    precision = rng.choice(["fp64", "mixed"])
    forcing = rng.choice(["3d3c", "3d3c", "2d2c", "none"])
    if kind == "ensemble":
        a, b = rng.choice([(16, 32), (32, 64), (64, 128)])
        return {"kind": kind, "precision": precision, "classes": f"{rng.randint(3, 12)}x{a},{rng.randint(1, 4)}x{b}",
                "steps": rng.randint(20, 80) if precision == "mixed" else rng.randint(5, 20), "forcing": "3d3c"}
    # total size from 8^3 to the largest of the kind, uniform in its logarithm; each axis a power of two
    top = {"run": 26, "diagnostics": 25, "transforms": 24, "start": 23, "gradient": 20, "linear": 22}[kind]
    lg = rng.uniform(9, top)
    while True:
        e = [round(lg / 3 + rng.uniform(-1.5, 1.5)) for _ in range(3)]
        if all(3 <= v <= 10 for v in e) and abs(sum(e) - lg) <= 1 and sum(e) <= top:
            if kind != "start" or e[1] + e[2] < 16:   # gt_set_state_physical takes fewer than 2^16 rows
                break
    points = 2 ** sum(e)
    case = {"kind": kind, "nx": 2 ** e[0], "ny": 2 ** e[1], "nz": 2 ** e[2], "precision": precision,
            "forcing": forcing, "lz": rng.choice([1.0, 1.0, 1.0, 2.0])}
    if kind in ("run", "start"):
        most = 30 if points <= 2 ** 21 else 6 if precision == "fp64" else 20
        case["steps"] = max(1, round(math.exp(rng.uniform(0, math.log(most)))))
    if kind == "run":
        case["out"] = rng.choice(["state", "velocity"]) if points < 2 ** 25 else "velocity"
    if kind == "gradient":
        case["steps"] = rng.randint(2, 8)
        case["every"] = rng.randint(1, case["steps"])
    return case


# --------------------------------------------------------------------------
# what a program has in hand
# --------------------------------------------------------------------------

def _axes(n, length, half=False):
    k = torch.arange(n // 2 + 1, dtype=torch.float64, device=DEVICE)
    if not half:
        k = torch.cat([k, torch.arange(-(n // 2) + 1, 0, dtype=torch.float64, device=DEVICE)])
    return k * (2.0 * math.pi / length)


def _grid(nx, ny, nz, lz):
    """kx, ky, kz (broadcastable), k^2 and the kept set of the 2/3 truncation."""
    kx = _axes(nx, 2.0 * math.pi, True)[None, None, :]
    ky = _axes(ny, 2.0 * math.pi)[None, :, None]
    kz = _axes(nz, 2.0 * math.pi * lz)[:, None, None]
    k2 = kx * kx + ky * ky + kz * kz
    frac = (kz * kz / kz.max() ** 2 + ky * ky / ky.max() ** 2) + kx * kx / kx.max() ** 2
    keep = frac <= RTRUNC2
    keep[0, 0, 0] = False
    return kx, ky, kz, k2, keep


def _cross_k(k, a, f=1.0):
    """i k x a, times f."""
    kx, ky, kz = k
    return [1j * f * (ky * a[2] - kz * a[1]), 1j * f * (kz * a[0] - kx * a[2]), 1j * f * (kx * a[1] - ky * a[0])]


def _weights(nh, edge, inner):
    w = torch.full((nh,), inner, dtype=torch.float64, device=DEVICE)
    w[0] = w[-1] = edge
    return w


def _potential(nx, ny, nz, lz, seed):
    """A vector potential b as complex128 tensors [nz, ny, nx/2+1]: real, solenoidal, inside the kept set."""
    gen = torch.Generator(device=DEVICE).manual_seed(int(seed))
    kx, ky, kz, k2, keep = _grid(nx, ny, nz, lz)
    kk = k2.sqrt()
    kd = 0.5 * (min(nx, ny, nz) / 3.0)   # viscous tail at half of the kept range
    amp = (kk / 3.0) ** 2 / (1.0 + (kk / 3.0) ** 2) ** (17.0 / 12.0 + 0.5) * torch.exp(-kk / kd)
    amp = torch.where(keep, amp / torch.where(k2 > 0, k2, torch.ones_like(k2)), torch.zeros_like(k2))
    b = []
    for _ in range(3):
        noise = torch.randn((nz, ny, nx), generator=gen, dtype=torch.float64, device=DEVICE)
        b.append(torch.fft.rfftn(noise, norm="forward") * amp)
    div = (kx * b[0] + ky * b[1] + kz * b[2]) / torch.where(k2 > 0, k2, torch.ones_like(k2))
    b = [b[0] - kx * div, b[1] - ky * div, b[2] - kz * div]
    u = _cross_k((kx, ky, kz), b)
    e = sum(((x.real ** 2 + x.imag ** 2) * _weights(nx // 2 + 1, 0.5, 1.0)).sum() for x in u)
    return [x * torch.sqrt(0.5 / e) for x in b]


def _numpy(fields):
    return [x.cpu().numpy() for x in fields]


def _params(nx, ny, nz, precision, forcing, lz=1.0, omega=OMEGA):
    p = g.make_params(nx, ny, nz, precision=precision, forcing=forcing, nu=NU, omega=omega, dt=DT,
                      xlz=2.0 * math.pi * lz)
    p.famp = g.forcing_amplitude(INJECTION, p)
    return p


def _members(case):
    """(grid, rotation rate) of each ensemble member."""
    out = []
    for part in case["classes"].split(","):
        count, n = (int(v) for v in part.split("x"))
        out += [n] * count
    return [(n, 1.0 + 19.0 * ((7 * i + 3) % 16) / 16.0) for i, n in enumerate(out)]


def _noise_seed(seed, member=0):
    """A forcing seed (a 31-bit state of the reference's generator)."""
    return (8299396 + 7919 * int(seed) + 104729 * member) % 0x7FFFFFFF


def prepare(case, seed):
    if case["kind"] == "ensemble":
        ms = _members(case)
        ens = g.Ensemble([_params(n, n, n, case["precision"], case["forcing"], omega=om) for n, om in ms])
        for i, (n, _) in enumerate(ms):
            ens.set_state(i, _numpy(_potential(n, n, n, 1.0, seed + 1000 * i)))
        return {"case": case, "ens": ens, "seeds": np.array([_noise_seed(seed, i) for i in range(len(ms))], np.int32)}
    dims = (case["nx"], case["ny"], case["nz"])
    sim = g.Simulation(_params(*dims, case["precision"], case["forcing"], case["lz"]))
    b = _potential(*dims, case["lz"], seed)
    s = {"case": case, "sim": sim, "seed": _noise_seed(seed)}
    if case["kind"] == "start":
        s["u"] = _numpy(_velocity(b, _grid(*dims, case["lz"]), dims))
    elif case["kind"] == "transforms":
        s["x"] = _numpy(_velocity(b, _grid(*dims, case["lz"]), dims)[:1])[0]
        s["z"] = _numpy(b[1:2])[0]
    else:
        sim.set_state(_numpy(b))
    if case["kind"] == "linear":
        s["db"] = _numpy(_potential(*dims, case["lz"], seed + 500))
        s["lam"] = _numpy(_potential(*dims, case["lz"], seed + 501))
    return s


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------

def _result(case, arrays):
    """The arrays in the precision that the form computes in."""
    if case["precision"] == "fp64":
        return list(arrays)
    out = []
    for x in arrays:
        t = torch.from_numpy(np.asarray(x, np.complex128 if np.iscomplexobj(x) else np.float64))
        out.append(t.to(torch.complex64 if t.is_complex() else torch.float32))
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "ensemble":
        ens = state["ens"]
        state["seeds"] = ens.step(case["steps"], state["seeds"])
        return [_result(case, ens.get_state(i)) for i in range(ens.n)]
    sim = state["sim"]
    if kind in ("run", "start"):
        if kind == "start":
            sim.set_state_physical(state["u"])
        state["seed"] = sim.step(case["steps"], state["seed"])
        return _result(case, sim.velocity() if case.get("out") == "velocity" else sim.get_state())
    if kind == "diagnostics":
        d = sim.diagnostics(flux=True)
        return _result(case, [d["energy"], d["enstrophy"], d["helicity"], d["spectrum"], d["spectrum2d"], d["flux"]])
    if kind == "transforms":
        return _result(case, [sim.fft_dir(state["x"]), sim.fft_inv(state["z"])])
    if kind == "gradient":
        j, grad = sim.gradient(case["steps"], state["seed"], case["every"], 4.0)
        return _result(case, [j] + grad)
    return _result(case, sim.tl_step(state["db"]) + sim.adj_step(state["lam"]))


def work(case):
    """State or field bytes in and out once per step (each step's state is its own result), and the flops of the
    transforms and products of the steps."""
    def one(nx, ny, nz, steps, value, transforms=18.0):
        n = nx * ny * nz
        kept = 0.155 * n   # modes inside the 2/3 ellipsoid of the half spectrum
        flops = steps * (transforms * 2.5 * n * math.log2(n) + 30.0 * n + 120.0 * kept)
        return 2.0 * 3.0 * kept * 2 * value * steps, flops

    value = 8 if case["precision"] == "fp64" else 4
    kind = case["kind"]
    if kind == "ensemble":
        parts = [one(n, n, n, case["steps"], value) for n, _ in _members(case)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    dims = (case["nx"], case["ny"], case["nz"])
    n = dims[0] * dims[1] * dims[2]
    if kind == "transforms":
        return {"bytes": 4.0 * n * value, "flops": 2 * 2.5 * n * math.log2(n)}
    if kind == "diagnostics":
        b, f = one(*dims, 1, value, 9.0)
        return {"bytes": b / 2, "flops": f}
    if kind == "linear":      # two linearised steps, each two nonlinear terms and their linearisations
        b, f = one(*dims, 2, value, 18.0 + 30.0)
        return {"bytes": b, "flops": f}
    if kind == "gradient":    # forward, recomputed forward, and an adjoint step each
        b, f = one(*dims, case["steps"], value, 18.0 + 18.0 + 60.0)
        return {"bytes": 3 * b, "flops": f}
    b, f = one(*dims, case["steps"], value)
    return {"bytes": b + (3.0 * n * value if case.get("out") == "velocity" else 0.0), "flops": f}


# --------------------------------------------------------------------------
# the same in plain 64-bit torch
# --------------------------------------------------------------------------

def _velocity(b, grid, dims):
    u = _cross_k(grid[:3], b)
    return [torch.fft.irfftn(x, s=(dims[2], dims[1], dims[0]), norm="forward") for x in u]


class _Flow:
    """The equations of one step (nlt.f90, rkstep.f90, forcing_*.f90)."""

    def __init__(self, dims, forcing, lz, omega):
        self.dims, self.forcing, self.omega = dims, forcing, omega
        self.kx, self.ky, self.kz, self.k2, self.keep = _grid(*dims, lz)
        self.k = (self.kx, self.ky, self.kz)
        self.ik2 = torch.where(self.k2 > 0, 1.0 / self.k2, torch.zeros_like(self.k2))
        self.emk = torch.exp(-0.5 * DT * NU * self.k2)
        self.origin = torch.ones_like(self.k2)
        self.origin[0, 0, 0] = 0.0
        self.modes = self._modes()
        self.famp = math.sqrt(INJECTION / len(self.modes)) if self.modes else 0.0

    def _modes(self):
        """Forced half-space modes (x, y, z) in the order in which the reference draws for them."""
        nx, ny, nz = self.dims
        hx, hy, hz = nx // 2, ny // 2, nz // 2
        if self.forcing == "3d3c":
            def plane(i):
                return ([(i, 0, k) for k in range(1, hz)] + [(i, j, k) for j in range(1, hy) for k in range(nz)]
                        + [(i, hy, k) for k in range(1, hz)])
            order = plane(0) + [(i, j, k) for i in range(1, min(hx, 5)) for j in range(ny) for k in range(nz)] + plane(hx)
        elif self.forcing == "2d2c":
            order = ([(0, j, 0) for j in range(1, hy)] + [(i, j, 0) for i in range(1, hx) for j in range(ny)]
                     + [(hx, j, 0) for j in range(1, hy)])
        else:
            return []
        k2, keep = self.k2.cpu().numpy(), self.keep.cpu().numpy()
        return [(i, j, k) for i, j, k in order
                if keep[k, j, i] and SHELL[0] ** 2 < k2[k, j, i] <= SHELL[1] ** 2]

    def force(self, b, seed):
        nx, ny, nz = self.dims
        kx, ky, kz = (v.flatten().cpu().tolist() for v in self.k)
        add = [torch.zeros_like(b[0]) for _ in range(3)]
        at, val = [], []

        def rann(s):
            s = (69069 * s + 1) & 0x7FFFFFFF
            return s, 2.0 * math.pi * float(np.float32(s / 0x7FFFFFFF))

        for i, j, k in self.modes:
            kk = math.sqrt(kx[i] ** 2 + ky[j] ** 2 + kz[k] ** 2)
            seed, t = rann(seed)
            f = math.sqrt(DT) * self.famp / kk * complex(math.cos(t), math.sin(t))
            if self.forcing == "2d2c":
                v = (0.0, 0.0, 1.0)
            else:
                seed, t = rann(seed)
                c, s = math.cos(t), math.sin(t)
                h = math.hypot(kx[i], ky[j])
                if i == 0 and j == 0:
                    v = (c, s, 0.0)
                else:
                    c1, s1, c2, s2 = kz[k] / kk, h / kk, kx[i] / h, ky[j] / h
                    v = (c * c2 * c1 - s * s2, c * s2 * c1 + s * c2, -c * s1)
            at.append((k, j, i))
            val.append([f * x for x in v])
            if i == 0 or (i == nx // 2):
                at.append(((nz - k) % nz, (ny - j) % ny, i))
                val.append([f.conjugate() * x for x in v])
        if at:
            idx = tuple(torch.tensor(col, device=DEVICE) for col in zip(*at))
            vals = torch.tensor(val, dtype=torch.complex128, device=DEVICE)
            for c in range(3):
                add[c].index_put_(idx, vals[:, c], accumulate=True)
        return [x + y for x, y in zip(b, add)], seed

    def nlt(self, a, bc):
        s = (self.dims[2], self.dims[1], self.dims[0])
        u = [torch.fft.irfftn(x, s=s, norm="forward") for x in _cross_k(self.k, a)]
        w = [torch.fft.irfftn(self.k2 * x, s=s, norm="forward") for x in a]
        c = [u[1] * w[2] - u[2] * w[1], u[2] * w[0] - u[0] * w[2], u[0] * w[1] - u[1] * w[0]]
        del u, w
        n = [torch.fft.rfftn(x, norm="forward") + 1j * self.omega * self.kz * y for x, y in zip(c, bc)]
        return [x * self.keep for x in _cross_k(self.k, n, self.ik2)]

    def smooth_step(self, b):
        """The step without its forcing."""
        n = self.nlt(b, b)
        c = [self.emk * (x + 0.5 * DT * y) * self.origin for x, y in zip(b, n)]
        n = self.nlt(c, b)
        return [self.emk * (self.emk * x + DT * y) * self.origin for x, y in zip(b, n)]

    def steps(self, b, n, seed):
        for _ in range(n):
            b, seed = self.force(self.smooth_step(b), seed)
        return b


def _diagnostics(flow, b):
    fac = _weights(flow.dims[0] // 2 + 1, 0.5, 1.0)
    u = _cross_k(flow.k, b)
    w = _cross_k(flow.k, u)
    sq = lambda x: x.real ** 2 + x.imag ** 2   # noqa: E731
    zero = torch.zeros(3, dtype=torch.float64, device=DEVICE)
    terms = []
    for f in (u, w):
        e = [fac * sq(x) for x in f]
        terms.append(torch.cat([torch.stack([x.sum() for x in e]),
                                torch.stack([(2.0 * NU * x * flow.k2).sum() for x in e]), zero]))
    hel = sum((fac * (x.real * y.real + x.imag * y.imag)).sum() for x, y in zip(u, w))
    nbin = flow.dims[0] // 2
    kk = flow.k2.sqrt()
    shell = torch.clamp(kk.long(), max=nbin).flatten()

    def binned(v, low):
        s = torch.zeros(nbin + 1, dtype=torch.float64, device=DEVICE)
        s.index_add_(0, shell, v.expand(flow.k2.shape).flatten())
        s[nbin - 1 if low else nbin:] = 0.0
        return s[:nbin]

    ek = binned(kk * kk * fac * sum(sq(x) for x in b), True)
    flat = kk * kk * fac * sq(b[2])
    flat = torch.cat([flat[:1], torch.zeros_like(flat[1:])])
    n1 = flow.nlt(b, b)
    t = _weights(flow.dims[0] // 2 + 1, 1.0, 2.0) * kk * kk * sum(
        x.real * y.real + x.imag * y.imag for x, y in zip(b, n1))
    per = binned(t, False)
    per[0] = 0.0
    flux = torch.flip(torch.cumsum(torch.flip(per, [0]), 0), [0])
    flux = torch.cat([flux[1:], torch.zeros(1, dtype=torch.float64, device=DEVICE)])
    return [terms[0], terms[1], hel, ek, binned(flat, True), flux]


def exact(case, seed):
    if case["kind"] == "ensemble":
        return [_numpy(_Flow((n, n, n), case["forcing"], 1.0, om).steps(
            _potential(n, n, n, 1.0, seed + 1000 * i), case["steps"], _noise_seed(seed, i)))
            for i, (n, om) in enumerate(_members(case))] if len(_members(case)) * case["steps"] <= 700 else None
    dims = (case["nx"], case["ny"], case["nz"])
    n = dims[0] * dims[1] * dims[2]
    if case.get("steps", 1) * n > 25 * 2 ** 27:
        return None
    flow = _Flow(dims, case["forcing"], case["lz"], OMEGA)
    b = _potential(*dims, case["lz"], seed)
    kind = case["kind"]
    if kind in ("run", "start"):
        if kind == "start":   # through physical space: only the transform of a real field remains
            u = [torch.fft.rfftn(x, norm="forward") for x in _velocity(b, flow.k, dims)]
            b = [x * flow.keep for x in _cross_k(flow.k, u, flow.ik2)]
        b = flow.steps(b, case["steps"], _noise_seed(seed))
        return _numpy(_velocity(b, flow.k, dims) if case.get("out") == "velocity" else b)
    if kind == "diagnostics":
        return _numpy(_diagnostics(flow, b))
    if kind == "transforms":
        x = _velocity(b, flow.k, dims)[0]
        return _numpy([torch.fft.rfftn(x, norm="forward"),
                       torch.fft.irfftn(b[1], s=(dims[2], dims[1], dims[0]), norm="forward")])
    # derivatives under <x, y> = sum w Re(conj(x) y), w = 1 on the planes kx = 0 and nx/2, 2 elsewhere
    w = _weights(dims[0] // 2 + 1, 1.0, 2.0)
    if kind == "gradient":
        b0 = [x.clone().requires_grad_(True) for x in b]
        u = _cross_k(flow.k, flow.steps(b0, case["steps"], _noise_seed(seed)))
        fac = _weights(dims[0] // 2 + 1, 0.5, 1.0) * (flow.k2 >= 16.0)
        j = sum((fac * (x.real ** 2 + x.imag ** 2)).sum() for x in u)
        grad = torch.autograd.grad(j, b0)
        return [float(j.detach())] + _numpy([x / w for x in grad])
    db, lam = (_potential(*dims, case["lz"], seed + s) for s in (500, 501))
    tl = torch.func.jvp(lambda *a: tuple(flow.smooth_step(list(a))), tuple(b), tuple(db))[1]
    b0 = [x.clone().requires_grad_(True) for x in b]
    out = flow.smooth_step(b0)
    pair = sum((w * (x.real * y.real + x.imag * y.imag)).sum() for x, y in zip(lam, out))
    adj = torch.autograd.grad(pair, b0)
    return _numpy(list(tl) + [x / w for x in adj])
