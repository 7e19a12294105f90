"""Measured workloads: what a program using this package has it do, through its public entry points.

Four families:

* ``run2d``: one ``FDTD(design=grid, ...).run()`` of the 2D solver on material arrays the
  program already holds, from zero fields to the final fields and the monitors' results;
* ``run3d``: the same for the 3D solver;
* ``adjoint``: one objective value and its gradient by ``FDTDObjective`` (forward and
  adjoint FDTD) for a batch of topology-optimisation designs;
* ``fno``: the surrogate network's predictions, or its loss gradient, for a batch of densities.

``exact`` restates each computation in float64 with plain torch operations.
"""
import math

import numpy as np
import torch

import beamz_b200 as bz

UM = 1e-6
DX = 0.02 * UM
C0 = 299792458.0
EPS_0 = 8.85e-12  # the constants of the solver, not the CODATA ones
MU_0 = 1.256e-6
WAVELENGTHS = (1.50 * UM, 1.525 * UM, 1.55 * UM, 1.575 * UM, 1.60 * UM)
SI, SIO2 = 12.25, 2.085


def listed():
    return [
        # a first try-out: the smallest domain that still holds a guide, a source and an
        # absorber, a few hundred steps, one recorded line
        dict(name="run2d_tryout", kind="run2d", nx=61, ny=47, steps=150, pml=8, source="point", monitors="record",
             precision="fp32", power=False),
        # the standard pulsed dipole: 400 x 400 cells, 2000 steps, four recorded edge lines
        dict(name="run2d_dipole", kind="run2d", nx=400, ny=400, steps=2000, pml=20, source="point",
             monitors="record", precision="fp32", power=False),
        # a device simulation: 2000 x 1000 cells, a mode line source with a real profile, three
        # frequency-domain flux lines, thousands of steps
        dict(name="run2d_device", kind="run2d", nx=2000, ny=1000, steps=6000, pml=30, source="line",
             monitors="dft", precision="fp32", power=False),
        # a mode source with a complex profile, as the numerical mode solver gives one: the
        # fields carry two components
        dict(name="run2d_complex", kind="run2d", nx=1000, ny=501, steps=2000, pml=24, source="complex_line",
             monitors="dft", precision="fp32", power=False),
        # a double-precision check run on an odd-sized grid
        dict(name="run2d_fp64", kind="run2d", nx=601, ny=397, steps=1000, pml=20, source="line", monitors="dft",
             precision="fp64", power=False),
        # a run that accumulates the power map over the whole domain
        dict(name="run2d_power", kind="run2d", nx=500, ny=300, steps=1000, pml=20, source="line",
             monitors="record", precision="fp32", power=True),
        # a small 3D domain (a coupler tip), odd number of layers
        dict(name="run3d_small", kind="run3d", nx=100, ny=50, nz=29, steps=300, pml=8, precision="fp32"),
        # a device-sized 3D domain: 27 million cells
        dict(name="run3d_device", kind="run3d", nx=600, ny=300, nz=150, steps=500, pml=16, precision="fp32"),
        # one step of a single-design topology optimisation
        dict(name="adjoint_one", kind="adjoint", nx=300, ny=200, steps=800, pml=16, region=60, designs=1),
        # one step of a batched topology optimisation: 64 designs
        dict(name="adjoint_batch", kind="adjoint", nx=600, ny=400, steps=1500, pml=20, region=120, designs=64),
        # the search ranks 256 candidate densities by their predicted transmission
        dict(name="fno_predict", kind="fno", n=120, batch=256, modes=16, layers=4, train=False),
        # one training batch: predictions and the loss gradient of every parameter
        dict(name="fno_gradient", kind="fno", n=120, batch=64, modes=16, layers=4, train=True),
    ]


def draw(rng):
    """One more case of the same ranges. Sizes are log-uniform; odd ones are as likely as even ones."""

    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["run2d", "run2d", "run2d", "run3d", "run3d", "adjoint", "adjoint", "fno", "fno"])
    if kind == "run2d":
        precision = "fp64" if rng.random() < 0.15 else "fp32"
        nx, ny = size(60, 2000), size(48, 1000)
        steps = min(size(150, 6000), 10 ** 10 // (nx * ny))
        return dict(kind=kind, nx=nx, ny=ny, steps=min(steps, 2000) if precision == "fp64" else steps,
                    pml=rng.randint(8, min(30, min(nx, ny) // 5)),
                    source=rng.choice(["point", "line", "complex_line"]), monitors=rng.choice(["record", "dft"]),
                    precision=precision, power=rng.random() < 0.15)
    if kind == "run3d":
        nx, ny, nz = size(64, 600), size(48, 300), size(24, 150)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=max(20, min(size(100, 600), 10 ** 10 // (nx * ny * nz))),
                    pml=rng.randint(6, min(16, min(nx, ny, nz) // 4)),
                    precision="fp64" if rng.random() < 0.1 else "fp32")
    if kind == "adjoint":
        nx, ny, b = size(160, 600), size(120, 400), size(1, 64)
        region = rng.randint(30, min(nx, ny) // 3)
        steps = size(8 * (region + 40), 1600)  # at least the time a pulse takes across the region
        return dict(kind=kind, nx=nx, ny=ny, steps=steps, pml=rng.randint(10, 20), region=region, designs=b)
    train = rng.random() < 0.5
    return dict(kind=kind, n=rng.choice([40, 60, 64, 90, 96, 100, 120]), batch=size(1, 64 if train else 256),
                modes=rng.choice([8, 12, 16]), layers=rng.choice([2, 3, 4]), train=train)


# ---- inputs -----------------------------------------------------------------------------
def _dt(dims):
    return 0.99 * DX / (C0 * math.sqrt(dims))


def _pulse(steps, dt, rng):
    """A Gaussian-pulsed carrier near 1.55 um whose envelope fits the run."""
    t = np.arange(steps) * dt
    f0 = C0 / (1.55 * UM) * (1.0 + 0.01 * rng.standard_normal())
    width = min(10e-15, steps * dt / 12)
    return np.exp(-((t - 3 * width) / width) ** 2 / 2) * np.cos(2 * np.pi * f0 * t + rng.uniform(0, 2 * np.pi))


def _continuous(steps, dt, rng):
    """A carrier near 1.55 um, switched on over ten periods (fewer in a short run) and left on."""
    t = np.arange(steps) * dt
    f0 = C0 / (1.55 * UM) * (1.0 + 0.01 * rng.standard_normal())
    ramp = min(10 / f0, steps * dt / 4)
    return np.clip(t / ramp, 0, 1) ** 2 * np.cos(2 * np.pi * f0 * t + rng.uniform(0, 2 * np.pi))


def _loss_profile(n, pml):
    """Order-3 conductivity grading along an axis of n cells: 0 inside, 1 at the outer faces."""
    i = np.arange(n)
    d = np.maximum(np.maximum(pml - i, i - (n - 1 - pml)), 0) / pml
    return d ** 3


def _materials(shape, pml, rng):
    """eps and sigma: a cladding with a guide along x and a few blocks, conductivity-graded faces."""
    eps = np.full(shape, SIO2)
    ny, nx = shape[-2:]
    core = max(3, min(25, ny // 6))
    y0 = ny // 2 - core // 2
    layers = (slice(shape[0] // 2 - 5, shape[0] // 2 + 6),) if len(shape) == 3 else ()
    eps[(*layers, slice(y0, y0 + core))] = SI
    for _ in range(6):  # scatterers: seed-dependent blocks away from the source
        h, w = int(rng.integers(3, max(4, ny // 4))), int(rng.integers(3, max(4, nx // 4)))
        yy, xx = int(rng.integers(0, ny - h)), int(rng.integers(nx // 2, max(nx // 2 + 1, nx - w)))
        eps[(*layers, slice(yy, yy + h), slice(xx, xx + w))] = rng.uniform(SIO2, SI)
    d = _loss_profile(nx, pml) + _loss_profile(ny, pml)[:, None]
    if len(shape) == 3:
        d = d[None] + _loss_profile(shape[0], pml)[:, None, None]
    smax = 4 * math.log(1e6) / (2 * math.sqrt(MU_0 / EPS_0) * pml * DX)
    return eps, smax * d / np.sqrt(eps)


def _grid(eps, sigma):
    """A mesh holding the program's own material arrays."""
    ny, nx = eps.shape[-2:]
    if eps.ndim == 2:
        d = bz.Design(width=(nx + 0.5) * DX, height=(ny + 0.5) * DX, auto_pml=False)
        g = bz.RegularGrid(d, DX)
    else:
        d = bz.Design(width=(nx + 0.5) * DX, height=(ny + 0.5) * DX, depth=(eps.shape[0] + 0.5) * DX, auto_pml=False)
        g = bz.RegularGrid3D(d, DX)
    np.copyto(g.permittivity, eps)
    np.copyto(g.conductivity, sigma)
    return g


def _case2d(case, seed):
    """Plain description of a 2D run: materials, time axis, source table and monitor lines."""
    rng = np.random.default_rng(seed)
    nx, ny, pml = case["nx"], case["ny"], case["pml"]
    eps, sigma = _materials((ny, nx), pml, rng)
    signal = (_pulse if case["source"] == "point" else _continuous)(case["steps"], _dt(2), rng)
    x_src = pml + max(3, (nx - 2 * pml) // 8)
    half = max(4, (ny - 2 * pml) // 4)
    rows = np.arange(ny // 2 - half, ny // 2 + half + 1)
    prof = np.exp(-((rows - ny // 2) / (0.4 * half)) ** 2)
    if case["source"] == "complex_line":
        prof = prof * np.exp(1j * (0.3 * (rows - ny // 2) / half + rng.uniform(0, 2 * np.pi)))
    if case["monitors"] == "record":
        lo, hx, hy = pml + 3, nx - pml - 4, ny - pml - 4
        lines = [(lo, lo, lo, hy), (hx, lo, hx, hy), (lo, lo, hx, lo), (lo, hy, hx, hy)]
        lines = lines if min(nx, ny) >= 100 else lines[1:2]
    else:
        xo, q = nx - pml - 5, max(3, half // 2)
        lines = [(x_src + 4, ny // 2 - half, x_src + 4, ny // 2 + half),
                 (xo, ny // 2 + 2, xo, ny // 2 + 2 + q), (xo, ny // 2 - 2 - q, xo, ny // 2 - 2)]
    return eps, sigma, signal, x_src, rows, prof, lines


def _case3d(case, seed):
    rng = np.random.default_rng(seed)
    nx, ny, nz, pml = case["nx"], case["ny"], case["nz"], case["pml"]
    eps, sigma = _materials((nz, ny, nx), pml, rng)
    signal = _pulse(case["steps"], _dt(3), rng)
    pos = (pml + max(3, (nx - 2 * pml) // 6), ny // 2, nz // 2)
    plane = (pos[0] + 2, pml + 1, min(nx - pml - 1, pos[0] + 42), ny - pml - 1, nz // 2 + 2)
    return eps, sigma, signal, pos, plane


def _case_adjoint(case, seed):
    rng = np.random.default_rng(seed)
    nx, ny, pml, r, b = case["nx"], case["ny"], case["pml"], case["region"], case["designs"]
    eps = np.full((ny, nx), SIO2)
    core = 25 if ny >= 200 else 11
    eps[ny // 2 - core // 2:ny // 2 - core // 2 + core, :] = SI
    d = _loss_profile(nx, pml) + _loss_profile(ny, pml)[:, None]
    sigma = 4 * math.log(1e6) / (2 * math.sqrt(MU_0 / EPS_0) * pml * DX) * d / np.sqrt(eps)
    box = (ny // 2 - r // 2, nx // 2 - r // 2, r, r)
    sigma[box[0]:box[0] + r, box[1]:box[1] + r] = 0.0
    rho = rng.random((b, r, r))
    for axis in (1, 2):  # densities as a filter leaves them: smooth over a few cells
        rho = sum(np.roll(rho, s, axis) for s in range(-2, 3)) / 5
    signal = _pulse(case["steps"], _dt(2), rng)
    src = (max(pml + 3, box[1] - 20), ny // 2)
    half = min(50, ny // 2 - pml - 6)
    x_mon = min(nx - pml - 4, box[1] + r + 20)
    mode = np.exp(-(np.arange(-half, half + 1) / (0.5 * core)) ** 2).astype(complex)
    # objective in units of a reference power, so that values and gradients are of order one
    weight = 1.0 / (case["steps"] * _dt(2) * DX * core) ** 2
    eps_box = (SIO2 + (SI - SIO2) * rho).astype(np.float32)
    return eps, sigma, box, eps_box, signal, src, half, x_mon, mode, weight


def _fno_weights(case, seed):
    """A float32 checkpoint of the network, as load_state_dict takes it, with a batch of densities."""
    g = torch.Generator().manual_seed(seed)
    c, hd, out, k = 32, 64, 5, 2 * case["modes"] ** 2

    def rnd(*shape, scale):
        return torch.randn(*shape, generator=g) * scale

    sd = {"W0": rnd(c, 3, scale=1 / math.sqrt(3)), "b0": rnd(c, scale=0.1)}
    for i in range(1, case["layers"] + 1):
        sd[f"W{i}"] = rnd(c, c, scale=1 / math.sqrt(c))
        sd[f"b{i}"] = rnd(c, scale=0.1)
        sd[f"R{i}"] = rnd(k, c, c, 2, scale=1 / c)
    sd["Q1"], sd["q1"] = rnd(hd, c, scale=1 / math.sqrt(c)), rnd(hd, scale=0.1)
    sd["Q2"], sd["q2"] = rnd(out, hd, scale=1 / math.sqrt(hd)), rnd(out, scale=0.1)
    n, b = case["n"], case["batch"]
    rho = torch.rand((b, 1, n + 8, n + 8), generator=g)
    rho = torch.nn.functional.avg_pool2d(rho, 9, stride=1)[:, 0] * 4 - 1.5  # smooth, mostly inside [0, 1]
    target = torch.rand((b, out), generator=g)
    return sd, rho.clamp(0, 1).contiguous(), target


# ---- a user's program ---------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "run2d":
        eps, sigma, signal, x_src, rows, prof, lines = _case2d(case, seed)
        grid = _grid(eps, sigma)
        if case["source"] == "point":
            src = bz.GaussianSource(position=(x_src * DX, (case["ny"] // 2) * DX), width=DX / 10, signal=signal)
        else:
            # a line source carrying the program's own mode profile
            src = bz.ModeSource(design=grid.design, position=(x_src * DX, (case["ny"] // 2) * DX),
                                width=(len(rows) - 1) * DX, wavelength=1.55 * UM, signal=signal, direction="+x",
                                num_modes=1, grid_resolution=200, npml=4)
            src.mode_profiles = [[[a, x_src * DX, y * DX, 0.0] for a, y in zip(prof, rows)]]
        return dict(case=case, grid=grid, source=src, lines=lines, time=np.arange(case["steps"]) * _dt(2))
    if kind == "run3d":
        eps, sigma, signal, pos, plane = _case3d(case, seed)
        grid = _grid(eps, sigma)
        src = bz.GaussianSource(position=tuple(p * DX for p in pos), width=1.5 * DX, signal=signal)
        return dict(case=case, grid=grid, source=src, plane=plane, time=np.arange(case["steps"]) * _dt(3))
    if kind == "adjoint":
        eps, sigma, box, eps_box, signal, src, half, x_mon, mode, weight = _case_adjoint(case, seed)
        from beamz_b200.optimization.adjoint import AdjointFDTD2D

        source = bz.GaussianSource(position=(src[0] * DX, src[1] * DX), width=2 * DX, signal=signal)
        yc = case["ny"] // 2
        mon = bz.Monitor(start=(x_mon * DX, (yc - half) * DX), end=(x_mon * DX, (yc + half) * DX))
        problem = AdjointFDTD2D(eps, sigma, DX, _dt(2), case["steps"], [source], mon, mode, C0 / (1.55 * UM), box,
                                n_designs=case["designs"], weights=[weight])
        return dict(case=case, problem=problem, eps=torch.from_numpy(eps_box).cuda().requires_grad_(True))
    from beamz_b200.surrogate.fno import FNO2d

    sd, rho, target = _fno_weights(case, seed)
    net = FNO2d(n=case["n"], width=32, modes=case["modes"], layers=case["layers"], head=64, n_out=5)
    net.load_state_dict(sd)
    return dict(case=case, net=net, rho=rho.cuda(), target=target.cuda())


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "run2d":
        dft = case["monitors"] == "dft"
        mons = [bz.Monitor(start=(x0 * DX, y0 * DX), end=(x1 * DX, y1 * DX), record_fields=not dft,
                           accumulate_power=not dft, wavelengths=WAVELENGTHS if dft else None)
                for x0, y0, x1, y1 in state["lines"]]
        sim = bz.FDTD(design=state["grid"], time=state["time"], devices=[state["source"], *mons],
                      backend_options={"precision": case["precision"]})
        sim.run(live=False, save=False, save_memory_mode=True, accumulate_power=case["power"])
        out = {"Ez": sim.Ez, "Hx": sim.Hx, "Hy": sim.Hy}
        for i, m in enumerate(mons):
            if dft:
                out.update({f"mon{i}_Ez": m.dft["Ez"], f"mon{i}_Hx": m.dft["Hx"], f"mon{i}_flux": m.flux()})
            else:
                out[f"mon{i}_Ez"], out[f"mon{i}_power"] = np.asarray(m.fields["Ez"]), np.asarray(m.power_history)
        if case["power"]:
            out["power"] = sim.power_accumulated
        return out
    if kind == "run3d":
        x0, y0, x1, y1, z = state["plane"]
        mon = bz.Monitor(design=state["grid"].design, start=(x0 * DX, y0 * DX, z * DX),
                         end=(x1 * DX, y1 * DX, z * DX), record_fields=False, accumulate_power=False,
                         wavelengths=WAVELENGTHS)
        sim = bz.FDTD(design=state["grid"], time=state["time"], devices=[state["source"], mon],
                      backend_options={"precision": case["precision"]})
        sim.run(live=False, save=False, save_memory_mode=True)
        out = {k: getattr(sim, k) for k in ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")}
        out.update(mon_Ez=mon.dft["Ez"], mon_Hx=mon.dft["Hx"], mon_flux=mon.flux())
        return out
    if kind == "adjoint":
        from beamz_b200.optimization.adjoint import FDTDObjective

        value = FDTDObjective.apply(state["eps"], state["problem"])
        (grad,) = torch.autograd.grad(value.sum(), state["eps"])
        return {"value": value.detach(), "grad": grad}
    net, rho = state["net"], state["rho"]
    if not case["train"]:
        return {"out": net.forward(rho)}
    net.zero_grad()
    out = net.forward(rho, keep=True)
    net.backward(2 * (out - state["target"]) / out.numel())
    return {"out": out, **{k: q.g for k, q in net.params.items()}}


def work(case):
    """Bytes: materials read and results written once. Flops: 14 per 2D cell update (H 6, E 8
    with two multiply-adds counted double), 36 per 3D one; the network's contractions."""
    kind = case["kind"]
    if kind == "run2d":
        cells, c = case["nx"] * case["ny"], 2 if case["source"] == "complex_line" else 1
        item = 8 if case["precision"] == "fp64" else 4
        return dict(bytes=cells * (16 + 3 * c * item + (8 if case["power"] else 0)),
                    flops=14.0 * c * cells * case["steps"])
    if kind == "run3d":
        cells = case["nx"] * case["ny"] * case["nz"]
        return dict(bytes=cells * (16 + 6 * (8 if case["precision"] == "fp64" else 4)),
                    flops=36.0 * cells * case["steps"])
    if kind == "adjoint":
        cells, box = case["nx"] * case["ny"], case["region"] ** 2
        return dict(bytes=16 * cells + 8 * box * case["designs"],
                    flops=2 * 14.0 * cells * case["designs"] * case["steps"])
    p, c, hd, k2 = case["n"] ** 2, 32, 64, 4 * case["modes"] ** 2
    # the truncated transforms as two passes of one-dimensional ones, the channel mixing, the head
    transform = 2 * c * case["n"] * (case["n"] * 2 * case["modes"] + 8 * case["modes"] ** 2)
    layer = 2 * transform + 2 * c * c * p + 8 * c * c * k2 // 2
    flops = case["batch"] * (case["layers"] * layer + 2 * 3 * c * p + 2 * c * hd * p) * (3 if case["train"] else 1)
    weights = 4 * (case["layers"] * (c * c + c + c * c * k2) + c * 4 + hd * (c + 6) + 5)
    return dict(bytes=4 * case["batch"] * p + weights * (2 if case["train"] else 1), flops=float(flops))


# ---- the same in float64 ------------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device=_dev())


def _gaussian_patch(centre, width, shape):
    """Cells and amplitudes of a Gaussian point source (centre and width in cells, x first)."""
    axes = []
    for c, n in zip(centre, shape):
        h, i = max(1, int(round(3 * width))), int(round(c))
        axes.append(np.arange(max(0, i - h), min(n, i + h + 1)))
    g = np.meshgrid(*axes[::-1], indexing="ij")[::-1]
    amp = np.exp(-sum((a - c) ** 2 / (2 * (width ** 2 + 1e-9)) for a, c in zip(g, centre)))
    return g, amp


def _phasors(steps, dt):
    f = C0 / np.asarray(WAVELENGTHS)
    n = np.arange(steps)[:, None]
    return np.exp(-2j * np.pi * f * (n + 1) * dt) * dt, np.exp(-2j * np.pi * f * (n + 0.5) * dt) * dt


def _exact2d(case, seed):
    eps, sigma, signal, x_src, rows, prof, lines = _case2d(case, seed)
    ny, nx, steps, dt = case["ny"], case["nx"], case["steps"], _dt(2)
    cplx = case["source"] == "complex_line"
    dtype = torch.complex128 if cplx else torch.float64
    a = _t(sigma) * dt / (2 * EPS_0)
    e = _t(eps)
    fh, cx = (1 - a) / (1 + a), dt / (MU_0 * DX) / (1 + a)
    fhx, chx, fhy, chy = fh[:, :-1].contiguous(), cx[:, :-1].contiguous(), fh[:-1].contiguous(), cx[:-1].contiguous()
    fe, ce = (1 - 2 * a / (e + a))[1:-1, 1:-1].contiguous(), (dt / (EPS_0 * DX * (e + a)))[1:-1, 1:-1].contiguous()
    ez = torch.zeros((ny, nx), dtype=dtype, device=_dev())
    hx, hy = torch.zeros_like(ez[:, :-1]).contiguous(), torch.zeros_like(ez[:-1]).contiguous()
    power = torch.zeros((ny, nx), dtype=torch.float64, device=_dev())
    if case["source"] == "point":
        (gx, gy), amp = _gaussian_patch((x_src * DX / DX, (ny // 2) * DX / DX), (DX / 10) / DX, (nx, ny))
        y0, y1, x0, x1 = int(gy.min()), int(gy.max()) + 1, int(gx.min()), int(gx.max()) + 1
        amp = _t(amp / 4)
    else:
        y0, y1, x0, x1 = int(rows[0]), int(rows[-1]) + 1, x_src, x_src + 1
        amp = _t(prof, dtype)[:, None]
    pe, ph = _phasors(steps, dt)
    pe, ph = _t(pe, torch.complex128), _t(ph, torch.complex128)
    dft = case["monitors"] == "dft"
    box = [(slice(ya, yb + 1), slice(xa, xb + 1)) for xa, ya, xb, yb in lines]
    recs = [torch.zeros((steps, 3, max(xb - xa, yb - ya) + 1), dtype=dtype, device=_dev()) for xa, ya, xb, yb in lines]
    hx_full, hy_full = torch.zeros_like(ez), torch.zeros_like(ez)
    for n in range(steps):
        hx.mul_(fhx).sub_(chx * (ez[:, 1:] - ez[:, :-1]))
        hy.mul_(fhy).add_(chy * (ez[1:] - ez[:-1]))
        curl = (hx[1:-1, :-1] - hx[1:-1, 1:]) + (hy[1:, 1:-1] - hy[:-1, 1:-1])
        inner = ez[1:-1, 1:-1]
        inner.mul_(fe).add_(ce * curl)
        ez[y0:y1, x0:x1].add_(amp, alpha=float(signal[n]))
        if case["source"] != "point":
            ez[y0:y1, x_src - 1] = 0  # the line radiates forwards: the field behind it is cleared
        if case["power"]:
            hx_full[:, :-1], hy_full[:-1] = hx, hy
            sx, sy = (ez * hy_full.conj()).real, (ez * hx_full.conj()).real
            power += sx ** 2 + sy ** 2
        for (ys, xs), r in zip(box, recs):
            r[n, 0] = ez[ys, xs].reshape(-1)
            if dft:  # Hx centred on the E nodes (vertical lines)
                r[n, 1] = (0.5 * (hx[ys, xs] + hx[ys, xs.start - 1:xs.stop - 1])).reshape(-1)
            else:
                r[n, 1] = hx[ys, xs].reshape(-1)
                r[n, 2] = hy[ys, xs].reshape(-1)
    out = {"Ez": ez, "Hx": hx, "Hy": hy}
    for i, r in enumerate(recs):
        if dft:
            r = r.real.to(torch.complex128)
            d_ez, d_hx = torch.einsum("np,nf->fp", r[:, 0], pe), torch.einsum("np,nf->fp", r[:, 1], ph)
            out.update({f"mon{i}_Ez": d_ez, f"mon{i}_Hx": d_hx,
                        f"mon{i}_flux": 0.5 * (d_ez * d_hx.conj()).real.sum(1) * DX})
        else:
            mag = (torch.sqrt((r[:, 0] * r[:, 2]) ** 2 + (r[:, 0] * r[:, 1]) ** 2)).sum(1)
            out.update({f"mon{i}_Ez": r[:, 0], f"mon{i}_power": mag})
    if case["power"]:
        out["power"] = power / steps
    return out


def _exact3d(case, seed):
    eps, sigma, signal, pos, plane = _case3d(case, seed)
    steps, dt = case["steps"], _dt(3)
    nz, ny, nx = eps.shape
    a, e = _t(sigma) * dt / (2 * EPS_0), _t(eps)
    fh, c, fe, ce = (1 - a) / (1 + a), dt / (MU_0 * DX) / (1 + a), 1 - 2 * a / (e + a), dt / (EPS_0 * DX * (e + a))
    ex, ey, ez, hx, hy, hz = (torch.zeros((nz, ny, nx), dtype=torch.float64, device=_dev()) for _ in range(6))
    (gx, gy, gz), amp = _gaussian_patch(tuple(p * DX / DX for p in pos), 1.5 * DX / DX, (nx, ny, nz))
    patch = tuple(slice(int(g.min()), int(g.max()) + 1) for g in (gz, gy, gx))
    amp = _t(amp)
    pe, ph = _phasors(steps, dt)
    x0, y0, x1, y1, z = plane
    sl = (z, slice(y0, y1), slice(x0, x1))
    rec = torch.zeros((5, steps, (y1 - y0) * (x1 - x0)), dtype=torch.float64, device=_dev())
    v0 = slice(None)

    def upd(f, s, fac, cc, curl):
        f[s].mul_(fac[s]).addcmul_(cc[s], curl)

    for n in range(steps):
        s = (slice(0, -1), slice(0, -1), v0)
        upd(hx, s, fh, c, (ey[1:, :-1] - ey[:-1, :-1]) - (ez[:-1, 1:] - ez[:-1, :-1]))
        s = (slice(0, -1), v0, slice(0, -1))
        upd(hy, s, fh, c, (ez[:-1, :, 1:] - ez[:-1, :, :-1]) - (ex[1:, :, :-1] - ex[:-1, :, :-1]))
        s = (v0, slice(0, -1), slice(0, -1))
        upd(hz, s, fh, c, (ex[:, 1:, :-1] - ex[:, :-1, :-1]) - (ey[:, :-1, 1:] - ey[:, :-1, :-1]))
        s = (slice(1, -1), slice(1, -1), slice(0, -1))
        upd(ex, s, fe, ce, (hz[1:-1, 1:-1, :-1] - hz[1:-1, :-2, :-1]) - (hy[1:-1, 1:-1, :-1] - hy[:-2, 1:-1, :-1]))
        s = (slice(1, -1), slice(0, -1), slice(1, -1))
        upd(ey, s, fe, ce, (hx[1:-1, :-1, 1:-1] - hx[:-2, :-1, 1:-1]) - (hz[1:-1, :-1, 1:-1] - hz[1:-1, :-1, :-2]))
        s = (slice(0, -1), slice(1, -1), slice(1, -1))
        upd(ez, s, fe, ce, (hy[:-1, 1:-1, 1:-1] - hy[:-1, 1:-1, :-2]) - (hx[:-1, 1:-1, 1:-1] - hx[:-1, :-2, 1:-1]))
        ez[patch].add_(amp, alpha=float(signal[n]))
        for q, f in enumerate((ez, hx, ex, ey, hy)):
            rec[q, n] = f[sl].reshape(-1)
    pe, ph = _t(pe, torch.complex128), _t(ph, torch.complex128)
    shp = (len(WAVELENGTHS), y1 - y0, x1 - x0)

    def dft(r, p):
        return torch.einsum("np,nf->fp", r.to(torch.complex128), p)

    d_ez, d_hx, d_ex, d_ey, d_hy = (dft(r, p) for r, p in zip(rec, (pe, ph, pe, pe, ph)))
    flux = 0.5 * (d_ex * d_hy.conj() - d_ey * d_hx.conj()).real.sum(1) * DX * DX
    return {"Ex": ex[:, :, :-1], "Ey": ey[:, :-1], "Ez": ez[:-1], "Hx": hx[:-1, :-1], "Hy": hy[:-1, :, :-1],
            "Hz": hz[:, :-1, :-1], "mon_Ez": d_ez.reshape(shp), "mon_Hx": d_hx.reshape(shp), "mon_flux": flux}


def _exact_adjoint(case, seed):
    eps, sigma, box, eps_box, signal, src, half, x_mon, mode, weight = _case_adjoint(case, seed)
    ny, nx, steps, dt = case["ny"], case["nx"], case["steps"], _dt(2)
    y0, x0, h, w = box
    a, base = _t(sigma) * dt / (2 * EPS_0), _t(eps)
    fh, cx = (1 - a) / (1 + a), dt / (MU_0 * DX) / (1 + a)
    fe = (1 - 2 * a / (base + a))[1:-1, 1:-1]  # 1 in the box, which is free of loss
    (gx, gy), amp = _gaussian_patch((src[0] * DX / DX, src[1] * DX / DX), 2 * DX / DX, (nx, ny))
    pad = torch.zeros((ny, nx), dtype=torch.float64, device=_dev())
    pad[int(gy.min()):int(gy.max()) + 1, int(gx.min()):int(gx.max()) + 1] = _t(amp / 4)
    pad = pad[1:-1, 1:-1]
    phi = np.exp(-2j * np.pi * C0 / (1.55 * UM) * (np.arange(steps) + 1.0) * dt) * dt
    wp = _t(np.conj(mode) * DX, torch.complex128)
    ym = slice(ny // 2 - half, ny // 2 + half + 1)
    mask = torch.zeros((ny, nx), dtype=torch.float64, device=_dev())
    mask[y0:y0 + h, x0:x0 + w] = 1

    def segment(ez, hx, hy, ce, n0, n1):
        acc_r = acc_i = 0.0
        for n in range(n0, n1):
            hx = fh[:, :-1] * hx - cx[:, :-1] * (ez[..., 1:] - ez[..., :-1])
            hy = fh[:-1] * hy + cx[:-1] * (ez[..., 1:, :] - ez[..., :-1, :])
            curl = (hx[..., 1:-1, :-1] - hx[..., 1:-1, 1:]) + (hy[..., 1:, 1:-1] - hy[..., :-1, 1:-1])
            inner = fe * ez[..., 1:-1, 1:-1] + ce * curl + pad * float(signal[n])
            ez = torch.nn.functional.pad(inner, (1, 1, 1, 1))
            line = ez[..., ym, x_mon]
            acc_r, acc_i = acc_r + line * float(phi[n].real), acc_i + line * float(phi[n].imag)
        return ez, hx, hy, acc_r, acc_i

    from torch.utils.checkpoint import checkpoint

    values, grads = [], []
    group = max(1, min(case["designs"], 4_000_000 // (nx * ny)))
    for b in range(0, case["designs"], group):
        er = _t(eps_box[b:b + group]).requires_grad_(True)
        full = base * (1 - mask) + torch.nn.functional.pad(er, (x0, nx - x0 - w, y0, ny - y0 - h))
        ce = (dt / (EPS_0 * DX * (full + a)))[:, 1:-1, 1:-1]
        ez = torch.zeros((er.shape[0], ny, nx), dtype=torch.float64, device=_dev())
        hx, hy = torch.zeros_like(ez[..., :-1]), torch.zeros_like(ez[:, :-1])
        sr = si = 0.0
        for n0 in range(0, steps, 40):
            ez, hx, hy, ar, ai = checkpoint(segment, ez, hx, hy, ce, n0, min(steps, n0 + 40), use_reentrant=False)
            sr, si = sr + ar, si + ai
        amp_f = (torch.complex(sr, si) * wp).sum(-1)
        j = weight * (amp_f.real ** 2 + amp_f.imag ** 2)
        (g,) = torch.autograd.grad(j.sum(), er)
        values.append(j.detach())
        grads.append(g)
    return {"value": torch.cat(values), "grad": torch.cat(grads)}


def _exact_fno(case, seed):
    sd, rho, target = _fno_weights(case, seed)
    n, m, b = case["n"], case["modes"], case["batch"]
    p = {k: _t(v).requires_grad_(case["train"]) for k, v in sd.items()}
    ky, kx = torch.cat([torch.arange(m), torch.arange(n - m, n)]).to(_dev()), torch.arange(m, device=_dev())

    def gelu(v):
        return 0.5 * v * (1 + torch.tanh(math.sqrt(2 / math.pi) * (v + 0.044715 * v ** 3)))

    cc = (torch.arange(n, dtype=torch.float64, device=_dev()) + 0.5) / n

    def net(r):
        x = torch.stack([r, cc[None, None, :].expand_as(r), cc[None, :, None].expand_as(r)], 1)
        v = torch.einsum("cj,bjyx->bcyx", p["W0"], x) + p["b0"][:, None, None]
        for i in range(1, case["layers"] + 1):
            u = torch.fft.rfft2(v)[:, :, ky][..., kx].reshape(r.shape[0], 32, -1)  # kept modes
            o = torch.einsum("bck,kco->bok", u, torch.view_as_complex(p[f"R{i}"]))
            s = torch.zeros((r.shape[0], 32, n, n // 2 + 1), dtype=torch.complex128, device=_dev())
            s = s.index_put((torch.arange(r.shape[0], device=_dev())[:, None, None, None],
                             torch.arange(32, device=_dev())[None, :, None, None], ky[None, None, :, None],
                             kx[None, None, None, :]), o.reshape(r.shape[0], 32, 2 * m, m))
            # kx = 0 columns carry weight 1 in the real inverse sum: Re over (ky, 0) alone
            full = torch.fft.ifft(s, dim=2)
            wx = torch.where(kx == 0, 1.0, 2.0)
            ph = torch.exp(2j * math.pi * kx[:, None] * torch.arange(n, device=_dev())[None, :] / n) * wx[:, None] / n
            sp = torch.einsum("bcyk,kx->bcyx", full[..., :m], ph.to(torch.complex128)).real
            v = torch.einsum("oc,bcyx->boyx", p[f"W{i}"], v) + p[f"b{i}"][:, None, None] + sp
            v = gelu(v) if i < case["layers"] else v
        hid = gelu(torch.einsum("hc,bcyx->bhyx", p["Q1"], v) + p["q1"][:, None, None]).mean((2, 3))
        return hid @ p["Q2"].T + p["q2"]

    outs, grads = [], None
    for i in range(0, b, 8):
        r = _t(rho[i:i + 8].numpy())
        with torch.set_grad_enabled(case["train"]):
            out = net(r)
            outs.append(out.detach())
            if case["train"]:
                loss = ((out - _t(target[i:i + 8].numpy())) ** 2).sum() / (b * out.shape[1])
                g = torch.autograd.grad(loss, list(p.values()))
                grads = list(g) if grads is None else [u + v for u, v in zip(grads, g)]
    res = {"out": torch.cat(outs)}
    if case["train"]:
        res.update(zip(p, grads))
    return res


def exact(case, seed):
    return {"run2d": _exact2d, "run3d": _exact3d, "adjoint": _exact_adjoint, "fno": _exact_fno}[case["kind"]](case, seed)
