"""The calls whose time is followed, over the sizes that users of this framework run.

Every case names a ``kind`` (one public entry point) and its sizes:

  tm        simulate_tm: one 2D run with a line source, a port, probes and a
            running DFT (float32 with complex64 phasors, or float64)
  tm_pulse  the gradient of the radiated power of a pulse-driven antenna with
            respect to its density (time_domain_objective + backward)
  tm_cw     the same for a CW drive (freq_adjoint_objective + backward), with
            P_rad - |S11|^2 as the objective
  tm_pop    freq_adjoint_gradient_batch: a population of uneven problems
  yee       simulate_3d: one 3D run with a current source, a port, probes and
            phasors on three boxes
  yee_cw    freq_adjoint_gradient_3d of a microstrip patch (S11 and the
            directivity from the near-to-far-field transform)
  unet      the surrogate network's loss and its gradients (the forward and
            backward passes of a training step)
  unet_grad the surrogate's predicted power and its gradient (the optimiser's
            inner step)
  ntff      ntff_3d: the radiation pattern from the phasors of a run

``exact`` restates each of them in plain torch float64, where that takes
seconds; the population and the 3D gradient are too long for it.
"""

from __future__ import annotations

import math

import numpy as np
import torch
import torch.nn.functional as F

C0 = 299792458.0
MU0 = 1.25663706212e-06
EPS0 = 1.0 / (MU0 * C0 * C0)
ETA0 = math.sqrt(MU0 / EPS0)
F64, C128 = torch.float64, torch.complex128


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------


def listed():
    return [
        # A first look at a structure: a short run on an odd-sized grid, where
        # the set-up and the launches weigh most.
        dict(name="tm_short", kind="tm", nx=70, ny=53, npml=8, steps=300, freqs=2, f64=False),
        # The README's antenna: 140 x 140 at 2 mm, 3500 steps of a 2-3 GHz pulse.
        dict(name="tm_readme_grad", kind="tm_pulse", n=140, npml=10, steps=3500, d0=44, d1=60,
             size=52, f64=False),
        # The antenna-growth hero at the default float64: 280 x 280 at 1 mm,
        # 104 x 104 design, 7000 steps at 2.45 GHz.
        dict(name="tm_hero_grad_f64", kind="tm_cw", n=280, npml=10, steps=7000, freqs=1, size=104,
             f64=True),
        # The large design gradient: 1024 x 1024, 512 x 512 design, four tones.
        dict(name="tm_large_grad", kind="tm_cw", n=1024, npml=16, steps=8000, freqs=4, size=512,
             f64=False),
        # A scan over frequency on a mid-sized grid with phasors everywhere.
        dict(name="tm_scan", kind="tm", nx=517, ny=384, npml=12, steps=2000, freqs=8, f64=False),
        # The large grid in float64 (reference runs of a converged design).
        dict(name="tm_large_f64", kind="tm", nx=1024, ny=1024, npml=16, steps=1000, freqs=2,
             f64=True),
        # A topology-optimisation population of uneven problems.
        dict(name="tm_population", kind="tm_pop", count=24, lo=128, hi=512, steps_lo=2000,
             steps_hi=6000),
        # A 3D structure on an odd-sized grid, float32 and float64.
        dict(name="yee_odd", kind="yee", nx=97, ny=83, nz=61, npml=8, steps=600, freqs=3,
             f64=False),
        dict(name="yee_f64", kind="yee", nx=64, ny=64, nz=48, npml=8, steps=400, freqs=2,
             f64=True),
        # The microstrip patch gradient: 160 x 160 x 64 at 0.5 mm, 96 x 96
        # design sheet, 11 tones; 3000 steps each way.
        dict(name="yee_patch_grad", kind="yee_cw", n=160, nz=64, npml=10, steps=3000, freqs=11,
             size=96),
        # The surrogate's training passes at its own batch and image size.
        dict(name="unet_train", kind="unet", batch=32, side=104, base=32),
        # A full-sphere pattern of the patch's size at five frequencies.
        dict(name="ntff_pattern", kind="ntff", nx=96, ny=96, nz=48, freqs=5, thetas=37, phis=72,
             f64=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tm", "tm", "tm", "tm_pulse", "tm_cw", "tm_cw", "tm_pop", "yee", "yee",
                       "yee_cw", "unet", "unet_grad", "ntff"])
    npml = rng.randint(8, 16)
    if kind == "tm":
        return dict(kind=kind, nx=_log_int(rng, 48, 1024), ny=_log_int(rng, 48, 1024), npml=npml,
                    steps=_log_int(rng, 200, 3000), freqs=rng.randint(1, 8),
                    f64=rng.random() < 0.35)
    if kind == "tm_pulse":
        n = _log_int(rng, 100, 300)
        size = rng.randint(n // 5, n // 3)
        return dict(kind=kind, n=n, npml=npml, steps=_log_int(rng, 800, 3500), d0=n // 3,
                    d1=n // 3 + 2, size=size, f64=rng.random() < 0.3)
    if kind == "tm_cw":
        n = _log_int(rng, 128, 1024)
        return dict(kind=kind, n=n, npml=npml, steps=_log_int(rng, 1500, 6000),
                    freqs=rng.randint(1, 6), size=rng.randint(n // 4, n // 2),
                    f64=rng.random() < 0.4)
    if kind == "tm_pop":
        lo = rng.randint(128, 200)
        return dict(kind=kind, count=rng.randint(3, 20), lo=lo, hi=rng.randint(lo + 60, 512),
                    steps_lo=1000, steps_hi=rng.randint(2000, 5000))
    if kind == "yee":
        return dict(kind=kind, nx=_log_int(rng, 40, 170), ny=_log_int(rng, 40, 170),
                    nz=_log_int(rng, 36, 100), npml=rng.randint(6, 12),
                    steps=_log_int(rng, 150, 1000), freqs=rng.randint(1, 6),
                    f64=rng.random() < 0.35)
    if kind == "yee_cw":
        n = rng.randint(90, 160)
        return dict(kind=kind, n=n, nz=rng.randint(48, 64), npml=rng.randint(8, 10),
                    steps=_log_int(rng, 500, 2500), freqs=rng.randint(2, 11), size=n // 2)
    if kind == "unet":
        return dict(kind=kind, batch=_log_int(rng, 2, 32), side=8 * rng.randint(6, 16),
                    base=rng.choice([16, 32]))
    if kind == "unet_grad":
        return dict(kind=kind, batch=_log_int(rng, 1, 64), side=8 * rng.randint(6, 16),
                    base=rng.choice([16, 32]))
    return dict(kind=kind, nx=rng.randint(40, 140), ny=rng.randint(40, 140),
                nz=rng.randint(36, 70), freqs=rng.randint(1, 6), thetas=rng.randint(5, 37),
                phis=rng.randint(4, 72), f64=rng.random() < 0.4)


# ---------------------------------------------------------------------------
# Inputs of a case (numpy, from the seed alone)
# ---------------------------------------------------------------------------


def _dt2(dx):
    return 0.99 / (C0 * math.sqrt(2.0 / dx**2))


def _dt3(dx):
    return 0.99 / (C0 * math.sqrt(3.0 / dx**2))


def _density(rng, shape, radius=2):
    """A blurred and projected random density in (0, 1), like a half-grown design."""
    x = rng.uniform(size=shape)
    for ax in range(len(shape)):
        if shape[ax] > 2 * radius:
            x = sum(np.roll(x, s, ax) for s in range(-radius, radius + 1)) / (2 * radius + 1)
    return 0.5 + 0.5 * np.tanh(16.0 * (x - 0.5))


def _sigma(rho):
    return 10.0 ** (9.0 * rho - 4.0)


def _tones(rng, k, lo=2.0e9, hi=3.0e9):
    return tuple(float(f) for f in np.sort(rng.uniform(lo, hi, k)))


def _cw(freqs, env, dt):
    n = np.arange(len(env))
    return env * sum(np.sin(2 * np.pi * f * (n + 0.5) * dt) for f in freqs)


def _tm_inputs(c, seed):
    rng = np.random.default_rng(seed)
    nx, ny, m = c["nx"], c["ny"], c["npml"]
    dx = 1e-3
    dt = _dt2(dx)
    t = (np.arange(c["steps"]) + 0.5) * dt
    u = (t - 60 * dt) / (15 * dt)
    src = -u * np.exp(0.5 * (1.0 - u**2)) * rng.uniform(0.5, 1.5)
    sigma = np.zeros((nx, ny))
    eps = np.ones((nx, ny))
    a, b = slice(nx // 3, nx // 3 + nx // 4), slice(ny // 3, ny // 3 + ny // 4)
    eps[a, b] = 1.0 + 3.0 * rng.uniform(size=eps[a, b].shape)
    sigma[a, b] = 0.5 * rng.uniform(size=eps[a, b].shape)
    cell = lambda: (int(rng.integers(m + 2, nx - m - 2)), int(rng.integers(m + 2, ny - m - 2)))  # noqa: E731
    return dict(dx=dx, dt=dt, eps=eps, sigma=sigma, src=cell(), cur=src, port=cell(),
                vs=0.3 * np.roll(src, 20), probes=[cell() for _ in range(4)],
                freqs=_tones(rng, c["freqs"], 1e9, 6e9))


def _pulse_inputs(c, seed):
    rng = np.random.default_rng(seed)
    dx, n = 2e-3, c["n"]
    dt = _dt2(dx)
    f0, fc = 2.5e9, 0.5e9
    s, t0 = 3.0 / (2.0 * math.sqrt(2.0) * math.pi * fc), 9.0 / (2.0 * math.pi * fc)
    t = (np.arange(c["steps"]) + 0.5) * dt - t0
    rho = 0.5 + 0.1 * (_density(rng, (c["size"], c["size"])) - 0.5)
    return dict(dx=dx, dt=dt, vs=np.cos(2 * np.pi * f0 * t) * np.exp(-t**2 / (2 * s**2)),
                rho=rho, port=(n // 2, c["d1"] - 5), freq=2.45e9, box=(20, n - 20, 20, n - 20))


def _cw_inputs(c, seed):
    rng = np.random.default_rng(seed)
    n, m = c["n"], c["npml"]
    dx = 1e-3
    dt = _dt2(dx)
    freqs = (2.45e9,) if c["freqs"] == 1 else tuple(float(f) for f in
                                                    np.linspace(2e9, 3e9, c["freqs"]))
    env = np.clip(np.arange(c["steps"]) / 300.0, 0.0, 1.0)
    d0 = (n - c["size"]) // 2
    b = m + 6
    return dict(dx=dx, dt=dt, freqs=freqs, env=env, vs=_cw(freqs, env, dt), d0=d0,
                rho=_density(rng, (c["size"], c["size"]), 3), box=(b, n - b - 1, b, n - b - 1),
                ports=((d0 - 4, n // 2), (n - d0 + 3, n // 2)))


def _pop_inputs(c, seed):
    rng = np.random.default_rng(seed)
    sizes = np.random.default_rng(c["count"] * 1000 + c["hi"])  # one population, its designs by the seed
    out = []
    for _ in range(c["count"]):
        n = int(sizes.integers(c["lo"], c["hi"] + 1))
        m = int(sizes.integers(10, 17))
        steps = int(sizes.integers(c["steps_lo"], c["steps_hi"] + 1))
        freqs = _tones(sizes, int(sizes.integers(1, 9)), 1e9, 6e9)
        dt = _dt2(1e-3)
        env = np.clip(np.arange(steps) / 300.0, 0.0, 1.0)
        lo, hi = m + 3, n // 4 - 2
        ports = [(int(sizes.integers(lo, hi)), int(sizes.integers(lo, n - lo)))
                 for _ in range(int(sizes.integers(1, 5)))]
        out.append(dict(n=n, npml=m, freqs=freqs, env=env, vs=_cw(freqs, env, dt), ports=ports,
                        sigma=_sigma(_density(rng, (n // 2, n // 2), 3))))
    return out


def _yee_inputs(c, seed):
    rng = np.random.default_rng(seed)
    shape = (c["nx"], c["ny"], c["nz"])
    m, dx = c["npml"], 1e-3
    dt = _dt3(dx)
    t = (np.arange(c["steps"]) + 0.5) * dt
    u = (t - 40 * dt) / (12 * dt)
    eps, sigma = np.ones(shape), np.zeros(shape)
    box = tuple(slice(s // 3, s // 3 + s // 4) for s in shape)
    eps[box] = 1.0 + 3.0 * rng.uniform(size=eps[box].shape)
    sigma[box] = 0.5 * rng.uniform(size=eps[box].shape)
    cell = lambda: tuple(int(rng.integers(m + 2, s - m - 3)) for s in shape)  # noqa: E731
    lo, hi = (m + 2,) * 3, tuple(s - m - 3 for s in shape)
    mid = shape[2] // 2
    return dict(dx=dx, dt=dt, eps=eps, sigma=sigma, src=cell(), port=cell(),
                cur=1e-3 * -u * np.exp(0.5 * (1.0 - u**2)) * rng.uniform(0.5, 1.5),
                vs=0.3 * np.exp(-0.5 * u**2), probes=[cell() for _ in range(3)],
                freqs=_tones(rng, c["freqs"], 2e9, 1e10),
                boxes=[(2, (lo[0], lo[1], mid), (hi[0], hi[1], mid + 1)),
                       (0, lo, (hi[0], hi[1], lo[2] + 2)),
                       (4, lo, (lo[0] + 2, hi[1], hi[2]))])


def _patch_inputs(c, seed):
    """A patch of random copper over a grounded substrate, fed by a pin."""
    rng = np.random.default_rng(seed)
    n, nz, m, size = c["n"], c["nz"], c["npml"], c["size"]
    d = 0.5e-3
    dt = _dt3(d)
    kg = m + 3
    kp = kg + 5
    d0 = (n - size) // 2
    d1 = d0 + size
    eps, sig = np.ones((n, n, nz)), np.zeros((n, n, nz))
    eps[d0 - 6:d1 + 6, d0 - 6:d1 + 6, kg + 1:kp] = 4.4
    sig[d0 - 6:d1 + 6, d0 - 6:d1 + 6, kg] = 1e7
    pi, pj = (d0 + d1) // 2, d0 + size // 4
    sig[pi, pj, kg + 1:kp - 1] = 1e7
    rho = _density(rng, (size, size), 3)
    rho[pi - d0, pj - d0] = 1.0
    freqs = tuple(float(f) for f in np.linspace(2e9, 3e9, c["freqs"]))
    env = np.clip(np.arange(c["steps"]) / 300.0, 0.0, 1.0)
    return dict(dx=d, dt=dt, freqs=freqs, env=env, vs=_cw(freqs, env, dt), eps=eps, sig=sig,
                design=(slice(d0, d1), slice(d0, d1), slice(kp, kp + 1)),
                sigma=(35e-6 / d * _sigma(rho))[:, :, None], port=(pi, pj, kp - 1), margin=m + 2)


LEVELS = 4


def _unet_layers(base):
    """(name, cin, cout, taps, w_off, b_off) in the flat parameter order."""
    ch = [base << lev for lev in range(LEVELS)]
    shapes = []
    for lev in range(LEVELS):
        shapes += [(f"enc{lev}a", 1 if lev == 0 else ch[lev - 1], ch[lev], 9),
                   (f"enc{lev}b", ch[lev], ch[lev], 9)]
    for lev in range(LEVELS - 2, -1, -1):
        shapes += [(f"up{lev}", ch[lev + 1], ch[lev], 9), (f"dec{lev}a", 2 * ch[lev], ch[lev], 9),
                   (f"dec{lev}b", ch[lev], ch[lev], 9)]
    shapes.append(("head", ch[0], 3, 1))
    out, off = [], 0
    for name, cin, cout, taps in shapes:
        w = off
        b = (w + taps * cin * cout + 7) // 8 * 8
        off = (b + cout + 7) // 8 * 8
        out.append((name, cin, cout, taps, w, b))
    return out, off


def _unet_inputs(c, seed):
    rng = np.random.default_rng(seed)
    n, s = c["batch"], c["side"]
    layers, count = _unet_layers(c["base"])
    theta = np.zeros(count, np.float32)
    for name, cin, cout, taps, w, b in layers:
        std = math.sqrt((1.0 if name == "head" else 2.0) / (taps * cin))
        theta[w:w + taps * cin * cout] = rng.normal(0.0, std, taps * cin * cout)
        theta[b:b + cout] = rng.normal(0.0, 0.02, cout)
    x = np.stack([_density(rng, (s, s)) for _ in range(n)]).astype(np.float32)
    return dict(theta=theta, x=x, field=rng.normal(0.0, 0.5, (n, s, s, 2)).astype(np.float32),
                power=rng.uniform(0.0, 1.0, n).astype(np.float32),
                weight=rng.uniform(0.5, 1.5, n).astype(np.float32))


def _ntff_inputs(c, seed):
    rng = np.random.default_rng(seed)
    n = (c["nx"], c["ny"], c["nz"])
    freqs = _tones(rng, c["freqs"], 2e9, 6e9)
    comps = []
    for k, off in enumerate(((1, 0, 0), (0, 1, 0), (0, 0, 1), (0, 1, 1), (1, 0, 1), (1, 1, 0))):
        # waves of a few random directions: phasors as smooth as a run's
        f = 0.0
        for _ in range(2):
            amp = (rng.normal(size=len(freqs)) + 1j * rng.normal(size=len(freqs)))
            f = f + torch.einsum("f,x,y,z->fxyz", *(
                torch.as_tensor(a.astype(np.complex64), device="cuda") for a in (
                    amp * (1.0 if k < 3 else 1.0 / 377.0),
                    *(np.exp(1j * q * np.arange(s - o))
                      for q, s, o in zip(rng.normal(size=3) * 0.05, n, off)))))
        comps.append(f)
    return dict(dx=1e-3, freqs=freqs, comps=comps, margin=10,
                thetas=np.linspace(0.0, np.pi, c["thetas"]),
                phis=np.linspace(0.0, 2 * np.pi, c["phis"], endpoint=False))


# ---------------------------------------------------------------------------
# prepare / run: what a user's program keeps, and the call it makes
# ---------------------------------------------------------------------------


def prepare(case, seed):
    import gradenna_b200 as gb

    c, kind = case, case["kind"]
    dev = torch.device("cuda")
    s = dict(case=c, dev=dev)
    if kind == "tm":
        i = _tm_inputs(c, seed)
        dt = F64 if c["f64"] else torch.float32
        to = lambda a: torch.as_tensor(a, dtype=dt, device=dev)  # noqa: E731
        s.update(grid=gb.Grid2D(c["nx"], c["ny"], i["dx"], i["dx"]), kw=dict(
            source_ij=i["src"], source_current=to(i["cur"]), eps_r=to(i["eps"]),
            sigma=to(i["sigma"]), ports=(gb.Port(i["port"], 50.0, to(i["vs"])),),
            probe_ij=i["probes"], dft_freqs=i["freqs"], cpml=gb.CPMLSpec(c["npml"]), dtype=dt))
    elif kind == "tm_pulse":
        i = _pulse_inputs(c, seed)
        dt = F64 if c["f64"] else torch.float32
        s.update(grid=gb.Grid2D(c["n"], c["n"], i["dx"], i["dx"]), dtype=dt, box=i["box"],
                 freq=i["freq"], cpml=gb.CPMLSpec(c["npml"]),
                 rho=torch.as_tensor(i["rho"], dtype=dt, device=dev),
                 ports=(gb.Port(i["port"], 50.0, torch.as_tensor(i["vs"], dtype=dt, device=dev)),),
                 region=(slice(c["d0"], c["d0"] + c["size"]), slice(c["d1"], c["d1"] + c["size"])))
    elif kind == "tm_cw":
        from gradenna_b200.monitors import port_monitors
        from gradenna_b200.objectives import RadiatedPowerS11

        i = _cw_inputs(c, seed)
        dt = F64 if c["f64"] else torch.float32
        grid = gb.Grid2D(c["n"], c["n"], i["dx"], i["dx"])
        obj = RadiatedPowerS11(grid, i["box"], i["ports"][0], i["freqs"])
        d = slice(i["d0"], i["d0"] + c["size"])
        s.update(grid=grid, obj=obj, mons=obj.monitors() + port_monitors(i["ports"][1]),
                 region=(d, d), freqs=i["freqs"], env=i["env"], dtype=dt,
                 cpml=gb.CPMLSpec(c["npml"]), rho=torch.as_tensor(i["rho"], dtype=dt, device=dev),
                 ports=(gb.Port(i["ports"][0], 50.0, torch.as_tensor(i["vs"], dtype=dt, device=dev)),
                        gb.Port(i["ports"][1], 50.0, None)))
    elif kind == "tm_pop":
        from gradenna_b200.monitors import port_monitors
        from gradenna_b200.objectives import RadiatedPowerS11

        specs = []
        for p in _pop_inputs(c, seed):
            n, m = p["n"], p["npml"]
            grid = gb.Grid2D(n, n, 1e-3, 1e-3)
            b = m + 4
            obj = RadiatedPowerS11(grid, (b, n - b - 1, b, n - b - 1), p["ports"][0], p["freqs"])
            mons = obj.monitors()
            for q in p["ports"][1:]:
                mons = mons + port_monitors(q)
            d = slice(n // 4, n // 4 + n // 2)
            specs.append(dict(
                grid=grid, objective=obj, design_region=(d, d), dft_freqs=p["freqs"], env=p["env"],
                design_sigma=torch.as_tensor(p["sigma"], dtype=F64, device=dev),
                ports=tuple(gb.Port(q, 50.0, p["vs"] if k == 0 else None)
                            for k, q in enumerate(p["ports"])),
                cpml=gb.CPMLSpec(m), dtype=torch.float32, objective_monitors=mons))
        s.update(specs=specs)
    elif kind == "yee":
        i = _yee_inputs(c, seed)
        dt = F64 if c["f64"] else torch.float32
        to = lambda a: torch.as_tensor(a, dtype=dt, device=dev)  # noqa: E731
        s.update(grid=gb.Grid3D(c["nx"], c["ny"], c["nz"], i["dx"], i["dx"], i["dx"]), kw=dict(
            source_ijk=i["src"], source_current=to(i["cur"]), port_ijk=i["port"],
            port_voltage=to(i["vs"]), eps_r=to(i["eps"]), sigma=to(i["sigma"]),
            probe_ijk=i["probes"], dft_freqs=i["freqs"], dft_monitors=i["boxes"],
            cpml=gb.CPMLSpec(c["npml"]), dtype=dt))
    elif kind == "yee_cw":
        i = _patch_inputs(c, seed)
        to = lambda a: torch.as_tensor(a, dtype=F64, device=dev)  # noqa: E731
        s.update(grid=gb.Grid3D(c["n"], c["n"], c["nz"], i["dx"], i["dx"], i["dx"]),
                 freqs=i["freqs"], margin=i["margin"], kw=dict(
            design_sigma=to(i["sigma"]), design_region=i["design"], dft_freqs=i["freqs"],
            env=i["env"], port_ijk=i["port"],
            port_voltage=torch.as_tensor(i["vs"], dtype=torch.float32, device=dev),
            cpml=gb.CPMLSpec(c["npml"]), dtype=torch.float32,
            objective_kind=("port", "ntff_box"), box_margin=i["margin"],
            eps_r_background=to(i["eps"]), sigma_background=to(i["sig"])))
    elif kind in ("unet", "unet_grad"):
        from gradenna_b200.unet import UNet, UNetSpec

        i = _unet_inputs(c, seed)
        spec = UNetSpec(c["side"], c["side"], c["base"], LEVELS)
        net = UNet(spec)
        net.load_state_dict({"spec": spec.__dict__.copy(), "theta": torch.as_tensor(i["theta"])})
        s.update(net=net, **{k: torch.as_tensor(i[k], device=dev)
                             for k in ("x", "field", "power", "weight")})
    elif kind == "ntff":
        from gradenna_b200.fdtd3d import DFTMonitor

        i = _ntff_inputs(c, seed)
        dt = C128 if c["f64"] else torch.complex64
        s.update(grid=gb.Grid3D(c["nx"], c["ny"], c["nz"], i["dx"], i["dx"], i["dx"]),
                 mon=DFTMonitor(torch.tensor(i["freqs"], device=dev),
                                *(torch.as_tensor(a, dtype=dt, device=dev) for a in i["comps"])),
                 args=(i["margin"], i["freqs"], i["thetas"], i["phis"]))
    else:
        raise ValueError(f"unknown kind {kind!r}")
    return s


def run(s):
    kind = s["case"]["kind"]
    if kind == "tm":
        from gradenna_b200 import simulate_tm

        r = simulate_tm(s["grid"], **s["kw"])
        return {k: getattr(r, k) for k in ("probe_ez", "port_v", "port_i", "ez", "hx", "hy",
                                           "dft_ez", "dft_hx", "dft_hy")}
    if kind == "tm_pulse":
        from gradenna_b200.materials import sigma_from_density
        from gradenna_b200.monitors import poynting_flux_box_2d
        from gradenna_b200.time_adjoint import time_domain_objective

        grid, box = s["grid"], s["box"]
        rho = s["rho"].detach().requires_grad_(True)
        loss = -time_domain_objective(
            sigma_from_density(rho), grid,
            lambda ph: poynting_flux_box_2d(ph.dft_ez, ph.dft_hx, ph.dft_hy, grid, box)[0],
            design_region=s["region"], dft_freqs=(s["freq"],), ports=s["ports"], cpml=s["cpml"],
            dtype=s["dtype"])
        loss.backward()
        return {"grad": rho.grad, "loss": loss.detach().to(rho.dtype)}
    if kind == "tm_cw":
        from gradenna_b200.freq_adjoint import freq_adjoint_objective
        from gradenna_b200.materials import sigma_from_density

        rho = s["rho"].detach().requires_grad_(True)
        loss = -freq_adjoint_objective(
            sigma_from_density(rho), s["grid"], s["obj"], design_region=s["region"],
            dft_freqs=s["freqs"], env=s["env"], ports=s["ports"], cpml=s["cpml"],
            dtype=s["dtype"], objective_monitors=s["mons"])
        loss.backward()
        return {"grad": rho.grad, "loss": loss.detach().to(rho.dtype)}
    if kind == "tm_pop":
        from gradenna_b200.batch import freq_adjoint_gradient_batch

        return [g["sigma"] for g in freq_adjoint_gradient_batch(s["specs"])]
    if kind == "yee":
        from gradenna_b200 import simulate_3d

        r = simulate_3d(s["grid"], **s["kw"])
        out = {k: getattr(r, k) for k in ("probe_ez", "port_v", "port_i", "ex", "ey", "ez", "hx",
                                          "hy", "hz")}
        return dict(out, monitors=r.monitors)
    if kind == "yee_cw":
        from gradenna_b200.fdtd3d import DFTMonitor
        from gradenna_b200.freq_adjoint3d import freq_adjoint_gradient_3d
        from gradenna_b200.ntff import directivity_3d, ntff_3d
        from gradenna_b200.sparams import s11_power_wave

        grid, freqs, margin = s["grid"], s["freqs"], s["margin"]
        th = np.linspace(0.0, np.pi, 13)
        phi = np.linspace(0.0, 2 * np.pi, 16, endpoint=False)

        def objective(ph):
            r = s11_power_wave(ph.port_v[:, 0], ph.port_i[:, 0], 50.0)
            mon = DFTMonitor(torch.tensor(freqs), ph.dft_ex, ph.dft_ey, ph.dft_ez, ph.dft_hx,
                             ph.dft_hy, ph.dft_hz)
            e = ntff_3d(mon, grid, margin, freqs, th, phi)
            d = directivity_3d(e[..., 0], e[..., 1], th, phi)
            return (r.real**2 + r.imag**2).sum() - d[:, 0, 0].mean()

        return freq_adjoint_gradient_3d(grid, objective, **s["kw"])["sigma"]
    if kind == "unet":
        return dict(zip(("loss", "theta", "x"),
                        s["net"].gradients(s["x"], s["field"], s["power"])))
    if kind == "unet_grad":
        power, grad = s["net"].power_grad(s["x"], s["weight"])
        return {"power": power, "grad": grad}
    from gradenna_b200.ntff import ntff_3d

    margin, freqs, th, phi = s["args"]
    return ntff_3d(s["mon"], s["grid"], margin, freqs, th, phi)


def work(case):
    """Bytes: inputs read once, outputs written once. Operations: the updates
    (2D: 12 a cell and step, 3D: 36), the DFT's 4 per sample and tone, the
    convolutions, the far field's 40 per point, direction and tone."""
    c, kind = case, case["kind"]
    w = 8 if c.get("f64") else 4
    if kind == "tm":
        cells = c["nx"] * c["ny"]
        return {"bytes": cells * w * (2 + 3 + 6 * c["freqs"]),
                "flops": cells * c["steps"] * (12 + 12 * c["freqs"])}
    if kind == "tm_pulse":
        cells, d = c["n"] ** 2, c["size"] ** 2
        return {"bytes": w * 2 * d, "flops": cells * c["steps"] * 24 + d * c["steps"] * 4}
    if kind == "tm_cw":
        cells, d = c["n"] ** 2, c["size"] ** 2
        return {"bytes": w * 2 * d, "flops": c["steps"] * (24 * cells + 8 * d * c["freqs"])}
    if kind == "tm_pop":
        cells = steps = 0
        flops = 0
        for p in _pop_inputs(dict(c), 0):
            d = (p["n"] // 2) ** 2
            cells += d
            flops += len(p["env"]) * (24 * p["n"] ** 2 + 8 * d * len(p["freqs"]))
        return {"bytes": 16 * cells, "flops": flops}
    if kind == "yee":
        cells = c["nx"] * c["ny"] * c["nz"]
        return {"bytes": cells * w * 8, "flops": cells * c["steps"] * 36}
    if kind == "yee_cw":
        cells = c["n"] ** 2 * c["nz"]
        return {"bytes": 16 * cells + 16 * c["size"] ** 2, "flops": cells * c["steps"] * 72}
    if kind in ("unet", "unet_grad"):
        layers, count = _unet_layers(c["base"])
        side, flops = c["side"], 0
        for name, cin, cout, taps, _, _ in layers:
            lev = 0 if name == "head" else int(name[-2] if name[-1] in "ab" else name[-1])
            lev = lev + 1 if name.startswith("up") else lev
            flops += 2 * c["batch"] * (side >> lev) ** 2 * taps * cin * cout
        px = c["batch"] * side * side
        return {"bytes": 4 * px * (4 if kind == "unet" else 2) + count * (8 if kind == "unet" else 4),
                "flops": flops * (3 if kind == "unet" else 2)}
    m = 10
    a, b, d = (c[k] - 1 - 2 * m for k in ("nx", "ny", "nz"))
    pts = 2 * (a * b + a * d + b * d)
    dirs = c["thetas"] * c["phis"]
    return {"bytes": c["freqs"] * 2 * w * (12 * pts + 2 * dirs),
            "flops": 40 * c["freqs"] * pts * dirs}


# ---------------------------------------------------------------------------
# exact: the same results in plain torch float64
# ---------------------------------------------------------------------------


def _axis64(n, d, dt, npml, half):
    """CPML tables b, c, 1/kappa of one axis (cubic grading, kappa 5, no CFS shift)."""
    pos = np.arange(n - 1) + 0.5 if half else np.arange(n, dtype=float)
    r = np.clip(np.maximum((npml - pos) / npml, (pos - (n - 1 - npml)) / npml), 0.0, 1.0)
    sig = 0.75 * 0.8 * 4.0 / (ETA0 * d) * r**3
    kap = 1.0 + 4.0 * r**3
    b = np.exp(-(sig / kap) * dt / EPS0)
    c = np.where(sig > 0.0, (b - 1.0) / kap, 0.0)
    cut = slice(None) if half else slice(1, -1)
    return [torch.as_tensor(a[cut], dtype=F64, device="cuda") for a in (b, c, 1.0 / kap)]


def _phases64(freqs, n, dt):
    t = torch.arange(n, dtype=F64, device="cuda")
    w = -2.0 * math.pi * torch.tensor(freqs, dtype=F64, device="cuda")
    return (torch.exp(1j * torch.outer((t + 1.0) * dt, w)), torch.exp(1j * torch.outer((t + 0.5) * dt, w)))


def _tm64(shape, dx, dt, npml, eps, sigma, steps, ports=(), jz=None, mx=None, my=None, probes=None,
          freqs=(), boxes=()):
    """The 2D TM loop. ports: (i, j, R, voltage or None); jz, mx, my: (flat
    cell indices, waveform (steps, m)); probes: flat Ez indices; boxes: (comp,
    lo_i, lo_j, hi_i, hi_j) whose phasors are accumulated."""
    nx, ny = shape
    dev = "cuda"
    sig = sigma
    pf = torch.tensor([i * ny + j for i, j, _, _ in ports], dtype=torch.long, device=dev)
    g = torch.tensor([1.0 / (r * dx * dx) for _, _, r, _ in ports], dtype=F64, device=dev)
    if ports:
        sig = sig.reshape(-1).index_add(0, pf, g).reshape(nx, ny)
        vs = torch.stack([torch.zeros(steps, dtype=F64, device=dev) if v is None
                          else v for _, _, _, v in ports], 1)
    h = sig * dt / (2.0 * EPS0 * eps)
    ca, cb = (1.0 - h) / (1.0 + h), (dt / (EPS0 * eps)) / (1.0 + h)
    cbf = cb.reshape(-1)
    ring = F.pad(torch.ones(nx - 2, ny - 2, dtype=F64, device=dev), (1, 1, 1, 1))
    ca, cb = ca * ring, cb * ring
    bxe, cxe, kxe = (a[:, None] for a in _axis64(nx, dx, dt, npml, False))
    bye, cye, kye = (a[None, :] for a in _axis64(ny, dx, dt, npml, False))
    bxh, cxh, kxh = (a[:, None] for a in _axis64(nx, dx, dt, npml, True))
    byh, cyh, kyh = (a[None, :] for a in _axis64(ny, dx, dt, npml, True))
    z = lambda *s: torch.zeros(s, dtype=F64, device=dev)  # noqa: E731
    ez, hx, hy = z(nx, ny), z(nx, ny - 1), z(nx - 1, ny)
    p1, p2, p3, p4 = z(nx, ny - 1), z(nx - 1, ny), z(nx - 2, ny - 2), z(nx - 2, ny - 2)
    phe, phh = _phases64(freqs, steps, dt) if freqs else (None, None)
    acc = [torch.zeros((len(freqs), b[3] - b[1], b[4] - b[2]), dtype=C128, device=dev) for b in boxes]
    pr, vo, io = [], [], []
    inv, dm = 1.0 / dx, dt / MU0

    def add(a, pts, w):
        return a.reshape(-1).index_add(0, pts, w).reshape(a.shape)

    for n in range(steps):
        d = (ez[:, 1:] - ez[:, :-1]) * inv
        p1 = byh * p1 + cyh * d
        hx = hx - dm * (d * kyh + p1)
        if mx is not None:
            hx = add(hx, mx[0], -dm * mx[1][n])
        d = (ez[1:] - ez[:-1]) * inv
        p2 = bxh * p2 + cxh * d
        hy = hy + dm * (d * kxh + p2)
        if my is not None:
            hy = add(hy, my[0], -dm * my[1][n])
        if ports:
            hyf, hxf = hy.reshape(-1), hx.reshape(-1)
            pi, pj = pf // ny, pf % ny
            hxi = pi * (ny - 1) + pj
            io.append((hyf[pf] - hyf[pf - ny]) * dx - (hxf[hxi] - hxf[hxi - 1]) * dx)
            eb = ez.reshape(-1)[pf]
        d = (hy[1:, 1:-1] - hy[:-1, 1:-1]) * inv
        p3 = bxe * p3 + cxe * d
        e = (hx[1:-1, 1:] - hx[1:-1, :-1]) * inv
        p4 = bye * p4 + cye * e
        ez = ca * ez + cb * F.pad((d * kxe + p3) - (e * kye + p4), (1, 1, 1, 1))
        if jz is not None:
            ez = add(ez, jz[0], -cbf[jz[0]] * (inv * inv) * jz[1][n])
        if ports:
            ez = add(ez, pf, -cbf[pf] * g * vs[n])
            vo.append(-0.5 * (eb + ez.reshape(-1)[pf]))
        for k, b in enumerate(boxes):
            f, ph = ((ez, phe), (hx, phh), (hy, phh))[b[0]]
            acc[k] = acc[k] + ph[n][:, None, None] * f[b[1]:b[3], b[2]:b[4]]
        if probes is not None:
            pr.append(ez.reshape(-1)[probes])
    st = lambda v: torch.stack(v) if v else None  # noqa: E731
    return dict(ez=ez, hx=hx, hy=hy, probe_ez=st(pr), port_v=st(vo), port_i=st(io),
                dft=[a * dt for a in acc])


def _box_of(box):
    il, ir, jb, jt = box
    return [(0, il, jb + 1, il + 2, jt + 1), (0, ir, jb + 1, ir + 2, jt + 1),
            (0, il + 1, jb, ir + 1, jb + 2), (0, il + 1, jt, ir + 1, jt + 2),
            (2, il, jb + 1, il + 1, jt + 1), (2, ir, jb + 1, ir + 1, jt + 1),
            (1, il + 1, jb, ir + 1, jb + 1), (1, il + 1, jt, ir + 1, jt + 1)]


def _flux64(ph, dx):
    """Radiated power per tone from the phasors of _box_of's boxes."""
    el, er, eb, et, hl, hr, hb, ht = ph
    s = lambda e, h: torch.real(0.5 * e * torch.conj(h)).flatten(1).sum(1) * 0.5 * dx  # noqa: E731
    return (s(el.sum(1, keepdim=True), hl) - s(er.sum(1, keepdim=True), hr)
            + s(et.sum(2, keepdim=True), ht) - s(eb.sum(2, keepdim=True), hb))


def _exact_tm(c, seed):
    i = _tm_inputs(c, seed)
    nx, ny = c["nx"], c["ny"]
    as32 = (lambda a: a) if c["f64"] else (lambda a: np.asarray(a, np.float32).astype(np.float64))
    to = lambda a: torch.as_tensor(as32(a), dtype=F64, device="cuda")  # noqa: E731
    flat = lambda ij: torch.tensor([a * ny + b for a, b in ij], device="cuda")  # noqa: E731
    r = _tm64((nx, ny), i["dx"], i["dt"], c["npml"], to(i["eps"]), to(i["sigma"]), c["steps"],
              ports=[(*i["port"], 50.0, to(i["vs"]))], jz=(flat([i["src"]]), to(i["cur"])[:, None]),
              probes=flat(i["probes"]), freqs=i["freqs"],
              boxes=[(0, 0, 0, nx, ny), (1, 0, 0, nx, ny - 1), (2, 0, 0, nx - 1, ny)])
    out = {k: r[k] for k in ("probe_ez", "port_v", "port_i", "ez", "hx", "hy")}
    return dict(out, **{k: a for k, a in zip(("dft_ez", "dft_hx", "dft_hy"), r["dft"])})


def _leaf(rho, f64):
    a = rho if f64 else rho.astype(np.float32).astype(np.float64)
    return torch.tensor(a, dtype=F64, device="cuda", requires_grad=True)


def _exact_pulse(c, seed):
    i = _pulse_inputs(c, seed)
    n = c["n"]
    rho = _leaf(i["rho"], c["f64"])
    pad = (c["d1"], n - c["d1"] - c["size"], c["d0"], n - c["d0"] - c["size"])
    vs = i["vs"] if c["f64"] else i["vs"].astype(np.float32)
    r = _tm64((n, n), i["dx"], i["dt"], c["npml"], torch.ones(n, n, dtype=F64, device="cuda"),
              F.pad(10.0 ** (9.0 * rho - 4.0), pad), c["steps"],
              ports=[(*i["port"], 50.0, torch.as_tensor(vs, dtype=F64, device="cuda"))],
              freqs=(i["freq"],), boxes=_box_of(i["box"]))
    loss = -_flux64(r["dft"], i["dx"])[0]
    loss.backward()
    return {"grad": rho.grad, "loss": loss.detach()}


@torch.no_grad()
def _exact_cw(c, seed):
    """Forward run, cotangents, adjoint run with CW sources, contraction."""
    i = _cw_inputs(c, seed)
    n, dx, dt, freqs = c["n"], i["dx"], i["dt"], i["freqs"]
    rho = _leaf(i["rho"], c["f64"])
    d = slice(i["d0"], i["d0"] + c["size"])
    pad = (i["d0"], n - d.stop) * 2
    sigma = F.pad(10.0 ** (9.0 * rho.detach() - 4.0), pad)
    eps = torch.ones(n, n, dtype=F64, device="cuda")
    vs = torch.as_tensor(i["vs"] if c["f64"] else i["vs"].astype(np.float32), dtype=F64, device="cuda")
    (pi, pj), (qi, qj) = i["ports"]
    design = (0, d.start, d.start, d.stop, d.stop)
    boxes = [design] + _box_of(i["box"]) + [(0, pi, pj, pi + 1, pj + 1), (2, pi - 1, pj, pi + 1, pj + 1),
                                            (1, pi, pj - 1, pi + 1, pj + 1)]
    fw = _tm64((n, n), dx, dt, c["npml"], eps, sigma, c["steps"], freqs=freqs, boxes=boxes,
               ports=[(pi, pj, 50.0, vs), (qi, qj, 50.0, None)])["dft"]
    w = 2.0 * math.pi * torch.tensor(freqs, dtype=F64, device="cuda")
    z, half = torch.exp(1j * w * dt), torch.exp(0.5j * w * dt)
    with torch.enable_grad():
        ph = [a.detach().requires_grad_(True) for a in fw[1:]]
        e, hy, hx = (a.reshape(len(freqs), -1) for a in ph[8:])
        v = -0.5 * (e[:, 0] / z + e[:, 0]) * half
        cur = (hy[:, 1] - hy[:, 0]) * dx - (hx[:, 1] - hx[:, 0]) * dx
        s11 = (v - 50.0 * cur) / (v + 50.0 * cur)
        val = _flux64(ph[:8], dx).sum() - (s11.real**2 + s11.imag**2).sum()
        cot = torch.autograd.grad(val, ph)
    env = torch.as_tensor(i["env"], dtype=F64, device="cuda")
    phe, phh = _phases64(freqs, c["steps"], dt)
    wid = (n, n - 1, n)
    src = []
    for comp, basis in ((0, -dx * dx / (dt / EPS0)), (1, (EPS0 / MU0) / (dt / MU0)), (2, (EPS0 / MU0) / (dt / MU0))):
        idx, wt = [], []
        for b, g in zip(boxes[1:], cot):
            if b[0] == comp:
                a = torch.arange(b[1], b[3], device="cuda")[:, None] * wid[comp]
                idx.append((a + torch.arange(b[2], b[4], device="cuda")).reshape(-1))
                wt.append(g.conj().reshape(len(freqs), -1) * basis)
        p = phe if comp == 0 else phh
        src.append((torch.cat(idx), torch.real(torch.conj(p) @ torch.cat(wt, 1)) * env[:, None]))
    lam = _tm64((n, n), dx, dt, c["npml"], eps, sigma, c["steps"], jz=src[0], mx=src[1], my=src[2],
                freqs=freqs, boxes=[design], ports=[(pi, pj, 50.0, None), (qi, qj, 50.0, None)])["dft"][0]
    sg = sigma[d, d]
    h = sg * dt / (2.0 * EPS0)
    ca, cb, den = (1.0 - h) / (1.0 + h), (dt / EPS0) / (1.0 + h), (1.0 + h) ** 2
    en = fw[0] / z[:, None, None]
    grad = (-dt / EPS0 / den) * en - (dt / EPS0) * (dt / (2.0 * EPS0)) / den * ((fw[0] - ca * en) / cb)
    grad = 2.0 / (float((env**2).sum()) * dt) * torch.real(torch.conj(lam) * torch.conj(grad)).sum(0) * (1.0 + h)
    return {"grad": -grad * sg * (9.0 * math.log(10.0)), "loss": -val.detach()}


@torch.no_grad()
def _exact_yee(c, seed):
    i = _yee_inputs(c, seed)
    nx, ny, nz = shape = (c["nx"], c["ny"], c["nz"])
    dx, dt, m = i["dx"], i["dt"], c["npml"]
    as32 = (lambda a: a) if c["f64"] else (lambda a: np.asarray(a, np.float32).astype(np.float64))
    to = lambda a: torch.as_tensor(as32(a), dtype=F64, device="cuda")  # noqa: E731
    eps, sig = EPS0 * to(i["eps"]), to(i["sigma"])
    h = sig * dt / (2.0 * eps)
    ca, cb = (1.0 - h) / (1.0 + h), (dt / eps) / (1.0 + h)
    tab = {}
    for ax, n in enumerate(shape):
        view = [1, 1, 1]
        view[ax] = -1
        for half in (False, True):
            tab[ax, half] = [a.reshape(view) for a in _axis64(n, dx, dt, m, half)]
    z = lambda *s: torch.zeros(s, dtype=F64, device="cuda")  # noqa: E731
    e = [z(nx - 1, ny, nz), z(nx, ny - 1, nz), z(nx, ny, nz - 1)]
    hf = [z(nx, ny - 1, nz - 1), z(nx - 1, ny, nz - 1), z(nx - 1, ny - 1, nz)]
    psi = {}

    def term(key, d, ax, half):
        b, cc, k = tab[ax, half]
        psi[key] = cc * d if key not in psi else psi[key].mul_(b).addcmul_(cc, d)
        return d * k + psi[key]

    cut = lambda a, ax: a.narrow(ax, 1, a.shape[ax] - 2)  # noqa: E731
    cur, vs = to(i["cur"]), to(i["vs"])
    p, q = i["port"], i["src"]
    ep, hp = eps[p], h[p]
    beta = dt / (2.0 * 50.0 * ep * dx)
    den = 1.0 + hp + beta
    a_p, b_p, c_p = (1.0 - hp - beta) / den, (dt / ep) / den, -dt / (50.0 * ep * dx * dx * den)
    phe, phh = _phases64(i["freqs"], c["steps"], dt)
    acc = [torch.zeros((len(i["freqs"]),) + tuple(b - a for a, b in zip(lo, hi)), dtype=C128,
                       device="cuda") for _, lo, hi in i["boxes"]]
    pr, vo, io = [], [], []
    coef = [tuple(cut(cut(x.narrow(a, 0, shape[a] - 1), (a + 1) % 3), (a + 2) % 3) for x in (ca, cb))
            for a in range(3)]
    for n in range(c["steps"]):
        for a in range(3):  # H_a += dt/mu (d_{a+2} E_{a+1} - d_{a+1} E_{a+2})
            u, v = (a + 1) % 3, (a + 2) % 3
            t = term(("h", a, v), torch.diff(e[u], dim=v) / dx, v, True)
            t = t - term(("h", a, u), torch.diff(e[v], dim=u) / dx, u, True)
            hf[a] = hf[a] + dt / MU0 * t
        io.append((hf[1][p] - hf[1][p[0] - 1, p[1], p[2]]) * dx + (hf[0][p[0], p[1] - 1, p[2]] - hf[0][p]) * dx)
        before = e[2][p].clone()
        for a in range(3):  # E_a = ca E_a + cb (d_{a+1} H_{a+2} - d_{a+2} H_{a+1})
            u, v = (a + 1) % 3, (a + 2) % 3
            t = term(("e", a, u), cut(torch.diff(hf[v], dim=u), v) / dx, u, False)
            t = t - term(("e", a, v), cut(torch.diff(hf[u], dim=v), u) / dx, v, False)
            ka, kb = coef[a]
            inner = cut(cut(e[a], u), v)
            new = e[a].clone()
            cut(cut(new, u), v).copy_(ka * inner + kb * t)
            e[a] = new
            if a == 2:
                curl = t[p[0] - 1, p[1] - 1, p[2]]
        plain = e[2][p].clone()
        e[2][q] -= cb[q] / (dx * dx) * cur[n]
        extra = e[2][p] - plain
        e[2][p] = a_p * before + b_p * curl + c_p * vs[n] + extra * (b_p / cb[p])
        vo.append(-0.5 * dx * (before + e[2][p]))
        for k, (comp, lo, hi) in enumerate(i["boxes"]):
            f = (e + hf)[comp][lo[0]:hi[0], lo[1]:hi[1], lo[2]:hi[2]]
            acc[k] += (phe if comp < 3 else phh)[n][:, None, None, None] * f
        pr.append(torch.stack([e[2][b] for b in i["probes"]]))
    out = dict(zip(("ex", "ey", "ez", "hx", "hy", "hz"), e + hf))
    return dict(out, probe_ez=torch.stack(pr), port_v=torch.stack(vo), port_i=torch.stack(io),
                monitors=[a * dt for a in acc])


def _unet64(theta, x, layers):
    by = {ly[0]: ly for ly in layers}

    def conv(name, v):
        _, cin, cout, taps, w, b = by[name]
        k = 3 if taps == 9 else 1
        wt = theta[w:w + taps * cin * cout].reshape(k, k, cin, cout).permute(3, 2, 0, 1)
        v = F.conv2d(v, wt, theta[b:b + cout], padding=k // 2)
        return v if name == "head" else F.leaky_relu(v, 0.1)

    v, skips = x[:, None], []
    for lev in range(LEVELS):
        v = conv(f"enc{lev}b", conv(f"enc{lev}a", v))
        if lev < LEVELS - 1:
            skips.append(v)
            v = F.max_pool2d(v, 2)
    for lev in range(LEVELS - 2, -1, -1):
        u = F.interpolate(conv(f"up{lev}", v), scale_factor=2, mode="nearest")
        v = conv(f"dec{lev}b", conv(f"dec{lev}a", torch.cat([skips[lev], u], 1)))
    return conv("head", v)


def _exact_unet(c, seed):
    i = _unet_inputs(c, seed)
    to = lambda a: torch.as_tensor(a, dtype=F64, device="cuda")  # noqa: E731
    layers, _ = _unet_layers(c["base"])
    theta, x = to(i["theta"]).requires_grad_(True), to(i["x"])
    out = _unet64(theta, x, layers)
    power = out[:, 2].mean(dim=(1, 2))
    # The gradient at the image has no such value: in bfloat16 some pooling
    # windows have another winner than in 64 bits, and the paths through them
    # are other paths (a quarter of its norm).
    if c["kind"] == "unet_grad":
        return {"power": power.detach(), "grad": None}
    loss = ((out[:, :2] - to(i["field"]).permute(0, 3, 1, 2)) ** 2).mean() + ((power - to(i["power"])) ** 2).mean()
    return {"loss": loss.detach(), "theta": torch.autograd.grad(loss, theta)[0], "x": None}


@torch.no_grad()
def _exact_ntff(c, seed):
    i = _ntff_inputs(c, seed)
    dx, m = i["dx"], i["margin"]
    n = (c["nx"], c["ny"], c["nz"])
    f = [torch.as_tensor(a, dtype=C128, device="cuda") for a in i["comps"]]
    lo, hi = (m, m, m), tuple(s - 1 - m for s in n)
    node = [torch.as_tensor((np.arange(s) - 0.5 * (s - 1)) * dx, dtype=F64, device="cuda") for s in n]
    pos, js, ms = [], [], []
    for a in range(3):
        u, v = (a + 1) % 3, (a + 2) % 3
        for at, s in ((hi[a], 1.0), (lo[a], -1.0)):

            def pick(comp, avg_cells, avg_node):
                """Field component on the face's cell centres: averaged over the
                two cells across the face and/or over neighbouring nodes."""
                out = 0.0
                rows = (at - 1, at) if avg_cells else (at,)
                for r in rows:
                    for k in (0, 1):
                        idx = [slice(None)] * 4
                        idx[1 + a] = slice(r, r + 1)
                        for ax in (u, v):
                            off = k if ax == avg_node else 0
                            idx[1 + ax] = slice(lo[ax] + off, hi[ax] + off)
                        out = out + f[comp][tuple(idx)]
                return (out / (2 * len(rows))).reshape(f[comp].shape[0], -1)

            # E_u lies on cell centres along u, on nodes along v; H_u on cells along a and v
            eu, ev = pick(u, False, v), pick(v, False, u)
            hu, hv = pick(3 + u, True, u), pick(3 + v, True, v)
            j, mm = [torch.zeros_like(eu)] * 3, [torch.zeros_like(eu)] * 3
            j[u], j[v] = -s * hv, s * hu
            mm[u], mm[v] = s * ev, -s * eu
            js.append(torch.stack(j, -1))
            ms.append(torch.stack(mm, -1))
            ax = [None, None, None]
            ax[a] = node[a][at:at + 1]
            for w in (u, v):
                ax[w] = node[w][lo[w]:hi[w]] + 0.5 * dx
            pos.append(torch.stack(torch.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3))
    pos, js, ms = torch.cat(pos), torch.cat(js, 1), torch.cat(ms, 1)
    th, ph = (torch.as_tensor(i[k], dtype=F64, device="cuda") for k in ("thetas", "phis"))
    tt, pp = (a.reshape(-1) for a in torch.meshgrid(th, ph, indexing="ij"))
    r = torch.stack([tt.sin() * pp.cos(), tt.sin() * pp.sin(), tt.cos()], -1)
    out = []
    for q, freq in enumerate(i["freqs"]):
        k = 2.0 * math.pi * freq / C0
        jm = torch.cat([js[q], ms[q]], -1) * (dx * dx)
        nl = torch.cat([torch.exp(1j * k * (b @ pos.T)) @ jm for b in r.split(256)])
        nv, lv = nl[:, :3], nl[:, 3:]
        theta = lambda x: (x[:, 0] * pp.cos() + x[:, 1] * pp.sin()) * tt.cos() - x[:, 2] * tt.sin()  # noqa: E731
        phi = lambda x: -x[:, 0] * pp.sin() + x[:, 1] * pp.cos()  # noqa: E731
        cf = 1j * k / (4.0 * math.pi)
        out.append(torch.stack([-cf * (phi(lv) + ETA0 * theta(nv)), cf * (theta(lv) - ETA0 * phi(nv))], -1))
    return torch.stack(out).reshape(len(i["freqs"]), len(th), len(ph), 2)


def exact(case, seed):
    kind = case["kind"]
    if kind == "tm":
        with torch.no_grad():
            return _exact_tm(case, seed)
    if kind == "tm_pulse":
        return _exact_pulse(case, seed)
    if kind == "tm_cw":
        return _exact_cw(case, seed)
    if kind == "yee":
        return _exact_yee(case, seed)
    if kind in ("unet", "unet_grad"):
        return _exact_unet(case, seed)
    if kind == "ntff":
        return _exact_ntff(case, seed)
    return None
