"""Benchmark cases of the focused-ultrasound engine, through its public entry points.

Each case is one call that a user of this package makes: a pressure solve, a heating run, a phased-array
gradient or a batch of bubbles, from host arrays to host arrays (the allocation-free heat run: device arrays).

  listed()           the named cases
  draw(rng)          one more case of the same ranges
  prepare(case, s)   the problem, made from the seed s
  run(state)         one pass
  work(case)         bytes and operations of one pass
  exact(case, s)     the outputs in 64-bit arithmetic, from plain torch
"""
import ctypes as C
import math

import numpy as np
import torch

from bubbledynamics_gb300 import abi, api, presets

_CTX = []


def _context():
    """The process's device context (a user's program keeps one for all its solves)."""
    if not _CTX:
        _CTX.append(api.Context(0))
    return _CTX[0]


# ---------------------------------------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------------------------------------
def listed():
    return [
        # one point of a parameter sweep on a small box: launches and set-up count as much as the steps
        dict(name="wv_sweep_small", kind="burst", nx=48, ny=48, nz=80, steps=400),
        # the headline benchmark: burst through a heterogeneous medium, 128 x 128 x 256, 3000 steps
        dict(name="wv_burst", kind="burst", nx=128, ny=128, nz=256, steps=3000),
        # the reference program's two-layer physics (mirror planes, Mur faces, harmonics of the absorbed
        # power) in single precision on an odd row length, as the reference's 851- and 426-cell rows are
        dict(name="wv_layers_odd", kind="layers", nx=107, ny=107, nz=401, steps=700, f64=False),
        # the same program at its own precision, the default of the command-line driver
        dict(name="wv_layers_f64", kind="layers", nx=64, ny=64, nz=201, steps=600, f64=True),
        # the acoustic half of a heating plan: water path and liver, 256 x 256 x 384
        dict(name="wv_liver", kind="liver", nx=256, ny=256, nz=384, steps=900),
        # three-tone field with nine spectra kept on the planes around the focus (drives bubble batches)
        dict(name="wv_spectrum", kind="spectrum", nx=192, ny=192, nz=288, steps=800, window=265),
        # heating of two focal spots on the liver grid, temperature and thermal dose
        dict(name="heat_liver", kind="spots", nx=256, ny=256, nz=384, steps=2000, spots=2, f64=False),
        # the reference's square-spiral scan on an odd grid, with a temperature snapshot
        dict(name="heat_spiral_odd", kind="spiral", nx=213, ny=213, nz=201, steps=900, f64=False),
        # the same scan at the reference's precision, the default of the command-line driver
        dict(name="heat_spiral_f64", kind="spiral", nx=107, ny=107, nz=126, steps=300, f64=True),
        # a few heat steps on device arrays from a control loop that may not allocate
        dict(name="heat_control_tick", kind="tick", nx=72, ny=72, nz=60, steps=12),
        # gradient of the focal loss of a 256-element array through water, fat and liver
        dict(name="adjoint_array", kind="adjoint", nx=192, ny=192, nz=192, steps=800, elements=256, every=0),
        # bubbles of a focal region over the first nanoseconds of a three-frequency drive
        dict(name="gilmore_batch", kind="bubbles", n=12000, t_ns=2.0, tones=3),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _box(rng, lo, hi, quantum, aspect):
    """nx, ny, nz of about lo..hi cells in all; sides are multiples of quantum (1: any)."""
    n = _log(rng, lo, hi)
    ny = n ** (1 / 3) * rng.uniform(0.75, 1.1)
    nx = ny * rng.uniform(0.85, 1.2)
    nz = n / (nx * ny) * aspect
    side = lambda v, least: max(least, int(round(v / quantum)) * quantum)  # noqa: E731
    return side(nx, 32), side(ny, 32), max(48, int(nz))


def _steps(rng, cells, most, lo, hi):
    """A step count of the range, with cells * steps no more than most."""
    return max(lo, min(int(_log(rng, lo, hi)), int(most / cells)))


def draw(rng):
    kind = rng.choice(["burst", "burst", "layers", "layers", "liver", "spectrum", "spots", "spiral", "tick", "adjoint",
                       "bubbles"])
    q = rng.choice([1, 1, 2, 4, 16])
    if kind == "burst":
        nx, ny, nz = _box(rng, 1.5e5, 6e6, q, 1.0)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=_steps(rng, nx * ny * nz, 1e10, 250, 2500))
    if kind == "layers":
        f64 = rng.random() < 0.5
        n = int(_log(rng, 32, 72 if f64 else 128))
        nz = int(n * rng.uniform(1.8, 3.8))
        per = rng.choice([5, 6, 7])
        return dict(kind=kind, nx=n, ny=n, nz=nz, steps=100 * per, f64=f64)
    if kind == "liver":
        nx, ny, nz = _box(rng, 4e5, 2e7, q, 1.0)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=_steps(rng, nx * ny * nz, 1.5e10, 400, 1200))
    if kind == "spectrum":
        nx, ny, nz = _box(rng, 4e5, 8e6, q, 1.0)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=_steps(rng, nx * ny * nz, 6e9, 400, 900),
                    window=rng.randrange(100, 300))
    if kind in ("spots", "spiral"):
        f64 = rng.random() < 0.3
        nx, ny, nz = _box(rng, 1e5, 1e6 if f64 else 2e7, q, 1.0)
        if kind == "spiral":
            ny = nx
        steps = _steps(rng, nx * ny * nz, 5e8 if f64 else 3e10, 100, 3000)
        case = dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=min(steps, 2000) if kind == "spiral" else steps, f64=f64)
        if kind == "spots":
            case["spots"] = rng.randrange(1, 6)
        return case
    if kind == "tick":
        nx, ny, nz = _box(rng, 1e5, 1.5e6, q, 1.0)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=rng.randrange(4, 65))
    if kind == "adjoint":
        nx, ny, nz = _box(rng, 1e5, 5e6, rng.choice([1, 4, 16]), 1.0)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=_steps(rng, nx * ny * nz, 3e9, 200, 800),
                    elements=rng.randrange(16, 257), every=rng.choice([0, 0, -1]))
    return dict(kind=kind, n=int(_log(rng, 200, 12000)), t_ns=round(rng.uniform(0.5, 2.0), 2), tones=rng.choice([1, 2, 3]))


# ---------------------------------------------------------------------------------------------------------
# problems
# ---------------------------------------------------------------------------------------------------------
def _smooth_noise(shape, sigma, seed):
    """Gaussian-correlated noise of largest magnitude 1 on the GPU (periodic)."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    w = torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32)
    F = torch.fft.rfftn(w)
    for ax, n in enumerate(shape):
        k = torch.fft.rfftfreq(n, device="cuda") if ax == 2 else torch.fft.fftfreq(n, device="cuda")
        view = [1, 1, 1]
        view[ax] = -1
        F = F * torch.exp(-2.0 * math.pi ** 2 * sigma ** 2 * k * k).reshape(view)
    g = torch.fft.irfftn(F, s=shape)
    return g / g.abs().max()


def _acoustic(case, seed):
    rng = np.random.default_rng(seed)
    nx, ny, nz, steps, kind = case["nx"], case["ny"], case["nz"], case["steps"], case["kind"]
    want = ("p_final", "peak", "energy", "Q", "dft")
    if kind == "burst":
        prob = presets.cfg1(nx, ny, nz, n_steps=steps, heterogeneity=False)
        c = 1500.0 * (1.0 + 0.02 * _smooth_noise((nz, ny, nx), 1.0e-3 / prob.grid.dx, seed))
        prob.set_c_map(c.cpu().numpy())
        prob.source.p0 *= rng.uniform(0.8, 1.2)
    elif kind == "layers":
        loop1 = steps // 100 - 4
        k = presets.ref_W_mini_constants(Nxy=nx, Nz=nz, loop1_periods=loop1, periods=4)
        s = 0.6 * nx * k["dxy"] / 0.004            # bowl and water path scaled with the box
        k["d"], k["water_tissue"] = 0.005 * s, 0.12 * nz * k["dz"] * rng.uniform(0.9, 1.1)
        k["p0"] = 2.0e5 * rng.uniform(0.8, 1.2)
        k["iz_tissue"] = next(iz for iz in range(nz) if not k["z_min"] + iz * k["dz"] < k["water_tissue"])
        prob = presets.make_ref_W(k, abi.BD_F64 if case["f64"] else abi.BD_F32)
        assert prob.params.n_steps == prob.meta["n_loop1"] + 400
        want = ("p_final", "peak", "energy", "Q")
    elif kind == "liver":
        prob = presets.cfg3_acoustic(nx, ny, nz, n_steps=steps)
        prob.source.p0 *= rng.uniform(0.8, 1.2)
        prob.source.phase[0] = rng.uniform(0.0, 2.0 * math.pi)
    else:
        prob = presets.cfg5(nx, ny, nz, n_steps=steps, window_steps=case["window"])
        prob.source.p0 *= rng.uniform(0.8, 1.2)
        for j in range(prob.source.n_tones):
            prob.source.phase[j] = rng.uniform(0.0, 2.0 * math.pi)
    return prob, want


def _heat_source(shape, rng):
    """A focal spot as a pressure solve leaves it: Gaussian, a few cells wide, longer along z [W/m^3]."""
    nz, ny, nx = shape
    q = torch.full((1, 1, 1), 1.0e7 * rng.uniform(0.5, 1.5), dtype=torch.float64, device="cuda")
    for ax, (n, s) in enumerate(((nz, 0.04 * nz), (ny, 4.0), (nx, 4.0))):
        x = torch.arange(n, dtype=torch.float64, device="cuda")
        g = torch.exp(-0.5 * ((x - n * rng.uniform(0.45, 0.55)) / (s * rng.uniform(0.9, 1.1))) ** 2)
        view = [1, 1, 1]
        view[ax] = -1
        q = q * g.reshape(view)
    return q


def _thermal(case, seed):
    rng = np.random.default_rng(seed)
    nx, ny, nz, steps = case["nx"], case["ny"], case["nz"], case["steps"]
    prec = abi.BD_F64 if case.get("f64") else abi.BD_F32
    if case["kind"] == "spots":
        # water path and perfused liver, spots of a 7 x 7 square spiral
        t = abi.Thermal()
        t.nx, t.ny, t.nz, t.precision = nx, ny, nz, prec
        t.dx, t.dz, t.dt, t.T_ref = 0.15e-3, 0.15e-3, 1e-3, 310.15
        t.n_materials, t.dose_init = 2, 0
        t.mat[0] = presets._thermal_material(1000.0, 4180.0, 0.6, 310.15)
        t.mat[1] = presets._thermal_material(1060.0, 3600.0, 0.52, 310.15, perfusion=0.0167, T_art=310.15)
        tr = abi.Trajectory()
        tr.dxy, tr.dt = t.dx, t.dt
        prob = presets.ThermalProblem("spots", t, tr)
        prob.set_plane_material([0 if iz < nz // 5 else 1 for iz in range(nz)])
        n = case["spots"]
        sx, sy = presets.square_spiral_spots(7, min(11.1, 0.03 * nx))
        at = rng.integers(0, 49 - n)
        prob.set_spots(sx[at:at + n], sy[at:at + n], [steps // n + (1 if k < steps % n else 0) for k in range(n)])
    else:
        k = presets.ref_T_mini_constants(Nxy=nx, Nz=nz, legs=13)
        k["water_tissue"] = 0.3 * nz * k["dz"] * rng.uniform(0.8, 1.2)
        prob = presets.make_ref_T(k, precision=prec)
        prob.thermal.ny = ny
    return prob, _heat_source((nz, ny, nx), rng)


def _bubbles(case, seed):
    tones = (1.0e6, 1.1e6, 1.2e6)[: case["tones"]]
    b = presets.cfg2_bubbles(case["n"], seed=seed, freqs=tones)
    return presets.cfg2_medium(), b, presets.cfg2_ode(t_end=case["t_ns"] * 1e-9)


def _array(case, seed):
    nx, ny, nz, steps = case["nx"], case["ny"], case["nz"], case["steps"]
    dx, half = 0.2e-3, 0.5 * min(nx, ny) * 0.2e-3
    sponge = 20 if min(nx, ny, nz) >= 96 else max(4, min(nx, ny, nz) // 10)
    prob, loss = presets.focal_array_problem(
        nx, ny, nz, dx, case["elements"], steps, (3 * steps // 4, steps), 0.65 * nz * dx, 0.73 * half, seed=seed % (1 << 30),
        sponge=sponge, focal_radius=max(2, nx // 48), side_radius=max(5, nx // 16))
    loss.checkpoint_every = case["every"]
    return prob, loss


def prepare(case, seed):
    ctx = _context()
    kind = case["kind"]
    if kind in ("burst", "layers", "liver", "spectrum"):
        prob, want = _acoustic(case, seed)
        return dict(kind=kind, ctx=ctx, prob=prob, want=want)
    if kind in ("spots", "spiral"):
        prob, q = _thermal(case, seed)
        return dict(kind=kind, ctx=ctx, prob=prob, Q=q.cpu().numpy(), steps=case["steps"])
    if kind == "tick":
        prob, q = _thermal(case, seed)
        T, dose = prob.initial_fields()
        th = prob.thermal
        theta = torch.from_numpy((T - th.T_ref).astype(np.float32)).cuda()
        d = torch.from_numpy(dose).cuda()
        hi = d.float()
        pair = torch.stack((hi, (d - hi.double()).float()), dim=-1).contiguous()
        sx, sy, _ = api.trajectory_shifts(prob.traj)
        at = int(np.random.default_rng(seed + 1).integers(0, len(sx) - case["steps"]))
        sh = np.stack([sx, sy], axis=1)[at:at + case["steps"]].astype(np.int32)
        return dict(kind=kind, ctx=ctx, prob=prob, theta=theta, Q=q.float().contiguous(), dose=pair,
                    shifts=np.ascontiguousarray(sh), steps=case["steps"])
    if kind == "adjoint":
        prob, loss = _array(case, seed)
        return dict(kind=kind, ctx=ctx, prob=prob, loss=loss)
    med, b, ode = _bubbles(case, seed)
    return dict(kind=kind, ctx=ctx, medium=med, bubbles=b, ode=ode)


def run(s):
    kind, ctx = s["kind"], s["ctx"]
    if kind in ("burst", "layers", "liver", "spectrum"):
        r = ctx.westervelt(s["prob"], want=s["want"])
        return {k: r[k] for k in ("p_final", "peak", "energy", "Q", "dft_re", "dft_im", "steps_done") if k in r}
    if kind == "spots":
        r = ctx.heat(s["prob"].thermal, s["Q"], s["prob"].traj)
        return {k: r[k] for k in ("T", "dose", "steps_done")}
    if kind == "spiral":
        r = ctx.heat(s["prob"].thermal, s["Q"], s["prob"].traj, max_steps=s["steps"], snapshot_legs=(1,))
        return {k: r[k] for k in ("T", "dose", "snapshots", "steps_done")}
    if kind == "tick":
        api.check(ctx.L.bd_heat_run_device_noalloc(ctx.h, C.byref(s["prob"].thermal), s["theta"].data_ptr(),
                                                   s["Q"].data_ptr(), s["dose"].data_ptr(), s["shifts"].ctypes.data,
                                                   s["steps"], None))
        return {"theta": s["theta"], "dose": s["dose"]}
    if kind == "adjoint":
        loss, gphase, gamp, _ = ctx.westervelt_adjoint(s["prob"], s["loss"])
        return {"loss": loss, "grad_phase": gphase, "grad_amp": gamp}
    r, _ = ctx.gilmore(s["medium"], s["bubbles"], s["ode"])
    return {k: np.ascontiguousarray(r[k]) for k in r.dtype.names}


def work(case):
    """Inputs read once and outputs written once; operations of every step of every cell (or bubble)."""
    kind = case["kind"]
    if kind == "bubbles":
        # about 2,000 operations an attempt; the start-up takes thousands of attempts whatever the window
        return {"bytes": case["n"] * (232 + 88), "flops": case["n"] * 2033.0 * (7000.0 + 300.0 * case["t_ns"])}
    n = case["nx"] * case["ny"] * case["nz"]
    e = 8 if case.get("f64") else 4
    if kind == "tick":
        return {"bytes": n * (8 + 4 + 16), "flops": 19.0 * n * case["steps"]}
    if kind in ("spots", "spiral"):
        snaps = 1 if kind == "spiral" else 0
        return {"bytes": n * 8 * (3 + snaps), "flops": 19.0 * n * case["steps"]}
    if kind == "adjoint":
        return {"bytes": n, "flops": (2.0 if case["every"] < 0 else 3.0) * 100.0 * n * case["steps"]}
    if kind == "burst":
        return {"bytes": 4 * n * e, "flops": 105.0 * n * case["steps"]}
    if kind == "layers":
        return {"bytes": n * (3 * e + 8), "flops": (110.0 * case["steps"] + 0.88 * 40.0 * 400) * n}
    if kind == "liver":
        return {"bytes": 3 * n * e, "flops": 115.0 * n * case["steps"]}
    planes = 2 * int(round(10e-3 * case["nz"] / 768 / 0.1e-3)) / case["nz"]
    return {"bytes": n * e * (3 + 18 * planes), "flops": (115.0 * case["steps"] + 36.0 * planes * case["window"]) * n}


# ---------------------------------------------------------------------------------------------------------
# the same outputs in 64 bits
# ---------------------------------------------------------------------------------------------------------
def _f64(x):
    return torch.as_tensor(np.asarray(x), dtype=torch.float64, device="cuda")


def _solve64(prob):
    """The Westervelt solve in float64: p_final, peak, energy, dft_re, dft_im, Q as flat layouts of run()."""
    g, m, src, p = prob.grid, prob.medium, prob.source, prob.params
    nx, ny, nz, dt = g.nx, g.ny, g.nz, g.dt
    Z = lambda: torch.zeros((nz, ny, nx), dtype=torch.float64, device="cuda")  # noqa: E731
    mirror_x, mirror_y = g.face[0] == abi.BD_FACE_MIRROR, g.face[2] == abi.BD_FACE_MIRROR
    mur = [g.face[f] == abi.BD_FACE_MUR for f in range(6)]
    L = g.mur_layers
    # media: per-plane or per-cell coefficients
    nm = m.n_materials
    if prob.array("material_map") is not None:
        idx = torch.from_numpy(prob.array("material_map").astype(np.int64)).cuda().reshape(nz, ny, nx)
    elif prob.array("plane_material") is not None:
        idx = torch.from_numpy(prob.array("plane_material").astype(np.int64)).cuda().reshape(nz, 1, 1)
    else:
        idx = torch.zeros((1, 1, 1), dtype=torch.int64, device="cuda")
    pick = lambda f: _f64([f(m.mat[k]) for k in range(nm)])[idx]  # noqa: E731
    c = _f64(prob.array("c_map")).reshape(nz, ny, nx) if prob.array("c_map") is not None else pick(lambda q: q.c0)
    kxy = c * c * (dt * dt / (g.dx * g.dx) / 180.0)
    kz = c * c * (dt * dt / (g.dz * g.dz) / 180.0)
    kd = pick(lambda q: q.delta / (2.0 * dt)) / (c * c)
    kn = pick(lambda q: 2.0 * q.beta / q.rho) / (c * c)
    kr = c * c * dt * dt
    nrel = max(m.mat[k].n_relax for k in range(nm))
    ra, rb = [], []
    for v in range(nrel):
        on = lambda q, v=v: 1.0 if v < q.n_relax else 0.0  # noqa: E731
        tau = lambda q, v=v: q.relax_tau[v] if v < q.n_relax else 1.0  # noqa: E731
        ra.append(pick(lambda q: on(q) * (4.0 * dt * q.relax_c[v] * tau(q)) / (2.0 * dt ** 3) / (2.0 * dt + 3.0 * tau(q))) / c ** 3)
        rb.append(pick(lambda q: on(q) * tau(q) / (2.0 * dt + 3.0 * tau(q))))
    semi = p.relax_scheme == abi.BD_RELAX_SEMI_IMPLICIT
    W = g.sponge_cells

    def profile(n, lo, hi):
        w = np.ones(n)
        for i in range(n):
            if W > 0 and lo == abi.BD_FACE_OPEN and i < W:
                w[i] *= math.exp(-g.sponge_strength * ((W - i) / W) ** 2)
            if W > 0 and hi == abi.BD_FACE_OPEN and i >= n - W:
                w[i] *= math.exp(-g.sponge_strength * ((i - (n - W) + 1) / W) ** 2)
        return _f64(w)

    sponge = None
    if W > 0:
        sponge = (profile(nz, g.face[4], g.face[5]).reshape(nz, 1, 1) * profile(ny, g.face[2], g.face[3]).reshape(1, ny, 1)
                  * profile(nx, g.face[0], g.face[1]).reshape(1, 1, nx))
    # source plane
    X = g.x0 + g.dx * _f64(np.arange(nx)).reshape(1, nx) - src.cx
    Y = g.y0 + g.dx * _f64(np.arange(ny)).reshape(ny, 1) - src.cy
    r = torch.sqrt(X * X + Y * Y)
    d = src.focal_length
    on = (r <= d * math.tan(src.alpha)) & (r >= d * math.tan(src.alpha_hole))
    var = torch.sqrt(1.0 + (r / d) ** 2)
    A, phi = torch.full_like(r, src.p0), torch.zeros_like(r)
    if src.kind == abi.BD_SRC_ARRAY:
        e = torch.from_numpy(prob.array("element_of_cell").astype(np.int64)).cuda().reshape(ny, nx)
        on = on & (e >= 0)
        A = A * _f64(prob.array("element_amp"))[e.clamp(min=0)]
        phi = _f64(prob.array("element_phase"))[e.clamp(min=0)]
    tau = torch.where(on, d * (var - 1.0) / src.c_delay, torch.zeros_like(r))
    A = torch.where(on, A / var, torch.zeros_like(r))
    tau_max = float(tau.max())
    ts = prob.array("t_src")

    def source(s):
        tt = (float(ts[s]) if ts is not None else p.t0 + (s + 1) * dt) + tau
        gate = 1.0
        if src.burst_cycles > 0:
            tt = tt - tau_max
            gate = ((tt >= 0) & (tt < src.burst_cycles / src.freq[0])).double()
        v = 0.0
        for k in range(src.n_tones):
            v = v + src.amp[k] * torch.sin(2 * math.pi * src.freq[k] * tt + src.phase[k] + phi)
        return A * v * gate

    zlo = src.plane_iz if mur[4] else 0
    zhi = nz - L if mur[5] else nz
    xhi, yhi = (nx - L if mur[1] else nx), (ny - L if mur[3] else ny)
    mk = lambda h: (c * (dt / h) - 1.0) / (c * (dt / h) + 1.0)  # noqa: E731
    mkx, mkz = mk(g.dx).expand(nz, ny, nx), mk(g.dz).expand(nz, ny, nx)
    P = [Z() for _ in range(5)]
    R = [[Z(), Z()] for _ in range(nrel)]
    peak, energy = Z(), Z()
    z0d, z1d = max(0, p.dft_z_lo), min(nz, p.dft_z_hi)
    dre = [Z()[z0d:z1d].clone() for _ in range(p.n_dft)]
    dim = [Z()[z0d:z1d].clone() for _ in range(p.n_dft)]
    pad = torch.zeros((nz + 6, ny + 6, nx + 6), dtype=torch.float64, device="cuda")
    body = pad[3:-3, 3:-3, 3:-3]

    def second(axis, pc):
        at = lambda o: pad[tuple(slice(3 + (o if a == axis else 0), 3 + (o if a == axis else 0) + n)  # noqa: E731
                                 for a, n in enumerate((nz, ny, nx)))]
        D = pc * -490.0
        for o, w in ((1, 270.0), (2, -27.0), (3, 2.0)):
            D.add_(at(o), alpha=w).add_(at(-o), alpha=w)
        return D

    for s in range(p.n_steps):
        p0, p1, p2, p3, p4 = P
        body.copy_(p0)
        for k in (1, 2, 3):
            if mirror_x:
                pad[:, :, 3 - k] = pad[:, :, 3 + k]
            if mirror_y:
                pad[:, 3 - k, :] = pad[:, 3 + k, :]
        D3 = 5 * p0 - 18 * p1 + 24 * p2 - 14 * p3 + 3 * p4
        s3 = 3 * p0 - 4 * p1 + p2
        V = p0 - p1 + kxy * (second(2, p0) + second(1, p0)) + kz * second(0, p0) + kd * D3
        V += kn * (0.25 * s3 * s3 + p0 * (2 * p0 - 5 * p1 + 4 * p2 - p3))
        if nrel and semi:
            E = -10 * p0 + 12 * p1 - 6 * p2 + p3
            B = [rb[v] * (4 * R[v][0] - R[v][1]) for v in range(nrel)]
            x = 3 * kr * sum(ra)
            pn = (p0 + V + kr * sum(ra[v] * E + B[v] for v in range(nrel))) / (1 - x)
            new = [ra[v] * (3 * pn + E) + B[v] for v in range(nrel)]
        else:
            new = [ra[v] * D3 + rb[v] * (4 * R[v][0] - R[v][1]) for v in range(nrel)]
            pn = p0 + V + (kr * sum(new) if nrel else 0.0)
        if sponge is not None:
            pn = pn * sponge
        F = p4                                     # cells outside the update box take their value below
        box = (slice(zlo, zhi), slice(0, yhi), slice(0, xhi))
        F[box] = pn[box]
        F[src.plane_iz] = source(s)
        for v in range(nrel):
            keep = R[v][1][src.plane_iz].clone()
            old = R[v][1]
            old[box] = new[v][box]
            old[src.plane_iz] = keep
            R[v] = [old, R[v][0]]
        if mur[4]:
            for iz in range(zlo):
                nb = p0[iz + 1] if iz + 1 < zlo else F[iz + 1]
                val = p0[iz + 1] + (nb - p0[iz]) * mkz[iz]
                F[iz, :yhi, :xhi] = val[:yhi, :xhi]
        if mur[5]:
            for iz in range(zhi, nz):
                val = p0[iz - 1] + (F[iz - 1] - p0[iz]) * mkz[iz]
                F[iz, :yhi, :xhi] = val[:yhi, :xhi]
        if mur[1]:
            for ix in range(xhi, nx):
                val = p0[:, :, ix - 1] + (F[:, :, ix - 1] - p0[:, :, ix]) * mkx[:, :, ix]
                F[:, :yhi, ix] = val[:, :yhi]
        if mur[3]:
            for iy in range(yhi, ny):
                F[:, iy] = p0[:, iy - 1] + (F[:, iy - 1] - p0[:, iy]) * mkx[:, iy]
        if p.peak_start <= s < p.peak_end:
            torch.maximum(peak, F.abs(), out=peak)
        if p.energy_start <= s < p.energy_end:
            v = (F - p1) / (2 * dt) if p.energy_mode == abi.BD_ENERGY_DPDT2 else F
            energy.addcmul_(v, v, value=dt)
        if p.n_dft and p.dft_start <= s < p.dft_start + p.dft_len:
            for j in range(p.n_dft):
                th = 2.0 * math.pi * p.dft_freq[j] * ((s - p.dft_start) * dt)
                dre[j].add_(F[z0d:z1d], alpha=math.cos(th))
                dim[j].add_(F[z0d:z1d], alpha=-math.sin(th))
        P = [F, p0, p1, p2, p3]
    out = {"p_final": P[0], "peak": peak, "energy": energy}
    if p.n_dft:
        out["dft_re"], out["dft_im"] = torch.stack(dre).reshape(-1), torch.stack(dim).reshape(-1)
    if p.q_mode == abi.BD_Q_REFERENCE:
        f = p.q_freq
        rho = pick(lambda q: q.rho)
        Q = 2.0 * pick(lambda q: q.absorption) * f * energy / ((2.0 * math.pi * f) ** 2 * rho * c)
        Q[p.q_iz_split:] = 0.0
        ha = pick(lambda q: q.harm_absorption)
        for h in range(1, min(p.q_n_harm, p.n_dft) + 1):
            a = torch.sqrt(dre[h - 1] ** 2 + dim[h - 1] ** 2) / p.dft_len
            q = Z()
            q[z0d:z1d] = a * a
            q = 2.0 * (ha * h * f / 1e6) * 2.0 * q / (rho * c)
            Q[p.q_iz_split:] += q[p.q_iz_split:]
        out["Q"] = Q
    return out


def _spiral_shifts(tr):
    """Per-step whole-cell shifts of the square spiral and the step count after each leg."""
    n_scale, n_acc = 1 + int(tr.scale / (tr.speed * tr.dt)), 1 + int(tr.t_acc / tr.dt)
    acc = (tr.speed - tr.speed_init) / tr.t_acc
    ramp = [tr.speed_init + i * tr.dt * acc for i in range(n_acc)]
    pos, near, after, cell, sign, out, legs, reach = [0.0, 0.0], [0.0, 0.0], [0.0, 0.0], [0, 0], [1, -1], [], [], 1
    for leg in range(tr.n_legs):
        a = leg % 2
        for b in (0, 1):
            after[b] = near[b] + sign[b] * tr.dxy
        hold = reach * n_scale
        for n in range(1 if leg == 0 else 0, hold + 2 * n_acc):
            v = ramp[n] if n < n_acc else tr.speed if n < hold + n_acc else ramp[hold + 2 * n_acc - n - 1]
            pos[a] += sign[a] * v * tr.dt
            if abs(after[a] - pos[a]) / tr.dxy < abs(pos[a] - near[a]) / tr.dxy:
                cell[a] += sign[a]
                near[a], after[a] = after[a], after[a] + sign[a] * tr.dxy
            out.append((cell[0], cell[1]))
        sign[1 - a] = -sign[1 - a]
        if a == 1:
            reach += 1
        legs.append(len(out))
    return out, legs


def _heat64(prob, q, shifts, snap=None):
    """Temperature (minus T_ref) and dose in float64; snap: also the temperature after that many steps."""
    t = prob.thermal
    pm = torch.from_numpy(prob._keep["plane_material"].astype(np.int64)).cuda().reshape(-1, 1, 1)
    pick = lambda f: _f64([f(t.mat[k]) for k in range(t.n_materials)])[pm]  # noqa: E731
    k = pick(lambda m: m.k_t / (m.rho * m.c_t)) * t.dt
    w = pick(lambda m: m.perfusion) * t.dt
    kxy, kz = (k / t.dx ** 2)[1:-1], (k / t.dz ** 2)[1:-1]
    a0 = 1.0 - 4.0 * kxy - 2.0 * kz - w[1:-1]
    qc = pick(lambda m: t.dt / (m.rho * m.c_t))[1:-1]
    wTa = (w * (pick(lambda m: m.T_art) - t.T_ref))[1:-1]
    T0, D0 = prob.initial_fields()
    th, dose = _f64(T0) - t.T_ref, _f64(D0)
    new, last, heat, taken = th.clone(), None, None, None
    for s, (sx, sy) in enumerate(shifts):
        if s == snap:
            taken = th.clone()
        if (sx, sy) != last:
            h = torch.zeros_like(q)
            ny, nx = q.shape[1:]
            ys, xs = slice(max(0, sy), min(ny, ny + sy)), slice(max(0, sx), min(nx, nx + sx))
            yq, xq = slice(max(0, -sy), min(ny, ny - sy)), slice(max(0, -sx), min(nx, nx - sx))
            h[:, ys, xs] = q[:, yq, xq]
            heat, last = (qc * h[1:-1, 1:-1, 1:-1] + wTa), (sx, sy)
        cc = th[1:-1, 1:-1, 1:-1]
        v = cc * a0 + kxy * (th[1:-1, 1:-1, :-2] + th[1:-1, 1:-1, 2:] + th[1:-1, :-2, 1:-1] + th[1:-1, 2:, 1:-1])
        v += kz * (th[:-2, 1:-1, 1:-1] + th[2:, 1:-1, 1:-1])
        v += heat
        new[1:-1, 1:-1, 1:-1] = v
        x = v + (t.T_ref - 273.15 - 43.0)
        dose[1:-1, 1:-1, 1:-1].add_(torch.exp2(torch.where(x < 0, 2 * x, x)), alpha=t.dt)
        th, new = new, th
    if snap == len(shifts):
        taken = th.clone()
    return th, dose, taken


# Dormand-Prince 5(4)
_A = [[], [1 / 5], [3 / 40, 9 / 40], [44 / 45, -56 / 15, 32 / 9],
      [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
      [9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656],
      [35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84]]
_E = [71 / 57600, 0, -71 / 16695, 71 / 1920, -17253 / 339200, 22 / 525, -1 / 40]
_C = [0, 1 / 5, 3 / 10, 4 / 5, 8 / 9, 1, 1]


def _bubbles64(med, b, ode):
    """The Gilmore-Zener bubbles to a tenth of the tolerance: R, Rdot, tau, q, t, R_max, R_min, t_threshold."""
    tones = int(b["n_tones"][0])
    R0 = _f64(b["R0"])
    w = [2 * math.pi * _f64(b["f"][:, k]) for k in range(tones)]
    a, ph = [_f64(b["a"][:, k]) for k in range(tones)], [_f64(b["phi"][:, k]) for k in range(tones)]
    g3, n = 3.0 * med.gamma, med.n
    rtol, atol = 0.1 * ode.rtol, 0.1 * ode.atol

    def rhs(t, R, U, T, q):
        p = sum(a[k] * torch.sin(w[k] * t + ph[k]) for k in range(tones))
        dp = sum(a[k] * w[k] * torch.cos(w[k] * t + ph[k]) for k in range(tones))
        x = R0 / R
        pin = (med.P0 + med.S2 / R0) * x ** g3
        el = -med.G4_3 * (1.0 - x * x * x) - med.mu4 * U / R
        dT = (el - T) / med.lambda_
        dq = el / (3.0 * med.lambda_) - q / med.lambda_ - U * T / R
        u, v = pin - med.S2 / R + T + med.B, med.P0 + p + med.B
        I = u / v
        Ip = I ** ((n - 1.0) / n)
        f = n / (med.rho * (n - 1.0))
        H = v * f * (Ip - 1.0)
        du = -g3 * pin * U / R + med.S2 * U / (R * R) + dT
        dH = dp * f * (Ip - 1.0) + v * f * (n - 1.0) / n * Ip / I * (du * v - u * dp) / (v * v)
        c = med.C_inf * torch.sqrt(Ip)
        m = U / c
        acc = -1.5 * U * U * (1.0 - m / 3.0) + (1.0 + m) * (H + (3.0 * q - T) / med.rho)
        acc = acc + (dH * (1.0 - m) + (3.0 * dq - dT) / med.rho) * R / c
        return U, acc / ((1.0 - m) * R), dT, dq

    zero = torch.zeros_like(R0)
    y = [R0.clone(), zero.clone(), zero.clone(), zero.clone()]
    t, h = zero.clone(), torch.full_like(R0, ode.h0)
    fac, hi, lo, hit = torch.full_like(R0, 5.0), R0.clone(), R0.clone(), torch.full_like(R0, -1.0)

    def attempt():
        live = t < ode.t_end
        hh = torch.where(live, torch.minimum(h, ode.t_end - t), zero)
        K = []
        for i in range(7):
            at = [y[c] + hh * sum((_A[i][j] * K[j][c] for j in range(i)), zero) for c in range(4)]
            K.append(rhs(t + _C[i] * hh, *at))
        err = zero
        for c in range(4):
            e = hh * sum((_E[j] * K[j][c] for j in range(7)), zero)
            err = err + (e / (atol + rtol * torch.maximum(y[c].abs(), at[c].abs()))) ** 2
        err = torch.sqrt(0.25 * err)
        grow = torch.clamp(0.9 * err.clamp(min=1e-30) ** -0.2, min=0.1)
        ok = live & (err <= 1.0)
        last = hh >= ode.t_end - t
        t.copy_(torch.where(ok, torch.where(last, torch.full_like(t, ode.t_end), t + hh), t))
        for c in range(4):
            y[c].copy_(torch.where(ok, at[c], y[c]))
        h.copy_(torch.where(live, hh * torch.minimum(torch.where(ok, fac, torch.full_like(fac, 0.9)), grow), h))
        fac.copy_(torch.where(ok, torch.full_like(fac, 5.0), torch.full_like(fac, 0.9)))
        hi.copy_(torch.maximum(hi, y[0]))
        lo.copy_(torch.minimum(lo, y[0]))
        hit.copy_(torch.where(ok & (hit < 0) & (y[1] <= -med.C_inf), t, hit))

    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        attempt()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        attempt()
    while bool((t < ode.t_end).any()):
        for _ in range(200):
            graph.replay()
    return dict(R=y[0], Rdot=y[1], tau=y[2], q=y[3], t=t, R_max=hi, R_min=lo, t_threshold=hit)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("burst", "layers", "liver", "spectrum"):
        prob, want = _acoustic(case, seed)
        r = _solve64(prob)
        return dict({k: v for k, v in r.items() if k.split("_")[0] in [x.split("_")[0] for x in want]},
                    steps_done=prob.params.n_steps)
    if kind in ("spots", "spiral"):
        prob, q = _thermal(case, seed)
        t, tr = prob.thermal, prob.traj
        if kind == "spots":
            sx, sy, st = (prob._keep[k] for k in ("spot_sx", "spot_sy", "spot_steps"))
            th, dose, _ = _heat64(prob, q, [(int(sx[k]), int(sy[k])) for k in range(len(sx)) for _ in range(int(st[k]))])
            return {"T": th + t.T_ref, "dose": dose, "steps_done": case["steps"]}
        sh, legs = _spiral_shifts(tr)
        sh = sh[: case["steps"]]
        th, dose, snap = _heat64(prob, q, sh, min(legs[0], len(sh)))
        return {"T": th + t.T_ref, "dose": dose, "snapshots": (snap + t.T_ref)[None], "steps_done": len(sh)}
    if kind == "tick":
        prob, q = _thermal(case, seed)
        sh, _ = _spiral_shifts(prob.traj)
        at = int(np.random.default_rng(seed + 1).integers(0, len(sh) - case["steps"]))
        th, dose, _ = _heat64(prob, q.float().double(), sh[at:at + case["steps"]])
        hi = dose.float().double()
        return {"theta": th, "dose": torch.stack((hi, dose - hi), dim=-1)}
    if kind == "adjoint":
        # the loss; its gradient in 64 bits would take the whole history
        prob, loss = _array(case, seed)
        E = _solve64(prob)["energy"]
        z, y, x = torch.meshgrid(*(torch.arange(n, device="cuda") for n in E.shape), indexing="ij")
        r2 = (x - loss.focus_ix) ** 2 + (y - loss.focus_iy) ** 2 + (z - loss.focus_iz) ** 2
        w = torch.zeros_like(E)
        w[(z == loss.focus_iz) & (r2 >= loss.side_radius ** 2)] = loss.side_weight
        w[r2 <= loss.focal_radius ** 2] = -1.0
        return {"loss": float((w * E).sum()), "grad_phase": None, "grad_amp": None}
    r = _bubbles64(*_bubbles(case, seed))
    return dict(r, n_accept=None, n_reject=None, status=None, threshold=None)
