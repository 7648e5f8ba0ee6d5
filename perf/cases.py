"""The workloads by which this framework's speed is measured, through its public Python entry points.

Each case is a plain dict. ``prepare`` builds, from the seed alone, what a user's program holds before the call (the model
arrays, an open handle on the GPU), ``run`` makes one pass (a shot, a batch, a gradient, an image) and returns its outputs,
``work`` counts what the pass cannot do without and ``exact`` gives the same outputs in 64 bits from plain torch and numpy.

Kinds of pass and what they stand for:

* ``rk4``       single RK4 steps launched one at a time by a program that owns its time loop (``Solver.update_rk4``);
* ``forward``   one shot: a source, the captured time loop, the receiver rows and the wavefield (``Solver.step``);
* ``batch``     several shots of one model stepped together (``Batch``);
* ``group``     models of uneven sizes stepped together (``Group``);
* ``solid``     a solid-only model, free surface or CFS-PML on all four sides (``SolidSolver``);
* ``adjoint``   the gradient of one shot's record energy (an L2 misfit against zero observations): checkpointed forward run,
                backward run, the gradient added to a device buffer as a multi-shot program does;
* ``noalloc``   steps on the caller's own device arrays (``step_noalloc``);
* ``image``     the phase-shift dispersion image of a shot gather (``dispersion_image``).
"""
import ctypes
import importlib
import math

import numpy as np
import torch

mfdm = importlib.import_module("marineseis-fdm-2d_b200")
modelgen = importlib.import_module("marineseis-fdm-2d_b200.modelgen")

H, NPD = 5.0, 20  # grid spacing (m) and CFS-PML width of every workload of this repository
FLUID, SOLID = ("fluid_vx", "fluid_vz", "fluid_p"), ("solid_vx", "solid_vz", "solid_sx", "solid_sz", "solid_sxz")
SNAPSHOT = ("fluid_vx", "fluid_vz", "solid_vx", "solid_vz")  # what the command line writes as a snapshot


def listed():
    return [
        # a program with its own time loop on a small exploratory grid: launches and latency
        {"name": "rk4_160x121", "kind": "rk4", "nx": 160, "nz": 121, "zf": 60, "bc": 2, "steps": 40, "out": "all"},
        # the flat 400x400 configuration: one shot with its receiver rows and final wavefield
        {"name": "flat_400x400", "kind": "forward", "nx": 400, "nz": 400, "zf": 203, "bc": 2, "amp": 0.0, "dt": 5e-4,
         "steps": 500, "out": "all"},
        # the curvilinear 1200x800 configuration, sinusoidal seafloor 1500 m down
        {"name": "curvilinear_1200x800", "kind": "forward", "nx": 1200, "nz": 800, "zf": 303, "bc": 2, "steps": 400, "out": "all"},
        # the headline configuration: 4096x2048, half water, half solid, with a velocity snapshot
        {"name": "curvilinear_4096x2048", "kind": "forward", "nx": 4096, "nz": 2048, "zf": 1023, "bc": 2, "steps": 256, "out": "snapshot"},
        # CFS-PML on all four sides, odd and ragged sizes
        {"name": "four_side_1001x611", "kind": "forward", "nx": 1001, "nz": 611, "zf": 251, "bc": 1, "steps": 250, "out": "all"},
        # 64 shots of the 1200x800 model in one batch
        {"name": "batch_64x1200x800", "kind": "batch", "nx": 1200, "nz": 800, "zf": 303, "bc": 2, "shots": 64, "steps": 32},
        # a survey of uneven models stepped as one group
        {"name": "group_8_uneven", "kind": "group", "models": 8, "nx_lo": 400, "nx_hi": 2000, "nz_lo": 300, "nz_hi": 1000, "steps": 96},
        # solid only with a free surface
        {"name": "solid_2048x2048", "kind": "solid", "nx": 2048, "nz": 2048, "bc": 2, "steps": 128, "out": "snapshot"},
        # a gradient on the 800x400 configuration, every segment recomputed
        {"name": "adjoint_800x400", "kind": "adjoint", "nx": 800, "nz": 400, "zf": 200, "bc": 2, "steps": 200, "every": 50},
        # a gradient on a grid that fills the GPU
        {"name": "adjoint_2048x1024", "kind": "adjoint", "nx": 2048, "nz": 1024, "zf": 303, "bc": 2, "steps": 80, "every": 20},
        # device-resident arrays stepped inside another framework's memory budget
        {"name": "noalloc_400x300", "kind": "noalloc", "nx": 400, "nz": 300, "zf": 150, "bc": 2, "steps": 100},
        # post-processing: the dispersion image of a recorded gather
        {"name": "image_2000x400", "kind": "image", "nt": 2000, "ntr": 400, "c_min": 1400.0, "c_max": 2000.0, "dc": 2.0},
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: a kind, its sizes spread over their logarithm, a step count that bounds its cost."""
    kind = rng.choice(["rk4", "forward", "forward", "forward", "batch", "group", "solid", "solid", "adjoint", "noalloc", "image"])
    if kind == "image":
        c0 = rng.uniform(300.0, 1500.0)
        return {"kind": kind, "nt": _size(rng, 256, 4000), "ntr": _size(rng, 24, 500), "c_min": round(c0, 1),
                "c_max": round(c0 * rng.uniform(1.2, 2.0), 1), "dc": rng.choice([2.0, 5.0, 10.0])}
    if kind == "group":
        lo, hi = _size(rng, 200, 500), _size(rng, 700, 1800)
        return {"kind": kind, "models": rng.randint(3, 8), "nx_lo": lo, "nx_hi": hi, "nz_lo": lo * 3 // 4, "nz_hi": hi // 2, "steps": rng.randint(33, 96)}
    top = {"rk4": 900, "forward": 4000, "batch": 1100, "solid": 2040, "adjoint": 1500, "noalloc": 480}[kind]
    nx = _size(rng, 100 if kind in ("rk4", "forward", "noalloc") else 200, top)
    nz = max(100, min(_size(rng, 0.5 * nx, nx), {"forward": 2000, "solid": 2040}.get(kind, 800)))
    if kind == "noalloc":
        nz = min(nz, 300)
    zf = int(nz * rng.uniform(0.35, 0.6))
    cells = nx * nz
    bc = 2 if kind == "noalloc" else rng.choice([2, 2, 1])
    c = {"kind": kind, "nx": nx, "nz": nz, "bc": bc}
    if kind != "solid":
        c["zf"] = zf
    if kind == "rk4":
        c.update(steps=rng.randint(10, 60), out="all")
    elif kind == "noalloc":
        c.update(steps=rng.randint(20, 200))
    elif kind in ("forward", "solid"):
        c.update(steps=max(40, min(400, int(1.5e9 / cells))), out=rng.choice(["all", "snapshot"]) if cells < 2e6 else "snapshot")
    elif kind == "batch":
        c.update(shots=rng.randint(2, 24), steps=rng.randint(33, 64))
    else:
        every = rng.choice([10, 25, 50])
        c.update(steps=max(60, min(150, int(6e7 / cells))) + rng.randint(0, 1), every=every)
    return c


# ---- inputs ----------------------------------------------------------------------------------------------------------

def _smooth_noise(rng, nz, nx, corr=10.0):
    """A smooth random field with values of about +-1 (a sum of separable waves no shorter than `corr` cells)."""
    k = 12
    kz, kx = rng.uniform(-math.pi / corr, math.pi / corr, (2, k))
    pz, px = rng.uniform(0.0, 2.0 * math.pi, (2, k))
    a = np.cos(np.arange(nz)[:, None] * kz + pz)
    b = np.cos(np.arange(nx)[:, None] * kx + px)
    return (a @ b.T) * (1.0 / math.sqrt(k))


def _limited(f):
    return np.clip(f, -2.0, 2.0) * 0.5


def _metric(nz, nx, z_xi, z_ze):
    J = (H * z_ze).astype(np.float32)
    inv = 1.0 / z_ze
    return {"J": J, "xi_x": np.full((nz, nx), 1.0 / H, np.float32), "xi_z": np.zeros((nz, nx), np.float32),
            "ze_x": (-z_xi * inv / H).astype(np.float32), "ze_z": inv.astype(np.float32)}


def _elastic(vp, vs, rho):
    mu = rho * vs * vs
    lam = rho * vp * vp - 2.0 * mu
    f = np.float32
    c11 = (lam + 2.0 * mu).astype(f)
    return {"C11": c11, "C13": lam.astype(f), "C33": c11.copy(), "C55": mu.astype(f), "rho": rho.astype(f)}


def _solid_rocks(rng, nz, nx, layers=0):
    """vp, vs, rho with +-5 % smooth perturbations, over a uniform background or flat-lying layers."""
    vp, vs, rho = (np.full((nz, 1), v) for v in (3000.0, 1732.0, 2000.0))
    if layers:
        edges = np.sort(rng.integers(1, nz, layers - 1))
        v = np.sort(rng.uniform(1900.0, 3300.0, layers))[np.searchsorted(edges, np.arange(nz), side="right")]
        vp, vs, rho = v[:, None], v[:, None] / math.sqrt(3.0), 310.0 * v[:, None] ** 0.25
    return [q * (1.0 + 0.05 * _limited(_smooth_noise(rng, nz, nx))) for q in (vp, vs, rho)]


def _fluid_solid(c, seed, layers=0):
    """Water over a solid on a curvilinear grid: modelgen.Model with float32 arrays."""
    rng = np.random.default_rng([seed, c["nx"], c["nz"]])
    nx, nz, zf, bc = c["nx"], c["nz"], c["zf"], c["bc"]
    nz_f, nz_s = zf + 1, nz - zf
    amp = c.get("amp", min(30.0, 0.15 * H * zf))
    dt, steps = c.get("dt", 4e-4), c["steps"]
    pad = NPD + 3
    x = np.clip(np.arange(nx), pad, nx - 1 - pad) - pad
    phase = rng.uniform(0.0, 2.0 * math.pi)
    k = 2.0 * math.pi * H / 600.0
    inside = (np.arange(nx) >= pad) & (np.arange(nx) < nx - pad)
    g, dg = amp * np.sin(k * x + phase), amp * k * np.cos(k * x + phase) * inside
    zeta = np.arange(nz, dtype=np.float64)
    a, b = float(pad if bc == 1 else 3), float(nz - 4 - NPD)
    t = np.clip((zeta - a) / (zf - a), 0.0, 1.0)
    w, dw = t * t * (3.0 - 2.0 * t), 6.0 * t * (1.0 - t) / (zf - a)
    s = np.clip((zeta - zf) / (b - zf), 0.0, 1.0)
    below = zeta > zf
    w = np.where(below, np.cos(0.5 * math.pi * s) ** 2, w)
    dw = np.where(below, -0.5 * math.pi / (b - zf) * np.sin(math.pi * s) * (s < 1.0), dw)
    vp, vs, rho = _solid_rocks(rng, nz_s, nx, layers)
    f, up = (30.0, 6) if c["kind"] == "adjoint" else (15.0, 10)  # peak frequency, source height over the seafloor (rows)
    vmin = min(float(vs.min()), 1500.0)
    return modelgen.Model(
        nx=nx, nz_f=nz_f, nz_s=nz_s, h=H, fpeak=f, dt=dt, nt=steps, snapshot=steps + 1,
        src_x=[int(rng.integers(pad + 5, nx - pad - 5))], src_z=[max(pad + 5 if bc == 1 else 8, zf - up)], npd=NPD, npow=2,
        thickness=(NPD - 1) * H, vp_max=float(vp.max()), rc=1e-3, beta0=max(1.0, round(vmin / (4.0 * H * f), 4)),
        fluid={"K": np.full((nz_f, nx), 1000.0 * 1500.0 ** 2, np.float32), "rho": np.full((nz_f, nx), 1000.0, np.float32)},
        solid=_elastic(vp, vs, rho), metric=_metric(nz, nx, dg[None, :] * w[:, None], H + g[None, :] * dw[:, None]),
        boundary_type=bc, pad=pad)


def _solid_only(c, seed):
    rng = np.random.default_rng([seed, c["nx"], c["nz"]])
    nx, nz, bc = c["nx"], c["nz"], c["bc"]
    pad = NPD + 3
    amp, k = 15.0 if bc == 2 else 5.0, 2.0 * math.pi * H / 600.0
    arg = k * np.arange(nx) + rng.uniform(0.0, 2.0 * math.pi)
    a, b = float(3 if bc == 2 else pad), float(nz - 4 - NPD)
    t = np.clip((np.arange(nz) - a) / (b - a), 0.0, 1.0)
    if bc == 2:
        w, dw = np.cos(0.5 * math.pi * t) ** 2, -0.5 * math.pi / (b - a) * np.sin(math.pi * t)
    else:
        w, dw = np.sin(math.pi * t) ** 2, math.pi / (b - a) * np.sin(2.0 * math.pi * t)
    dw = dw * ((t > 0.0) & (t < 1.0))
    vp, vs, rho = _solid_rocks(rng, nz, nx)
    f = 15.0
    return modelgen.SolidModel(
        nx=nx, nz=nz, h=H, fpeak=f, dt=4e-4, nt=c["steps"], snapshot=c["steps"] + 1,
        src_x=[int(rng.integers(pad + 5, nx - pad - 5))], src_z=[10 if bc == 2 else pad + 12], npd=NPD, npow=2,
        thickness=(NPD - 1) * H, vp_max=float(vp.max()), rc=1e-3, beta0=max(1.0, round(float(vs.min()) / (4.0 * H * f), 4)),
        solid=_elastic(vp, vs, rho), metric=_metric(nz, nx, amp * k * np.cos(arg)[None, :] * w[:, None],
                                                    H + amp * np.sin(arg)[None, :] * dw[:, None]), boundary_type=bc)


def _shots(c, seed, m):
    """Sources along a line, two peak frequencies (with the PML beta0 that goes with each)."""
    rng = np.random.default_rng([seed, 7])
    xs = np.linspace(m.pad + 6, m.nx - m.pad - 7, c["shots"]) + rng.integers(-2, 3, c["shots"])
    fs = [15.0 if k % 2 == 0 else 10.0 for k in range(c["shots"])]
    vmin = min(float(np.sqrt((m.solid["C55"] / m.solid["rho"]).min())), 1500.0)
    return [(int(x), m.src_z[0], f, max(1.0, round(vmin / (4.0 * H * f), 4))) for x, f in zip(xs, fs)]


def _group_sizes(c):
    """(nx, nz, zf) of the group's models: the case's own sizes, whatever the seed."""
    rng = np.random.default_rng([c["models"], c["nx_lo"], c["nx_hi"]])
    sizes = [(int(rng.integers(c["nx_lo"], c["nx_hi"] + 1)), int(rng.integers(c["nz_lo"], c["nz_hi"] + 1))) for _ in range(c["models"])]
    return [(nx, nz, int(nz * rng.uniform(0.3, 0.6))) for nx, nz in sizes]


def _group_models(c, seed):
    """Layered models (2 to 6 flat-lying solid layers) of those sizes."""
    return [_fluid_solid({"kind": c["kind"], "nx": nx, "nz": nz, "zf": zf, "bc": 2, "dt": 3e-4, "steps": c["steps"]}, seed * 16 + k,
                         layers=2 + (seed + k) % 5) for k, (nx, nz, zf) in enumerate(_group_sizes(c))]


def _gather(c, seed):
    """A gather of two dispersive arrivals and noise: [nt][ntr] float32, offsets (m), sampling rate (Hz)."""
    rng = np.random.default_rng([seed, c["nt"], c["ntr"]])
    nt, ntr, fs = c["nt"], c["ntr"], 1000.0
    x = 40.0 + 10.0 * np.arange(ntr) * (1.0 if seed % 2 else -1.0) + rng.uniform(-1.0, 1.0, ntr)
    f = np.fft.rfftfreq(nt, 1.0 / fs)
    spec = np.zeros((f.size, ntr), complex)
    for f0 in (12.0, 25.0):
        v = rng.uniform(c["c_min"], c["c_max"]) * (1.0 + 0.1 * np.exp(-f / f0))
        spec += (np.exp(-((f - f0) / f0) ** 2))[:, None] * np.exp(-2j * math.pi * f[:, None] * (np.abs(x)[None, :] / v[:, None] + 0.05))
    g = np.fft.irfft(spec, nt, axis=0)
    g = g / np.abs(g).max() + 1e-3 * rng.standard_normal((nt, ntr))
    return g.astype(np.float32), x, fs


# ---- a pass ----------------------------------------------------------------------------------------------------------

def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "image":
        return {"c": c, "gather": _gather(c, seed)}
    if kind in ("rk4", "forward"):
        return {"c": c, "s": mfdm.Solver.from_model(_fluid_solid(c, seed))}
    if kind == "solid":
        return {"c": c, "s": mfdm.SolidSolver.from_model(_solid_only(c, seed))}
    if kind == "batch":
        m = _fluid_solid(c, seed)
        return {"c": c, "s": mfdm.Batch.from_model(m, _shots(c, seed, m))}
    if kind == "group":
        ss = [mfdm.Solver.from_model(m) for m in _group_models(c, seed)]
        return {"c": c, "ss": ss, "g": mfdm.Group(ss)}
    if kind == "adjoint":
        # a handle whose operators are assembled, and the device buffer that sums the shots' gradients
        m = _fluid_solid(c, seed)
        s = mfdm.Solver.from_model(m)
        s.adjoint_forward(1, c["every"])
        rows = [m.nz_f] * 2 + [m.nz_s] * 5
        return {"c": c, "s": s, "rows": rows, "sum": torch.zeros(sum(rows), m.nx, device="cuda")}
    m = _fluid_solid(c, seed)
    dev = {k: torch.from_numpy(v).cuda() for part in (m.fluid, m.solid, m.metric) for k, v in part.items() if k != "rho"}
    dev["rho_f"], dev["rho_s"] = torch.from_numpy(m.fluid["rho"]).cuda(), torch.from_numpy(m.solid["rho"]).cuda()
    state = {"vx_f": m.nz_f, "vz_f": m.nz_f, "p_f": m.nz_f, "vx_s": m.nz_s, "vz_s": m.nz_s, "sx_s": m.nz_s, "sz_s": m.nz_s, "sxz_s": m.nz_s}
    state = {k: torch.zeros(rows, m.nx, device="cuda") for k, rows in state.items()}
    dm = mfdm.DeviceModel(nx=m.nx, nz_f=m.nz_f, nz_s=m.nz_s, fpeak=m.fpeak, dt=m.dt, npd=m.npd, npow=m.npow, thickness=m.thickness,
                          vp_max=m.vp_max, rc=m.rc, beta0=m.beta0, src_x=m.src_x[0], src_z=m.src_z[0],
                          **{k: ctypes.c_void_p(v.data_ptr()) for part in (dev, state) for k, v in part.items()})
    return {"c": c, "dm": dm, "dev": dev, "state": state}


def run(state):
    c = state["c"]
    kind = c["kind"]
    if kind == "image":
        g, x, fs = state["gather"]
        return mfdm.dispersion_image(g, x, fs, c["c_min"], c["c_max"], c["dc"])
    if kind == "noalloc":
        for v in state["state"].values():
            v.zero_()
        mfdm.step_noalloc(state["dm"], 0, c["steps"], torch.cuda.current_stream().cuda_stream)
        return state["state"]
    if kind == "group":
        for s in state["ss"]:
            s.set_shot(0)
        state["g"].step(c["steps"])
        return [s.records() for s in state["ss"]]
    s = state["s"]
    if kind == "batch":
        s.reset()
        s.step(c["steps"])
        recs = [s.records(shot=k) for k in range(c["shots"])]
        return {q: np.stack([r[q] for r in recs]) for q in recs[0]}
    if kind == "adjoint":
        rec = s.adjoint_forward(c["steps"], c["every"])
        s.adjoint_backward_only(rec)
        state["sum"].zero_()
        s.adjoint_accumulate_grad(state["sum"], torch.cuda.current_stream().cuda_stream)
        return {"rec": rec, "grad": dict(zip(mfdm.GRAD_COEFS, state["sum"].split(state["rows"])))}
    s.set_shot(0)
    if kind == "rk4":
        for it in range(c["steps"]):
            s.update_rk4(it)
        s.synchronize()
    else:
        s.step(c["steps"])
    names = (FLUID if kind != "solid" else ()) + SOLID if c["out"] == "all" else SNAPSHOT if kind != "solid" else SNAPSHOT[2:]
    return {"rec": s.records(), "field": {n: s.field(n) for n in names}}


def work(case):
    """The coefficients read once, the state written once, the records, and the arithmetic of every step."""
    c = case
    if c["kind"] == "image":
        nt, ntr, nf = c["nt"], c["ntr"], c["nt"] // 2 + 1
        nv = math.ceil((c["c_max"] + c["dc"] / 2 - c["c_min"]) / c["dc"])
        return {"bytes": 4 * nt * ntr + 8 * ntr + 4 * nf * nv + 8 * (nf + nv), "flops": 2.5 * nt * math.log2(nt) * ntr + 8 * nf * nv * ntr}
    if c["kind"] == "group":
        sizes = [(nx, zf + 1, nz - zf) for nx, nz, zf in _group_sizes(c)]
    elif c["kind"] == "solid":
        sizes = [(c["nx"], 0, c["nz"])]
    else:
        sizes = [(c["nx"], c["zf"] + 1, c["nz"] - c["zf"])]
    passes, shots = (4 if c["kind"] == "adjoint" else 1), c.get("shots", 1)  # a gradient: forward, recompute and a reverse of two
    b = sum(nx * (4 * (6 * f + 9 * s) + shots * 4 * (3 * f + 5 * s) + shots * 4 * c["steps"]) for nx, f, s in sizes)
    fl = sum(nx * (260.0 * f + 580.0 * s) for nx, f, s in sizes) * c["steps"] * shots * passes
    if c["kind"] == "adjoint":
        b += 4 * sum(nx * (2 * f + 5 * s) for nx, f, s in sizes)
    return {"bytes": b, "flops": fl}


# ---- the same outputs in 64 bits ---------------------------------------------------------------------------------------

A5 = [float(np.float32(v)) for v in (-0.30874, -0.63260, 1.23300, -0.33340, 0.04168)]  # biased 5-point operator, taps -1 .. 3
M42 = [float(np.float32(-7.0 / 6.0)), float(np.float32(8.0 / 6.0)), float(np.float32(-2.0 / 12.0))]
W5 = [0.0030, 0.0133, 0.0219, 0.0133, 0.0030, 0.0133, 0.0596, 0.0983, 0.0596, 0.0133, 0.0219, 0.0983, 0.1621, 0.0983, 0.0219,
      0.0133, 0.0596, 0.0983, 0.0596, 0.0133, 0.0030, 0.0133, 0.0219, 0.0133, 0.0030]
W7 = [1.1e-13, 1.678e-06, 0.03419, 0.93163, 0.03419, 1.678e-06, 1.1e-13]
F, B = 0, 1


def _f32(v):
    return float(np.float32(v))


def _taps(d):
    return [(k if d == F else -k, a if d == F else -a) for k, a in zip(range(-1, 4), A5)]


def _dx(f, d):
    """Biased derivative along x at columns 3 .. nx-4."""
    n = f.shape[-1] - 6
    return sum(a * f[..., 3 + k:3 + k + n] for k, a in _taps(d))


def _dz(f, d, r0, r1):
    """Biased derivative along z at rows r0 .. r1-1 (full order), columns 3 .. nx-4."""
    g = f[..., 3:-3]
    return sum(a * g[..., r0 + k:r1 + k, :] for k, a in _taps(d))


def _dz_low(f, d, r, dist, solid_side):
    """One row near a boundary `dist` rows away."""
    g = f[..., 3:-3]
    if dist == 2:
        s = 1 if d == F else -1
        return s * sum(w * g[..., r + s * k:r + s * k + 1, :] for k, w in enumerate(M42))
    forward = d == F if dist == 1 else solid_side
    return g[..., r + 1:r + 2, :] - g[..., r:r + 1, :] if forward else g[..., r:r + 1, :] - g[..., r - 1:r, :]


def _ricker(f, t):
    T = 1.2 / f
    q = (math.pi * f * (t - T)) ** 2
    return 0.0 if t - T > T else (1.0 - 2.0 * q) * math.exp(-q)


def _pml(m, f, beta0, n, lo, hi, dev):
    """d/beta, alpha + d/beta, 1/beta of every cell of an axis."""
    npd, npow = m.npd, m.npow
    d0 = -(npow + 1) * _f32(m.vp_max) * math.log(_f32(m.rc)) / (2.0 * _f32(m.thickness))
    i = np.arange(n)
    k = np.zeros(n)
    if hi:
        k = np.where((i >= n - 3 - npd) & (i <= n - 4), i - (n - 4 - npd), k)
    if lo:
        k = np.where((i >= 3) & (i <= 2 + npd), 3 + npd - i, k)
    r = k / npd
    be = 1.0 + (_f32(beta0) - 1.0) * r * r
    dpb = d0 * r ** npow / be
    return [torch.tensor(v, dtype=torch.float64, device=dev) for v in (dpb, 2.0 * math.pi * f * (1.0 - r) + dpb, 1.0 / be)]


class _Exact:
    """The time step in 64 bits on full arrays: state (fields, strip memory) in, state out, nothing in place (autograd passes through)."""

    def __init__(self, m, dev, solid_only=False, shot=None):
        self.m, self.dev, self.solid_only = m, dev, solid_only
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float32)).to(dev).double()  # noqa: E731
        self.cpml = m.boundary_type == 1
        self.nx, self.npd = m.nx, m.npd
        self.nzf, self.nzs = (0, m.nz) if solid_only else (m.nz_f, m.nz_s)
        sx, sz, f, beta0 = shot if shot else (m.src_x[0], m.src_z[0], m.fpeak, m.beta0)
        self.f, self.dt, self.src = _f32(f), _f32(m.dt), (sx, sz)
        self.gap = max(1, int(1e-3 / self.dt + 0.5))
        M = [t(m.metric[k]) for k in ("xi_x", "xi_z", "ze_x", "ze_z")]
        J = t(m.metric["J"])
        self.par = {k: t(m.solid[k]) for k in ("C11", "C13", "C33", "C55")}
        self.par["rcp_rho_s"] = 1.0 / t(m.solid["rho"])
        npd, nx = self.npd, self.nx
        cols = list(range(npd)) + list(range(nx - 6 - npd, nx - 6))  # side-strip columns among 3 .. nx-4
        self.side = torch.tensor(cols, device=dev)
        self.px = [v[3:-3][self.side] for v in _pml(m, self.f, beta0, nx, True, True, dev)]
        c = slice(3, -3)
        if not solid_only:
            z0 = self.nzf - 1
            self.par["K"], self.par["rcp_rho_f"] = t(m.fluid["K"]), 1.0 / t(m.fluid["rho"])
            self.Mf, self.Jf = [q[:self.nzf] for q in M], J[:self.nzf]
            self.Ms, self.Js = [q[z0:] for q in M], J[z0:]
            self.Mb = [q[:self.nzs] for q in M] if self.cpml else self.Ms  # the four-side sxz line's metric rows
            n = torch.stack([self.Mf[2][z0, c], self.Mf[3][z0, c]])
            self.n = n / n.norm(dim=0)
            if self.cpml:
                self.pzf = [v[3:3 + npd, None] for v in _pml(m, self.f, beta0, self.nzf, True, False, dev)]
            w = torch.tensor([float(np.float32(v)) for v in W7], dtype=torch.float64, device=dev)
            one = torch.ones(nx - 6, dtype=torch.float64, device=dev)
            self.w7, self.wsum = w, self._smooth(one, w)
        else:
            self.Ms, self.Js = M, J
            self.Mb = M
            if not self.cpml:
                self.alm = self._alm()
        self.zb0 = self.nzs - 3 - npd
        self.pz = [v[:, None] for v in _pml(m, self.f, beta0, self.nzs, solid_only and self.cpml, True, dev)]
        self.w5 = torch.tensor([float(np.float32(v)) for v in W5], dtype=torch.float64, device=dev).reshape(5, 5)

    def _smooth(self, v, w):
        p = torch.nn.functional.pad(v, (3, 3))
        n = v.shape[-1]
        return sum(w[k] * p[..., k:k + n] for k in range(7))

    def _alm(self):
        """Elimination of the zeta derivatives on the traction-free row."""
        c11, c13, c33, c55 = (self.par[k][3, 3:-3] for k in ("C11", "C13", "C33", "C55"))
        xx, xz, zx, zz = (q[3, 3:-3] for q in self.Ms)
        # traction (sx zx + sxz zz, sxz zx + sz zz) = Dz v_zeta + Dx v_xi = 0, so v_zeta = -M v_xi
        Dz = torch.stack([torch.stack([c11 * zx * zx + c55 * zz * zz, (c13 + c55) * zx * zz]),
                          torch.stack([(c13 + c55) * zx * zz, c55 * zx * zx + c33 * zz * zz])]).permute(2, 0, 1)
        Dx = torch.stack([torch.stack([c11 * zx * xx + c55 * zz * xz, c13 * zx * xz + c55 * zz * xx]),
                          torch.stack([c13 * zz * xx + c55 * zx * xz, c55 * zx * xx + c33 * zz * xz])]).permute(2, 0, 1)
        Q = torch.linalg.solve(Dz, Dx)
        m11, m12, m21, m22 = Q[:, 0, 0], Q[:, 0, 1], Q[:, 1, 0], Q[:, 1, 1]
        return [xx - zx * m11, -zz * m21, xz - zz * m11 - zx * m21, -zx * m12, xz - zz * m22, xx - zz * m12 - zx * m22]

    def rest(self):
        z = lambda *s: torch.zeros(*s, dtype=torch.float64, device=self.dev)  # noqa: E731
        ns, npd = self.nzs, self.npd
        S = {"s": z(5, ns, self.nx), "sx": z(4, ns, 2 * npd), "sz": z(4, 2 * npd if self.solid_only and self.cpml else npd, self.nx - 6)}
        if not self.solid_only:
            S["f"], S["fx"] = z(3, self.nzf, self.nx), z(4, self.nzf, 2 * npd)
            if self.cpml:
                S["fz"] = z(4, npd, self.nx - 6)
        return S

    # rates of the solid: rows lo .. nzs-4, columns 3 .. nx-4
    def _solid(self, S, d, lo):
        par, npd, nz, c = self.par, self.npd, self.nzs, slice(3, -3)
        U, hi = S["s"], self.nzs - 3
        q = lambda a: a[lo:hi, c]  # noqa: E731
        xx, xz, zx, zz = (q(a) for a in self.Ms)
        free = self.solid_only and not self.cpml  # free surface on row 3
        near = 0 if self.solid_only and self.cpml else 3  # rows with lower-order operators
        T = U[2:5]
        full = lo + near
        Tx = _dx(T[:, lo:hi], d)
        Tz = _dz(T, d, full, hi)
        if near:
            low = [_dz_low(T, d, lo + k, k, True) for k in range(near)] if free else [torch.zeros_like(Tz[:, :1])] * near
            Tz = torch.cat(low + [Tz], 1)
        rvx = xx * Tx[0] + zx * Tz[0] + xz * Tx[2] + zz * Tz[2]
        rvz = xx * Tx[2] + zx * Tz[2] + xz * Tx[1] + zz * Tz[1]
        gxx, gzz, gxz = xx * xx + xz * xz, zx * zx + zz * zz, xx * zx + xz * zz
        R = gxz / gxx
        dxx = xx * (Tx[0] + R * Tz[0]) + xz * (Tx[2] + R * Tz[2])
        dxz = xx * (Tx[2] + R * Tz[2]) + xz * (Tx[1] + R * Tz[1])
        if near:
            # flux form of the first rows, ghosts mirrored through the surface or the interface
            e = lo + 6
            Js, (ax, az, bx, bz) = self.Js[lo:e], [a[lo:e] for a in self.Ms]
            sx, sz, t = (T[k][lo:e] for k in range(3))
            Fx = torch.stack([Js * (ax * sx + az * t), Js * (ax * t + az * sz)])
            Fz = torch.stack([Js * (bx * sx + bz * t), Js * (bx * t + bz * sz)])
            mirror = Fz[:, 1:4].flip(1)
            ghost = -mirror if free else 2.0 * Fz[:, :1] - mirror
            G = torch.cat([ghost, Fz], 1)
            Sx = (_dx(Fx[:, :near], d) + _dz(G, d, 3, 3 + near)) / self.Js[lo:lo + near, c]
            rvx, rvz = torch.cat([Sx[0], rvx[near:]]), torch.cat([Sx[1], rvz[near:]])
            if not free:
                P, n = xx[:near] * Sx[0] + xz[:near] * Sx[1], gxx[:near]
                dxx, dxz = torch.cat([xx[:near] * P / n, dxx[near:]]), torch.cat([xz[:near] * P / n, dxz[near:]])
        vx, vz = rvx, rvz
        V = U[0:2]
        Vx = _dx(V[:, lo:hi], d)
        Vz = torch.cat([_dz_low(V, d, lo + k, k, True) for k in range(near)] + [_dz(V, d, full, hi)], 1)
        c11, c13, c33, c55 = (q(par[k]) for k in ("C11", "C13", "C33", "C55"))
        yx, yz, wx, wz = (q(a) for a in self.Mb)
        X, Z = xx * Vx[0] + zx * Vz[0], xz * Vx[1] + zz * Vz[1]
        Y = yz * Vx[0] + wz * Vz[0] + yx * Vx[1] + wx * Vz[1]
        # side strips: derivatives replaced by (1/beta) D - (1/beta) memory
        s = self.side
        dpb, ap, ib = self.px
        A = S["sx"][:, lo:hi]
        D = torch.stack([dxx[:, s], dxz[:, s], (Vx[0] + R * Vz[0])[:, s], (Vx[1] + R * Vz[1])[:, s]])
        if free:
            # on the surface row the strips act on the xi derivatives alone
            D = torch.cat([D[:, :1].clone().index_copy(0, torch.tensor([2, 3], device=self.dev), Vx[:, :1][:, :, s]), D[:, 1:]], 1)
        kx = -ap * A + dpb * D
        E = (ib - 1.0) * D - ib * A
        add = lambda a, v: a.index_add(1, s, v)  # noqa: E731
        vx, vz = add(vx, E[0]), add(vz, E[1])
        X, Z = add(X, xx[:, s] * E[2]), add(Z, xz[:, s] * E[3])
        Y = add(Y, xz[:, s] * E[2] + xx[:, s] * E[3])
        # zeta bands
        S_ = gxz / gzz
        bands = [(self.zb0, hi, 0)] + ([(3, 3 + npd, npd)] if self.solid_only and self.cpml else [])
        kz = []
        for r0, r1, o in bands:
            i = slice(r0 - lo, r1 - lo)
            dpb, ap, ib = (v[r0:r1] for v in self.pz)
            A = S["sz"][:, o:o + npd]
            b, g, k = S_[i], zx[i], zz[i]
            D = torch.stack([g * (Tz[0][i] + b * Tx[0][i]) + k * (Tz[2][i] + b * Tx[2][i]),
                             g * (Tz[2][i] + b * Tx[2][i]) + k * (Tz[1][i] + b * Tx[1][i]),
                             Vz[0][i] + b * Vx[0][i], Vz[1][i] + b * Vx[1][i]])
            kz.append(-ap * A + dpb * D)
            E = (ib - 1.0) * D - ib * A
            put = lambda a, v: torch.cat([a[:i.start], a[i] + v, a[i.stop:]])  # noqa: E731
            vx, vz, X, Z = put(vx, E[0]), put(vz, E[1]), put(X, g * E[2]), put(Z, k * E[3])
            Y = put(Y, k * E[2] + g * E[3])
        ir = q(par["rcp_rho_s"])
        K = [vx * ir, vz * ir, c11 * X + c13 * Z, c13 * X + c33 * Z, c55 * Y]
        if free:
            # traction-free row; its strip terms scale the same derivatives
            a0, a1, a2, a3, a4, a5 = self.alm
            e0, e1 = Vx[0, 0], Vx[1, 0]
            dpb, ap, ib = self.px
            A = S["sx"][2:4, lo]
            e0, e1 = (e.index_add(0, s, (ib - 1.0) * e[s] - ib * a) for e, a in ((e0, A[0]), (e1, A[1])))
            h = [v[0] for v in (c11, c13, c33, c55)]
            top = [(h[0] * a0 + h[1] * a1) * e0 + (h[0] * a3 + h[1] * a4) * e1, (h[1] * a0 + h[2] * a1) * e0 + (h[1] * a3 + h[2] * a4) * e1,
                   h[3] * (a2 * e0 + a5 * e1)]
            K[2:] = [torch.cat([r[None], k[1:]]) for r, k in zip(top, K[2:])]
        return torch.stack(K), kx, torch.cat(kz, 1)

    # rates of the fluid: rows 3 .. nzf-1, columns 3 .. nx-4
    def _fluid(self, S, d):
        par, c, n, npd = self.par, slice(3, -3), self.nzf, self.npd
        U = S["f"]
        q = lambda a: a[3:, c]  # noqa: E731
        xx, xz, zx, zz = (q(a) for a in self.Mf)
        gxx, gzz, gxz = xx * xx + xz * xz, zx * zx + zz * zz, xx * zx + xz * zz
        p = U[2]
        first = 0 if self.cpml else 3  # flux-form rows under the free surface
        px, mid = _dx(p[3:], d), _dz(p, d, 3 + first, n - 3)
        pz = torch.cat([torch.zeros_like(mid[:1])] * first + [mid] + [torch.zeros_like(mid[:1])] * 3)
        rvx, rvz = -(xx * px + zx * pz), -(xz * px + zz * pz)
        Fx = torch.stack([-self.Jf * self.Mf[0] * p, -self.Jf * self.Mf[1] * p])
        Fz = torch.stack([-self.Jf * self.Mf[2] * p, -self.Jf * self.Mf[3] * p])
        bot = torch.cat([Fz[:, n - 6:], 2.0 * Fz[:, n - 1:] - Fz[:, n - 4:n - 1].flip(1)], 1)
        rows = [(n - 3, _dx(Fx[:, n - 3:], d) + _dz(bot, d, 3, 6))]
        if first:
            top = torch.cat([-Fz[:, 4:7].flip(1), Fz[:, 3:9]], 1)
            rows.append((3, _dx(Fx[:, 3:6], d) + _dz(top, d, 3, 6)))
        for r, f in rows:
            f = f / self.Jf[r:r + 3, c]
            i = r - 3
            rvx, rvz = (torch.cat([a[:i], b, a[i + 3:]]) for a, b in ((rvx, f[0]), (rvz, f[1])))
        V = U[0:2]
        Vx = _dx(V[:, 3:], d)
        low = [_dz_low(V, d, r, dist, False) for r, dist in ((n - 3, 2), (n - 2, 1), (n - 1, 0))]
        head = [] if self.cpml else [torch.zeros_like(Vx[:, :1])] + [_dz_low(V, d, r, r - 3, False) for r in (4, 5)]
        Vz = torch.cat(head + [_dz(V, d, 3 + first, n - 3)] + low, 1)
        div = xx * Vx[0] + zx * Vz[0] + xz * Vx[1] + zz * Vz[1]
        s = self.side
        dpb, ap, ib = self.px
        A = S["fx"][:, 3:]
        R = gxz / gxx
        # projections of the momentum rate on grad(xi), of grad(zeta)
        P = (xx * rvx + xz * rvz) / gxx
        D = torch.stack([(xx * P)[:, s], (xz * P)[:, s], (Vx[0] + R * Vz[0])[:, s], (Vx[1] + R * Vz[1])[:, s]])
        kx = -ap * A + dpb * D
        E = (ib - 1.0) * D - ib * A
        vx, vz = rvx.index_add(1, s, E[0]), rvz.index_add(1, s, E[1])
        div = div.index_add(1, s, xx[:, s] * E[2] + xz[:, s] * E[3])
        kz = None
        if self.cpml:
            i = slice(0, npd)
            dpb, ap, ib = self.pzf
            A = S["fz"]
            Q, b = (zx * rvx + zz * rvz)[i] / gzz[i], (gxz / gzz)[i]
            D = torch.stack([zx[i] * Q, zz[i] * Q, Vz[0][i] + b * Vx[0][i], Vz[1][i] + b * Vx[1][i]])
            kz = -ap * A + dpb * D
            E = (ib - 1.0) * D - ib * A
            put = lambda a, v: torch.cat([a[i] + v, a[npd:]])  # noqa: E731
            vx, vz, div = put(vx, E[0]), put(vz, E[1]), put(div, zx[i] * E[2] + zz[i] * E[3])
        else:
            # the surface row holds p and its strip memory of the velocities
            kx = torch.cat([torch.cat([kx[:2, :1], torch.zeros_like(kx[2:, :1])]), kx[:, 1:]], 1)
            div = torch.cat([torch.zeros_like(div[:1]), div[1:]])
        ir = q(par["rcp_rho_f"])
        return torch.stack([vx * ir, vz * ir, -q(par["K"]) * div]), kx, kz

    def _source(self, K, row, amp):
        """The 5x5 spread source into rate K[row] (rows from 3, columns from 3)."""
        if amp == 0.0:
            return K
        sx, sz = self.src
        add = torch.zeros_like(K)
        last = K.shape[1] - (0 if self.solid_only else 3)  # not within three rows of the interface
        for i in range(5):
            for j in range(5):
                z, x = sz - 2 + i - 3, sx - 2 + j - 3
                if 0 <= z < last and 0 <= x < K.shape[2]:
                    for k in row:
                        add[k, z, x] = amp * self.w5[i, j]
        return K + add

    def rate(self, S, d, amp):
        pad = torch.nn.functional.pad
        out = {}
        lo = 3 if self.solid_only else 0
        ks, sx, sz = self._solid(S, d, lo)
        if self.solid_only:
            ks = self._source(ks, (2, 3), amp)
        else:
            kf, fx, fz = self._fluid(S, d)
            kf = self._source(kf, (2,), amp)
            # coupling of the interface row: F takes the solid's normal velocity and traction, B the fluid's
            a, b = self.n
            f, s = kf[:, -1], ks[:, 0]
            vnf, vtf, vns, vts = a * f[0] + b * f[1], b * f[0] - a * f[1], a * s[0] + b * s[1], b * s[0] - a * s[1]
            snn = a * a * s[2] + 2 * a * b * s[4] + b * b * s[3]
            snt = 0.0
            stt = b * b * s[2] - 2 * a * b * s[4] + a * a * s[3]
            pf = f[2]
            if d == F:
                vnf, pf = vns, -snn
            else:
                vns, snn = vnf, -pf
            fi = torch.stack([a * vnf + b * vtf, b * vnf - a * vtf, pf])
            si = torch.stack([a * vns + b * vts, b * vns - a * vts, a * a * snn + b * b * stt, b * b * snn + a * a * stt,
                              -a * b * stt + (b * b - a * a) * snt])
            kf = torch.cat([kf[:, :-1], fi[:, None]], 1)
            ks = torch.cat([si[:, None], ks[:, 1:]], 1)
            out["f"], out["fx"] = pad(kf, (3, 3, 3, 0)), pad(fx, (0, 0, 3, 0))
            if fz is not None:
                out["fz"] = fz
        out["s"], out["sx"], out["sz"] = pad(ks, (3, 3, lo, 3)), pad(sx, (0, 0, lo, 3)), sz
        return out

    def step(self, U, it):
        d, dt, t = it % 2, self.dt, it * self.dt
        dirs = (d, 1 - d, d, 1 - d)
        amps = [_ricker(self.f, t + h * dt) for h in (0.0, 0.5, 0.5, 1.0)]
        Y, acc = U, U
        for k in range(4):
            r = self.rate(Y, dirs[k], amps[k])
            acc = {q: acc[q] + (dt / (6.0, 3.0, 3.0, 6.0)[k]) * r[q] for q in U}
            if k < 3:
                Y = {q: U[q] + (0.5 * dt, 0.5 * dt, dt)[k] * r[q] for q in U}
        return acc if self.solid_only else self._filter(acc)

    def _filter(self, U):
        """The interface smoothing and the continuity average."""
        c, z0 = slice(3, -3), self.nzf - 1
        v = self._smooth(torch.cat([U["f"][:, z0, c], U["s"][:, 0, c]]), self.w7) / self.wsum
        a, b = self.n
        vnf, vtf, vns, vts = a * v[0] + b * v[1], b * v[0] - a * v[1], a * v[3] + b * v[4], b * v[3] - a * v[4]
        snn = a * a * v[5] + 2 * a * b * v[7] + b * b * v[6]
        stt = b * b * v[5] - 2 * a * b * v[7] + a * a * v[6]
        vn, sn = 0.5 * (vnf + vns), 0.5 * (snn - v[2])
        f = torch.stack([a * vn + b * vtf, b * vn - a * vtf, -sn])
        s = torch.stack([a * vn + b * vts, b * vn - a * vts, a * a * sn + b * b * stt, b * b * sn + a * a * stt, a * b * (sn - stt)])
        pad = torch.nn.functional.pad
        return {**U, "f": torch.cat([U["f"][:, :z0], pad(f, (3, 3))[:, None]], 1), "s": torch.cat([pad(s, (3, 3))[:, None], U["s"][:, 1:]], 1)}

    def sample(self, U):
        if self.solid_only:
            return {"svz": U["s"][1, 30 if self.cpml else 3]}
        keep = torch.zeros(self.nx, dtype=torch.float64, device=self.dev)
        keep[3:-3] = 1.0
        return {"svx": U["s"][0, 0] * keep, "svz": U["s"][1, 0] * keep, "fp": U["f"][2, self.nzf - 1] * keep}

    def forward(self, steps, run=None):
        """Records and the final state; `run` wraps a step (checkpointing)."""
        U, rec = self.rest(), []
        for it in range(steps):
            U = run(self.step, U, it) if run else self.step(U, it)
            if it % self.gap == 0:
                rec.append(self.sample(U))
        return {k: torch.stack([r[k] for r in rec]) for k in rec[0]}, U


def _gradient(c, seed, dev):
    """The gradient of the record energy by reverse-mode differentiation of the 64-bit step."""
    from torch.utils.checkpoint import checkpoint
    e = _Exact(_fluid_solid(c, seed), dev)
    names = ("K", "rcp_rho_f", "C11", "C13", "C33", "C55", "rcp_rho_s")
    for k in names:
        e.par[k].requires_grad_(True)
    rec, _ = e.forward(c["steps"], lambda f, U, it: checkpoint(f, U, it, use_reentrant=False, preserve_rng_state=False))
    sum((rec[k] ** 2).sum() for k in rec).mul(0.5).backward()
    return {"rec": {k: v.detach() for k, v in rec.items()}, "grad": {k: e.par[k].grad for k in names}}


def _image(c, seed):
    g, x, fs = _gather(c, seed)
    nt = g.shape[0]
    S = np.fft.rfft(g.astype(np.float64), axis=0)
    mag = np.abs(S)
    P = np.where(mag > 0.0, np.conj(S) / np.where(mag > 0.0, mag, 1.0), 0.0)
    nv = math.ceil((c["c_max"] + c["dc"] / 2 - c["c_min"]) / c["dc"])
    vel = c["c_min"] + c["dc"] * np.arange(nv)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    Pt, xt, vt = torch.from_numpy(P).to(dev), torch.from_numpy(x).to(dev), torch.from_numpy(vel).to(dev)
    A = torch.empty(P.shape[0], nv, dtype=torch.float64, device=dev)
    for k in range(P.shape[0]):
        ph = (2.0 * math.pi * k * fs / nt) * xt[:, None] / vt[None, :]
        A[k] = (Pt[k][:, None] * torch.complex(torch.cos(ph), -torch.sin(ph))).sum(0).abs() / x.size
    return np.arange(P.shape[0]) * (fs / nt), vel, A


def exact(case, seed):
    c, kind = case, case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "image":
        return _image(c, seed)
    if kind == "adjoint":
        return _gradient(c, seed, dev)
    with torch.no_grad():
        if kind == "group":
            return [_Exact(m, dev).forward(c["steps"])[0] for m in _group_models(c, seed)]
        if kind == "batch":
            m = _fluid_solid(c, seed)
            recs = [_Exact(m, dev, shot=s).forward(c["steps"])[0] for s in _shots(c, seed, m)]
            return {q: torch.stack([r[q] for r in recs]) for q in recs[0]}
        if kind == "solid":
            rec, U = _Exact(_solid_only(c, seed), dev, solid_only=True).forward(c["steps"])
            names = SOLID if c["out"] == "all" else SNAPSHOT[2:]
            return {"rec": rec, "field": {n: U["s"][SOLID.index(n)] for n in names}}
        rec, U = _Exact(_fluid_solid(c, seed), dev).forward(c["steps"])
    fields = {**{n: U["f"][k] for k, n in enumerate(FLUID)}, **{n: U["s"][k] for k, n in enumerate(SOLID)}}
    if kind == "noalloc":
        return {k: fields[("fluid_" if k.endswith("_f") else "solid_") + k[:-2]] for k in
                ("vx_f", "vz_f", "p_f", "vx_s", "vz_s", "sx_s", "sz_s", "sxz_s")}
    names = FLUID + SOLID if c["out"] == "all" else SNAPSHOT
    return {"rec": rec, "field": {n: fields[n] for n in names}}
