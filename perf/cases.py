"""What is measured: the work that a user of wgnet_gb300 has it do, through its public entry points.

A case is a dict of plain numbers and texts; `kind` says which path it takes, the rest are its sizes. Sizes are this
repository's own: the reference's default engine (5 shots, nt 2001, 0.5 ms), the 1 ms surveys of the benchmark and the
trainer, the 70/100/140 generation mix, the 800 x 300 survey at 5 m, and ragged grids between them.

`exact` restates each path in 64 bits with plain torch: the wave equation step by step with autograd for its gradient,
the renderer as a sum over slots, the update network as torch convolutions.
"""

from __future__ import annotations

import math

import numpy as np
import torch

FULL_BAND = 0.0  # `band_hz` of a case without a passband


def listed():
    return [
        # One forward solve of the reference's default engine on host arrays: what its Python calls most often, a
        # line-search trial of refine() or one model of its wave cache. Five units: latency.
        {"name": "simulate_one", "kind": "simulate", "models": 1, "shots": 5, "nt": 2001, "dt": 0.0005, "h": 10.0,
         "nx": 70, "nz": 70, "pml": 20},
        # One misfit and gradient of that engine in a refinement's 12 Hz band, on CUDA tensors: refine()'s other call.
        {"name": "gradient_one", "kind": "gradient", "models": 1, "shots": 5, "nt": 2001, "dt": 0.0005, "h": 10.0,
         "nx": 70, "nz": 70, "pml": 20, "band_hz": 12.0, "checkpoint": 0},
        # The differentiable physics loss of a training batch: dense fields plus rendered Gaussians, forward and
        # backward through autograd, checkpoints every 100 steps.
        {"name": "physics_loss_256", "kind": "physics_loss", "models": 256, "shots": 5, "nt": 1000, "dt": 0.001,
         "h": 10.0, "nx": 70, "nz": 70, "pml": 20, "checkpoint": 100},
        # A small batch on a ragged rectangular grid, the default checkpointing: surveys other than OpenFWI's.
        {"name": "gradient_ragged", "kind": "gradient", "models": 13, "shots": 3, "nt": 900, "dt": 0.001, "h": 10.0,
         "nx": 93, "nz": 77, "pml": 20, "band_hz": FULL_BAND, "checkpoint": 0},
        # Generation of FP16 gathers for mixed grid sizes in one graph launch: the wave cache of a training set.
        {"name": "datagen_mixed", "kind": "datagen", "total": 96, "shots": 5, "nt": 1000, "dt": 0.001, "factor": 4},
        # A survey beyond one SM's memory: forward and exact adjoint of 800 x 300 cells at 5 m.
        {"name": "survey_gradient", "kind": "gradient", "models": 1, "shots": 16, "nt": 800, "dt": 0.0005, "h": 5.0,
         "nx": 800, "nz": 300, "pml": 20, "band_hz": FULL_BAND, "checkpoint": 0},
        # A middle-sized survey's shots, forward only: synthetic data for it.
        {"name": "survey_simulate", "kind": "simulate", "models": 1, "shots": 10, "nt": 1200, "dt": 0.0005, "h": 5.0,
         "nx": 300, "nz": 150, "pml": 20},
        # The Gaussian renderer, forward and backward, on a training batch of the benchmark's size.
        {"name": "render_256", "kind": "render", "models": 256},
        # The update network's proposals for a batch of refinements (an odd batch: whoever is still running).
        {"name": "net_forward_45", "kind": "net_forward", "models": 45, "nx": 70, "nz": 70},
        # One Adam step of the update network at the trainer's batch size: loss and weight gradients.
        {"name": "net_train_32", "kind": "net_train", "models": 32, "nx": 70, "nz": 70},
        # A passband applied to the observed data of a batch: each band of a refinement starts with it.
        {"name": "bandlimit_16", "kind": "bandlimit", "models": 16, "shots": 5, "nt": 2001, "dt": 0.0005, "nrec": 70,
         "band_hz": 8.0},
        # A short refinement of a few models, whole: dense-block L-BFGS over two passbands, host control and all.
        {"name": "refine_8", "kind": "refine", "models": 8, "shots": 5, "nt": 1000, "dt": 0.001, "budget": 12},
    ]


def draw(rng):
    """One more case of the same ranges."""

    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def survey(most, nt):
        """Models and shots of at most `most` wave units."""
        shots = rng.randint(1, 5)
        return {"models": logint(1, max(1, most // shots)), "shots": shots, "nt": nt, "dt": 0.001, "h": 10.0}

    kind = rng.choice(("simulate", "gradient", "gradient", "physics_loss", "datagen", "survey", "render", "net_forward",
                       "net_train", "bandlimit", "refine"))
    if kind in ("simulate", "gradient"):
        square = rng.random() < 0.5
        nx = rng.choice((70, 70, 100, 140)) if square else rng.randint(40, 100)
        case = {"kind": kind, **survey(240, rng.randint(300, 1500)), "nx": nx,
                "nz": nx if square else rng.randint(70, 100), "pml": 20}
        if kind == "gradient":
            case |= {"band_hz": rng.choice((6.0, 9.0, 12.0, FULL_BAND)), "checkpoint": rng.choice((0, 25, 50, 100))}
        return case
    if kind == "physics_loss":
        return {"kind": kind, **survey(640, rng.randint(400, 1000)), "nx": 70, "nz": 70, "pml": 20,
                "checkpoint": rng.choice((25, 50, 100))}
    if kind == "datagen":
        return {"kind": kind, "total": logint(6, 160), "shots": rng.randint(1, 5), "nt": rng.randint(400, 1000),
                "dt": 0.001, "factor": rng.choice((2, 4, 8))}
    if kind == "survey":
        case = {"models": 1, "shots": rng.randint(2, 14), "nt": rng.randint(200, 700), "dt": 0.0005, "h": 5.0,
                "nx": 4 * rng.randint(60, 200), "nz": rng.randint(110, 300), "pml": 20}
        if rng.random() < 0.5:
            return {"kind": "simulate", **case}
        return {"kind": "gradient", **case, "band_hz": FULL_BAND, "checkpoint": 0}
    if kind == "render":
        return {"kind": kind, "models": logint(1, 256)}
    if kind == "net_forward":
        return {"kind": kind, "models": logint(1, 200), "nx": 70, "nz": 70}
    if kind == "net_train":
        return {"kind": kind, "models": 16 * rng.randint(1, 6), "nx": 70, "nz": 70}
    if kind == "bandlimit":
        return {"kind": kind, "models": logint(1, 64), "shots": rng.randint(1, 5), "nt": rng.randint(400, 2001),
                "dt": rng.choice((0.0005, 0.001)), "nrec": rng.choice((70, 70, rng.randint(40, 140))),
                "band_hz": rng.choice((6.0, 8.0, 9.0, 12.0))}
    return {"kind": "refine", "models": logint(1, 24), "shots": rng.randint(1, 5), "nt": rng.randint(400, 1000),
            "dt": 0.001, "budget": rng.randint(8, 16)}


# -- inputs ----------------------------------------------------------------------------------------


def _seed(seed, *more):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, *more])


def _models(n, seed, nz, nx):
    """Seeded velocity models of the flat / curved / faulted / blob families, and their smoothed starts (m/s)."""
    from wgnet_gb300.models_synth import make_batch, smooth

    true = make_batch(n, seed=seed, nz=nz, nx=nx)
    return true, smooth(true, 5.0)


def _gather(rng, models, shots, nt, dt, nx, h, nrec, device):
    """Observed shot gathers [models, shots, nt, nrec]: a direct arrival and eight hyperbolic reflections per shot as
    15 Hz Ricker pulses over weak noise, at the amplitudes of this survey's synthetics."""
    events = 9
    f32 = {"device": device, "dtype": torch.float32}
    t0 = torch.as_tensor(np.concatenate([np.zeros((models, 1, 1)), rng.uniform(0.05, 0.9 * nt * dt, (models, 1, events - 1))], 2),
                         **f32)
    vel = torch.as_tensor(rng.uniform(1600.0, 4200.0, (models, 1, events)), **f32)
    amp = torch.as_tensor(np.concatenate([np.full((models, 1, 1), 6.0), rng.normal(0.0, 3.0, (models, 1, events - 1))], 2),
                          **f32)
    xs = (nx - 1) * h * (torch.arange(shots, **f32) / max(shots - 1, 1) if shots > 1 else torch.full((1,), 0.5, **f32))
    off = (torch.arange(nrec, **f32) * h).view(1, -1) - xs.view(-1, 1)
    t = torch.arange(nt, **f32) * dt
    out = torch.as_tensor(rng.normal(0.0, 0.01, (1, 1, nt, nrec)), **f32).expand(models, shots, nt, nrec).clone()
    for e in range(events):
        arrival = torch.sqrt((t0[:, :, e:e + 1] ** 2) + (off.unsqueeze(0) / vel[:, :, e:e + 1]) ** 2) + 0.1
        a = (math.pi * 15.0 * (t.view(1, 1, -1, 1) - arrival.unsqueeze(2))) ** 2
        spread = amp[:, :, e].view(models, 1, 1, 1) / (1.0 + off.abs().view(1, shots, 1, nrec) / (10.0 * h))
        out += spread * (1.0 - 2.0 * a) * torch.exp(-a)
    return out.contiguous()


def _gaussians(rng, models, device):
    """Activated slot parameters [models, 1225, 6] within their bounds, most amplitudes small."""
    p = np.empty((models, 1225, 6), np.float32)
    p[..., 0:2] = rng.uniform(-2.0, 2.0, (models, 1225, 2))
    p[..., 2:4] = rng.uniform(math.log(0.5), math.log(6.0), (models, 1225, 2))
    p[..., 4] = rng.uniform(-math.pi / 2, math.pi / 2, (models, 1225))
    p[..., 5] = 0.05 * np.tanh(rng.normal(0.0, 1.0, (models, 1225)))
    return torch.from_numpy(p).to(device)


def _net_inputs(case, seed, device):
    n, nz, nx = case["models"], case["nz"], case["nx"]
    true, start = _models(n, seed, nz, nx)
    rng = _seed(seed, 4)
    grad = torch.from_numpy((rng.normal(0.0, 1.0, (n, nz, nx)) * 10.0 ** rng.uniform(-4, -1, (n, 1, 1))).astype(np.float32))
    band = torch.from_numpy(rng.integers(0, 4, n).astype(np.int32))
    vel = torch.from_numpy(start / np.float32(1000.0))
    target = torch.from_numpy(((true - start) / np.float32(1000.0)).astype(np.float32))
    return [t.to(device) for t in (vel, grad, band, target)]


def _engine(case):
    from wgnet_gb300.engine import WaveEngine

    eng = WaveEngine(shots=case["shots"], nt=case["nt"], dt=case["dt"], peak_hz=15.0, pml=case["pml"], vmin=1000.0,
                     vmax=5000.0, nx_vis=case["nx"], nz_vis=case["nz"], h=case["h"])
    if case.get("checkpoint"):
        eng.checkpoint_every = case["checkpoint"]
    return eng


def _is_default(case):
    """The reference's own engine: 5 shots, nt 2001, 0.5 ms, 70 x 70 at 10 m."""
    return (case["nx"], case["nz"], case["h"], case["dt"], case["pml"]) == (70, 70, 10.0, 0.0005, 20)


def _wave_inputs(case, seed, device):
    """Starting velocities (m/s) and observed gathers of a survey."""
    _, start = _models(case["models"], seed, case["nz"], case["nx"])
    obs = _gather(_seed(seed, 1), case["models"], case["shots"], case["nt"], case["dt"], case["nx"], case["h"], case["nx"],
                  device)
    return start, obs


def prepare(case, seed):
    kind = case["kind"]
    dev = torch.device("cuda")
    if kind == "simulate":
        true, _ = _models(case["models"], seed, case["nz"], case["nx"])
        if case["models"] == 1 and _is_default(case):
            from wgnet_gb300.wave_gauss_rs import PyWaveEngine

            return {"kind": "simulate_host", "engine": PyWaveEngine(case["shots"], case["nt"], case["dt"]),
                    "vel": np.ascontiguousarray(true.reshape(-1))}
        return {"kind": "simulate", "engine": _engine(case), "vel": torch.from_numpy(true).to(dev)}
    if kind == "gradient":
        from wgnet_gb300.physics import WavePhysics

        start, obs = _wave_inputs(case, seed, dev)
        if _is_default(case):
            physics = WavePhysics(case["shots"], case["nt"])
            if case["checkpoint"]:
                physics.wave.checkpoint_every = case["checkpoint"]
        else:
            physics = WavePhysics(case["shots"], case["nt"], engine=_engine(case))
        if case["band_hz"] != FULL_BAND:
            physics.set_band(case["band_hz"])
        return {"kind": kind, "physics": physics, "field": torch.from_numpy(start / np.float32(1000.0)).to(dev), "obs": obs}
    if kind == "physics_loss":
        start, obs = _wave_inputs(case, seed, dev)
        return {"kind": kind, "engine": _engine(case), "obs": obs,
                "dense": torch.from_numpy(start / np.float32(1000.0)).to(dev).requires_grad_(True),
                "gauss": _gaussians(_seed(seed, 2), case["models"], dev).requires_grad_(True)}
    if kind == "datagen":
        from wgnet_gb300.datagen import GatherGenerator, round_robin_counts

        counts = round_robin_counts(case["total"])
        gen = GatherGenerator(counts, shots=case["shots"], nt=case["nt"], dt=case["dt"], factor=case["factor"], autotune=False)
        return {"kind": kind, "gen": gen,
                "vel": {n: torch.from_numpy(_models(m, seed, n, n)[0]).to(dev) for n, m in counts.items()}}
    if kind == "render":
        rng = _seed(seed, 3)
        return {"kind": kind, "gauss": _gaussians(rng, case["models"], dev).requires_grad_(True),
                "cot": torch.from_numpy(rng.normal(0.0, 1.0, (case["models"], 70, 70)).astype(np.float32)).to(dev)}
    if kind in ("net_forward", "net_train"):
        from wgnet_gb300.precond import UpdateNet

        vel, grad, band, target = _net_inputs(case, seed, dev)
        return {"kind": kind, "net": UpdateNet.load("wgnet_gb300/weights/update_net.npz"), "vel": vel, "grad": grad,
                "band": band, "target": target}
    if kind == "bandlimit":
        obs = _gather(_seed(seed, 1), case["models"], case["shots"], case["nt"], case["dt"], case["nrec"], 10.0,
                      case["nrec"], dev)
        return {"kind": kind, "physics": _band_physics(case), "obs": obs}
    if kind == "refine":
        from wgnet_gb300.learned import physics_for

        true, start = _models(case["models"], seed, 70, 70)
        shots = tuple(range(case["shots"]))
        physics = physics_for(shots, case["nt"])
        obs = _gather(_seed(seed, 1), case["models"], case["shots"], case["nt"], case["dt"], 70, 10.0, 70, dev)
        return {"kind": kind, "physics": physics, "start": torch.from_numpy(start / np.float32(1000.0)).to(dev), "obs": obs,
                "budget": case["budget"]}
    raise ValueError(kind)


def _band_physics(case):
    from wgnet_gb300.engine import WaveEngine
    from wgnet_gb300.physics import WavePhysics

    physics = WavePhysics(case["shots"], case["nt"], engine=WaveEngine(shots=case["shots"], nt=case["nt"], dt=case["dt"]))
    physics.set_band(case["band_hz"])
    return physics


def run(state):
    kind = state["kind"]
    if kind == "simulate_host":
        return state["engine"].simulate(state["vel"])
    if kind == "simulate":
        return state["engine"].simulate_torch(state["vel"])
    if kind == "gradient":
        return state["physics"].loss_and_grad(state["field"], state["obs"])
    if kind == "physics_loss":
        from wgnet_gb300.physics import WaveLoss
        from wgnet_gb300.render import render_residual

        loss = WaveLoss.apply(state["dense"] + render_residual(state["gauss"]), state["obs"], state["engine"])
        grads = torch.autograd.grad(loss.mean(), [state["dense"], state["gauss"]])
        return {"loss": loss.detach(), "dense": grads[0], "gauss": grads[1]}
    if kind == "datagen":
        return {str(n): g for n, g in state["gen"].run(state["vel"]).items()}
    if kind == "render":
        from wgnet_gb300.render import render_residual

        field = render_residual(state["gauss"])
        (grad,) = torch.autograd.grad(field, [state["gauss"]], grad_outputs=state["cot"])
        return {"field": field.detach(), "grad": grad}
    if kind == "net_forward":
        return state["net"].forward(state["vel"], state["grad"], state["band"])
    if kind == "net_train":
        loss = state["net"].train_step(state["vel"], state["grad"], state["band"], state["target"], lr=1e-3)
        return {"loss": loss, "grads": state["net"].weight_gradients()}
    if kind == "bandlimit":
        return state["physics"].bandlimit(state["obs"])
    from wgnet_gb300.refine import refine_batch

    r = refine_batch(state["start"], state["obs"], state["physics"], budget_solves=state["budget"], bands_hz=(6.0, None),
                     dense_block=True)
    return {"field": r["final_field_km"], "coarse": r["coarse_km"], "loss": r["final_loss"], "solves": r["solves"]}


# -- the work a pass cannot do without -------------------------------------------------------------


def _step_flops(nx, nz, pml):
    """Operations of one time step of one unit, forward or adjoint: 24 a cell inside, 30 more for each axis's C-PML."""
    px, pz = nx + 2 * pml, nz + 2 * pml
    return 24.0 * px * pz + 30.0 * (2 * pml * pz + 2 * pml * px)


def work(case):
    kind = case["kind"]
    if kind in ("simulate", "gradient", "physics_loss"):
        b, s, nt, cells = case["models"], case["shots"], case["nt"], case["nx"] * case["nz"]
        traces = 4.0 * b * s * nt * case["nx"]
        step = b * s * nt * _step_flops(case["nx"], case["nz"], case["pml"])
        if kind == "simulate":
            return {"bytes": 4.0 * b * cells + traces, "flops": step}
        more = 2 * 4.0 * b * 1225 * 6 if kind == "physics_loss" else 0.0
        return {"bytes": 2 * 4.0 * b * cells + traces + more, "flops": 2 * step + 3.0 * b * s * nt * cells}
    if kind == "datagen":
        n_of = [(n, (case["total"] - i + 2) // 3) for i, n in enumerate((70, 100, 140))]
        out = -(-case["nt"] // case["factor"])
        return {"bytes": sum(m * (4.0 * n * n + 2.0 * case["shots"] * out * n) for n, m in n_of),
                "flops": sum(m * case["shots"] * case["nt"] * _step_flops(n, n, 20) for n, m in n_of)}
    if kind == "render":
        b = case["models"]
        return {"bytes": 4.0 * b * (2 * 4900 + 3 * 1225 * 6), "flops": 45.0 * b * 635209.0}  # in-grid window pixels
    if kind in ("net_forward", "net_train"):
        m = case["models"] * case["nx"] * case["nz"]
        passes = 1 if kind == "net_forward" else 3
        return {"bytes": 4.0 * m * (3 if kind == "net_forward" else 4) + 2.0 * 447552 * passes,
                "flops": 2.0 * 447552 * m * passes}
    if kind == "bandlimit":
        n = case["models"] * case["shots"] * case["nt"] * case["nrec"]
        return {"bytes": 8.0 * n, "flops": 2.0 * n * (2 * _half_taps(case["band_hz"], case["dt"]) + 1)}
    b, s, nt = case["models"], case["shots"], case["nt"]
    return {"bytes": 2 * 4.0 * b * 4900 + 4.0 * b * s * nt * 70, "flops": case["budget"] * b * s * nt * _step_flops(70, 70, 20)}


# -- the same in 64 bits ---------------------------------------------------------------------------


def _half_taps(fmax, dt):
    return int(math.ceil(4.0 * math.sqrt(math.log(2.0) / 2.0) / (math.pi * fmax) / dt))


def _lowpass64(fmax, dt):
    sigma = math.sqrt(math.log(2.0) / 2.0) / (math.pi * fmax)
    half = _half_taps(fmax, dt)
    h = np.exp(-0.5 * (np.arange(-half, half + 1) * dt / sigma) ** 2)
    return h / h.sum()


def _ricker64(nt, dt, peak):
    a = (np.pi * peak * (np.arange(nt) * dt - 1.5 / peak)) ** 2
    return (1.0 - 2.0 * a) * np.exp(-a)


def _cpml64(n, h, dt, width, vmax, freq):
    x = np.arange(n, dtype=np.float64)
    frac = np.clip(np.maximum((2 + width - x) / width, (x - (n - 3 - width)) / width), 0.0, 1.0)
    sigma = -(3.0 * vmax * math.log(0.001)) / (2.0 * width * h) * frac * frac
    alpha = math.pi * freq * (1.0 - frac)
    e = np.exp(-(sigma + alpha) * dt)
    b = sigma / (sigma + alpha) * (e - 1.0)
    a = np.where(frac == 0.0, 0.0, e)
    db = np.zeros(n)
    db[2:-2] = ((8.0 / 12.0) * (b[3:-1] - b[1:-3]) - (1.0 / 12.0) * (b[4:] - b[:-4])) / h
    return a, b, db


class _Wave64:
    """The C-PML acoustic time step in 64 bits on [units, nz, nx] tensors."""

    def __init__(self, case, wavelet, device):
        nxv, nzv, pml, h, dt = case["nx"], case["nz"], case["pml"], case["h"], case["dt"]
        self.pad = pml + 2
        self.nx, self.nz, self.h, self.dt, self.nt = nxv + 2 * self.pad, nzv + 2 * self.pad, h, dt, case["nt"]
        self.shots, self.dev = case["shots"], device
        put = lambda a: torch.as_tensor(a, device=device, dtype=torch.float64)  # noqa: E731
        self.px = [put(p[2:-2]).view(1, 1, -1) for p in _cpml64(self.nx, h, dt, pml, 5000.0, 15.0)]
        self.pz = [put(p[2:-2]).view(1, -1, 1) for p in _cpml64(self.nz, h, dt, pml, 5000.0, 15.0)]
        self.wav = [float(v) for v in wavelet]
        xmax = (nxv - 1) * h
        xs = [xmax * 0.5] if self.shots == 1 else [xmax * k / (self.shots - 1) for k in range(self.shots)]
        self.set_sources([(x, h) for x in xs])
        corners = [self._corner(k * h, h) for k in range(nxv)]
        self.rcell = torch.tensor([c for c, _ in corners], device=device)
        self.rw = put([w for _, w in corners])
        iz = torch.arange(self.nz, device=device).sub(self.pad).clamp(0, nzv - 1)
        ix = torch.arange(self.nx, device=device).sub(self.pad).clamp(0, nxv - 1)
        self.fold = (iz.view(-1, 1) * nxv + ix.view(1, -1)).reshape(-1)

    def _corner(self, px, pz):
        gx, gz = px / self.h + self.pad, pz / self.h + self.pad
        # the stations sit on nodes or between two of them in 32 bits, too: their f32 positions
        gx, gz = float(np.float32(gx)), float(np.float32(gz))
        x0, z0 = min(int(math.floor(gx)), self.nx - 2), min(int(math.floor(gz)), self.nz - 2)
        fx, fz = gx - x0, gz - z0
        c = z0 * self.nx + x0
        return (c, c + 1, c + self.nx, c + self.nx + 1), ((1 - fx) * (1 - fz), fx * (1 - fz), (1 - fx) * fz, fx * fz)

    def set_sources(self, xz):
        corners = [self._corner(x, z) for x, z in xz]
        self.scell = torch.tensor([c for c, _ in corners], device=self.dev)
        self.sw = torch.tensor([w for _, w in corners], device=self.dev, dtype=torch.float64)

    def padded(self, vel):
        """Visible [M, nz, nx] m/s onto the padded grid of every unit: [M * shots, nz, nx]."""
        v = vel.double().flatten(1)[:, self.fold].view(-1, self.nz, self.nx)
        return v.repeat_interleave(self.shots, 0)

    def zero(self, units):
        z = torch.zeros((units, self.nz, self.nx), device=self.dev, dtype=torch.float64)
        return [z, z, z, z, z[:, 2:-2, 2:-2], z[:, 2:-2, 2:-2]]

    def _axis(self, u, ap, zeta, prof, dim):
        a, b, db = prof
        n = u.shape[dim] - 4
        s = [u.narrow(dim, k, n).narrow(3 - dim, 2, u.shape[3 - dim] - 4) for k in range(5)]
        p = [ap.narrow(dim, k, n).narrow(3 - dim, 2, u.shape[3 - dim] - 4) for k in range(5)]
        d2 = (-2.5 * s[2] + (4.0 / 3.0) * (s[3] + s[1]) - (1.0 / 12.0) * (s[4] + s[0])) / (self.h * self.h)
        d1 = ((2.0 / 3.0) * (s[3] - s[1]) - (1.0 / 12.0) * (s[4] - s[0])) / self.h
        da = ((2.0 / 3.0) * (p[3] - p[1]) - (1.0 / 12.0) * (p[4] - p[0])) / self.h
        tmp = (1.0 + b) * d2 + db * d1 + da
        az = a * zeta
        grow = lambda t: torch.nn.functional.pad(t, (2, 2, 2, 2))  # noqa: E731
        return (1.0 + b) * tmp + az, grow(a * (b * d1 + p[2])), b * tmp + az

    def steps(self, state, v, t0, t1):
        """Steps [t0, t1): the state after them and the traces before each."""
        u, up, ax, az, zx, zz = state
        v2 = (v * v) * (self.dt * self.dt)
        units = v.shape[0]
        cell = self.scell.repeat(units // self.shots, 1)
        src = -v2.flatten(1).gather(1, cell) * self.sw.repeat(units // self.shots, 1)
        out = []
        for t in range(t0, t1):
            out.append((u.flatten(1)[:, self.rcell] * self.rw).sum(-1))
            wx, ax, zx = self._axis(u, ax, zx, self.px, 2)
            wz, az, zz = self._axis(u, az, zz, self.pz, 1)
            nu = torch.nn.functional.pad(v2[:, 2:-2, 2:-2] * (wx + wz) + 2.0 * u[:, 2:-2, 2:-2] - up[:, 2:-2, 2:-2],
                                         (2, 2, 2, 2))
            nu = nu.flatten(1).scatter_add(1, cell, src * self.wav[t]).view_as(u)
            u, up = nu, u
        return [u, up, ax, az, zx, zz], torch.stack(out, 1)

    def traces(self, vel):
        v = self.padded(vel)
        with torch.no_grad():
            _, tr = self.steps(self.zero(v.shape[0]), v, 0, self.nt)
        return tr.view(vel.shape[0], self.shots, self.nt, -1)

    def gradient(self, vel, obs, seg):
        """0.5 |p - d|^2 / |d|^2 of each model and its gradient with respect to the visible velocities (m/s)."""
        obs = obs.double()
        scale = 1.0 / obs.flatten(1).square().sum(1)
        bounds = list(range(0, self.nt, seg)) + [self.nt]
        vis = vel.double().requires_grad_(True)
        v = self.padded(vis)
        vd = v.detach()
        state, kept, res = self.zero(v.shape[0]), [], []
        with torch.no_grad():
            for t0, t1 in zip(bounds[:-1], bounds[1:]):
                kept.append(state)
                state, tr = self.steps(state, vd, t0, t1)
                res.append(tr)
        tr = torch.cat(res, 1).view_as(obs)
        loss = 0.5 * (tr - obs).flatten(1).square().sum(1) * scale
        cot = ((tr - obs) * scale.view(-1, 1, 1, 1)).view(v.shape[0], self.nt, -1)
        back, gv = None, torch.zeros_like(vd)
        for k in reversed(range(len(kept))):
            leaf = vd.clone().requires_grad_(True)
            first = [s.detach().requires_grad_(True) for s in kept[k]]
            last, tr = self.steps(first, leaf, bounds[k], bounds[k + 1])
            outs, grads = [tr], [cot[:, bounds[k]:bounds[k + 1]]]
            if back is not None:
                outs, grads = outs + last, grads + back
            got = torch.autograd.grad(outs, [leaf] + first, grads, allow_unused=True)
            gv += got[0]
            back = [g if g is not None else torch.zeros_like(s) for g, s in zip(got[1:], first)]
        (g,) = torch.autograd.grad(v, [vis], gv)
        return loss, g


def _render64(gauss):
    """Sum over slots of their Gaussians within a 25 x 25 window, [B, 70, 70]."""
    b = gauss.shape[0]
    slot = torch.arange(1225, device=gauss.device)
    k = torch.arange(625, device=gauss.device)
    rows = (2 * (slot // 35)).view(-1, 1) + (k // 25 - 12)
    cols = (2 * (slot % 35)).view(-1, 1) + (k % 25 - 12)
    ok = (rows >= 0) & (rows < 70) & (cols >= 0) & (cols < 70)
    s, w = torch.nonzero(ok, as_tuple=True)
    r, c = rows[s, w], cols[s, w]
    p = gauss[:, s]
    dx = c.double() + 0.5 - (2.0 * (s % 35) + 1.0) - p[..., 0]
    dz = r.double() + 0.5 - (2.0 * (s // 35) + 1.0) - p[..., 1]
    co, si = torch.cos(p[..., 4]), torch.sin(p[..., 4])
    u = (dx * co + dz * si) * torch.exp(-p[..., 2])
    v = (dz * co - dx * si) * torch.exp(-p[..., 3])
    value = p[..., 5] * torch.exp(-0.5 * (u * u + v * v))
    return torch.zeros((b, 4900), device=gauss.device, dtype=torch.float64).index_add(1, r * 70 + c, value).view(b, 70, 70)


def _net64(case, seed, device, train):
    vel, grad, band, target = (t.double() if t.is_floating_point() else t for t in _net_inputs(case, seed, device))
    b, nz, nx = vel.shape
    dil = (1, 2, 4, 8, 4, 2)
    with np.load("wgnet_gb300/weights/update_net.npz") as d:
        raw = {k: torch.from_numpy(d[k].astype(np.float64)).to(device) for k in d.files if k != "step"}
    weights = {}
    for name, w in raw.items():
        cin, rows = (8 if name == "in" else 64), (1 if name == "out" else 64)
        weights[name] = w[:rows, :9 * cin].reshape(rows, 3, 3, cin).permute(0, 3, 1, 2).contiguous().requires_grad_(train)
    rms = grad.flatten(1).square().mean(1).sqrt().view(-1, 1, 1)
    f = [vel - 3.0, torch.where(rms > 0, grad / rms, 0.0)] + [(band == k).double().view(-1, 1, 1).expand(b, nz, nx)
                                                             for k in range(4)]
    f += [(torch.arange(nz, device=device, dtype=torch.float64) / nz).view(1, -1, 1).expand(b, nz, nx),
          torch.zeros_like(vel)]
    conv = lambda x, name, d: torch.nn.functional.conv2d(x, weights[name], padding=d, dilation=d)  # noqa: E731
    h = torch.relu(conv(torch.stack(f, 1), "in", 1))
    for i, d in enumerate(dil):
        h = h + conv(torch.relu(conv(h, f"b{i}a", d)), f"b{i}b", 1)
    out = conv(h, "out", 1)[:, 0] * 0.25
    if not train:
        return out
    loss = (out - target).square().mean()
    names = list(weights)
    grads = {}
    for name, g in zip(names, torch.autograd.grad(loss, [weights[n] for n in names])):
        full = torch.zeros_like(raw[name])
        full[:g.shape[0], :9 * g.shape[1]] = g.permute(0, 2, 3, 1).reshape(g.shape[0], -1)
        grads[name] = full
    return {"loss": float(loss.detach()), "grads": grads}


def _bandlimit64(x, taps):
    """Causal FIR along time of [models, shots, nt, nrec]."""
    k = len(taps)
    y = torch.nn.functional.pad(x.double(), (0, 0, k - 1, 0))
    out = torch.zeros(x.shape, device=x.device, dtype=torch.float64)
    for i, w in enumerate(taps):
        out += float(w) * y[:, :, i:i + x.shape[2]]
    return out


def exact(case, seed):
    kind = case["kind"]
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    if kind in ("simulate", "gradient"):
        wav = _ricker64(case["nt"], case["dt"], 15.0)
        cells = case["models"] * case["shots"] * (case["nx"] + 44) * (case["nz"] + 44)
        if cells * case["nt"] > (8e9 if kind == "simulate" else 4e9):
            return None
        if kind == "simulate":
            true, _ = _models(case["models"], seed, case["nz"], case["nx"])
            tr = _Wave64(case, wav, dev).traces(torch.from_numpy(true).to(dev))
            return tr[0] if case["models"] == 1 and _is_default(case) else tr
        start, obs = _wave_inputs(case, seed, dev)
        if case["band_hz"] != FULL_BAND:
            wav = np.convolve(wav, _lowpass64(case["band_hz"], case["dt"]))[:case["nt"]]
        field = torch.from_numpy(start / np.float32(1000.0)).to(dev).double()
        loss, g = _Wave64(case, wav, dev).gradient(field * 1000.0, obs, max(4, min(64, int(4e8 / (cells * 4)))))
        return loss, g * 1000.0
    if kind == "datagen":
        if case["total"] > 128:
            return None
        out = {}
        taps = torch.from_numpy(_lowpass64(round(0.4 * 0.5 / (case["factor"] * case["dt"]), 6), case["dt"])).to(dev)
        half = len(taps) // 2
        for i, n in enumerate((70, 100, 140)):
            m = (case["total"] - i + 2) // 3
            sub = {**case, "models": m, "nx": n, "nz": n, "pml": 20, "h": 10.0}
            tr = _Wave64(sub, _ricker64(case["nt"], case["dt"], 15.0), dev).traces(
                torch.from_numpy(_models(m, seed, n, n)[0]).to(dev))
            win = torch.nn.functional.pad(tr, (0, 0, half, half)).unfold(2, len(taps), case["factor"])
            out[str(n)] = win @ taps
        return out
    if kind == "render":
        rng = _seed(seed, 3)
        gauss = _gaussians(rng, case["models"], dev).double()
        cot = torch.from_numpy(rng.normal(0.0, 1.0, (case["models"], 70, 70)).astype(np.float32)).to(dev).double()
        fields, grads = [], []
        for k in range(0, case["models"], 16):
            g = gauss[k:k + 16].clone().requires_grad_(True)
            f = _render64(g)
            grads.append(torch.autograd.grad(f, [g], cot[k:k + 16])[0])
            fields.append(f.detach())
        return {"field": torch.cat(fields), "grad": torch.cat(grads)}
    if kind == "net_forward":
        return _net64(case, seed, dev, False)
    if kind == "net_train":
        return _net64(case, seed, dev, True)
    if kind == "bandlimit":
        obs = _gather(_seed(seed, 1), case["models"], case["shots"], case["nt"], case["dt"], case["nrec"], 10.0,
                      case["nrec"], dev)
        return _bandlimit64(obs, _lowpass64(case["band_hz"], case["dt"]))
    # the whole batch of a training step is beyond twenty seconds in 64 bits, and a refinement's decisions follow the
    # rounding of its solves
    return None
