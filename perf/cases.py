"""The workloads this framework's speed is measured on: what a user's program has it do, through its public entry points.

Four kinds, over the range the library is used at:
  - "gravity": P2 alone on device buffers (`sr_gravity_solve_static`, worlds up to 256 x 256): the smallest calls;
  - "step":    a world carried through some steps — the state uploaded from pinned host memory, `run(steps)`, the state
               read back: gas alone, gas with self-gravity, implicit radiative diffusion alone (multigrid, Jacobi or the
               learned preconditioner), everything together, 4 channels or the 14 of reference mode;
  - "batch":   many worlds of uneven sizes advanced together;
  - "network": the learned preconditioner's forward and backward pass on a training batch.

Every input comes from the seed. `exact` restates the physics in plain 64-bit torch: MUSCL-Hancock/HLL gas with the
half-step gravity work, the free-space FFT potential, the flux-limited implicit diffusion step by Newton and
Jacobi-preconditioned CG to 1e-11, the floors and the Δt rule, and the U-Net by autograd.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch
import torch.nn.functional as F

from sandbox_reactions_b200.abi import Config
from sandbox_reactions_b200.engine import Batch, Learner, Step, load_library

DEV = "cuda" if torch.cuda.is_available() else "cpu"
F64 = torch.float64
VAC = float(np.float32(1e-6))    # sigma_vac and sigma_floor as the FP32 planes are compared with them
FLOOR = float(np.float32(1e-8))
FLOOR_GAS = 4e-6                 # the thin gas around a disk, above sigma_vac
TRAIN = 100                      # Adam steps behind the learned preconditioner


# ------------------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # one gravity solve on a small ragged world inside somebody else's loop: launches and latency
        {"name": "gravity_136x104", "kind": "gravity", "w": 136, "h": 104, "kernel": "self_cell"},
        # the largest world of the call that allocates nothing
        {"name": "gravity_256", "kind": "gravity", "w": 256, "h": 256, "kernel": "softened"},
        # the shock-tube configuration: 512², minmod, open edges, gas alone
        {"name": "sod_512", "kind": "step", "scene": "sod", "w": 512, "h": 512, "steps": 100, "limiter": "minmod",
         "edge": "leave", "gamma": 1.4},
        # a small wide tube whose axes divide no tile, walls around it: short kernels, many steps
        {"name": "sod_328x120", "kind": "step", "scene": "sod", "w": 328, "h": 120, "steps": 60, "limiter": "mc",
         "edge": "bounce", "gamma": 5.0 / 3.0},
        # the self-gravitating disk configuration: 1024², softened kernel, hydro and gravity
        {"name": "disk_1024", "kind": "step", "scene": "disk", "w": 1024, "h": 1024, "steps": 20, "limiter": "mc",
         "edge": "leave", "gamma": 5.0 / 3.0, "kernel": "softened"},
        # a ragged world with vacuum around the gas, the exact self-cell kernel, reflecting walls
        {"name": "disk_1304x712", "kind": "step", "scene": "disk", "w": 1304, "h": 712, "steps": 10, "limiter": "mc",
         "edge": "bounce", "gamma": 2.0, "kernel": "self_cell", "rim": 0.42},
        # the implicit diffusion configuration alone: 2048², V(2,2) multigrid, a stiff step
        {"name": "fld_2048", "kind": "step", "scene": "fld", "w": 2048, "h": 2048, "steps": 1, "precond": "mg",
         "sweeps": 2, "stiff": 2000.0},
        # the same configuration's solver with the learned preconditioner (trained beforehand) in flexible CG
        {"name": "fld_learned_512", "kind": "step", "scene": "fld", "w": 512, "h": 512, "steps": 1,
         "precond": "learned", "sweeps": 2, "stiff": 50.0},
        # the whole step at the headline size: hydro, gravity, radiation, opacity over six decades
        {"name": "full_2048", "kind": "step", "scene": "full", "w": 2048, "h": 2048, "steps": 3, "limiter": "mc",
         "edge": "leave", "gamma": 5.0 / 3.0, "kernel": "softened", "precond": "mg", "sweeps": 4},
        # reference mode: 14 channels, cold pressures, ten species, gravity, radiation and its force
        {"name": "ref_512", "kind": "step", "scene": "ref", "w": 512, "h": 512, "steps": 4, "limiter": "mc",
         "edge": "leave", "kernel": "self_cell", "precond": "mg", "sweeps": 4},
        # uneven small and middle worlds advanced together, each the whole step
        {"name": "batch_7", "kind": "batch", "sizes": "256x256 128x200 384x256 64x64 256x512 512x328 512x512",
         "steps": 2},
        # one training batch of the learned preconditioner: forward, loss, every gradient
        {"name": "network_16x64", "kind": "network", "n": 16, "crop": 64},
    ]


def _axis(rng, lo, hi):
    """A multiple of 8 in lo..hi, spread over the logarithm."""
    return int(min(hi, max(lo, 8 * round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 8))))


def draw(rng):
    kind = rng.choice(["gravity", "sod", "disk", "disk", "fld", "full", "full", "ref", "batch", "network"])
    mg = {"precond": "mg", "sweeps": rng.choice([2, 4])}
    scheme = {"limiter": rng.choice(["mc", "minmod"]), "edge": rng.choice(["leave", "bounce"]),
              "gamma": rng.choice([1.4, 5.0 / 3.0, 2.0])}
    grav = {"kernel": rng.choice(["softened", "self_cell"])}
    rim = {"rim": round(rng.uniform(0.3, 0.5), 3)} if rng.random() < 0.4 else {}
    if kind == "gravity":
        return {"kind": "gravity", "w": _axis(rng, 16, 256), "h": _axis(rng, 16, 256), **grav}
    if kind == "sod":
        return {"kind": "step", "scene": "sod", "w": _axis(rng, 64, 1024), "h": _axis(rng, 64, 1024),
                "steps": rng.randint(10, 60), **scheme}
    if kind == "disk":
        return {"kind": "step", "scene": "disk", "w": _axis(rng, 64, 1536), "h": _axis(rng, 64, 1536),
                "steps": rng.randint(2, 12), **scheme, **grav, **rim}
    if kind == "fld":
        pre = {"precond": "jacobi"} if rng.random() < 0.25 else mg
        return {"kind": "step", "scene": "fld", "w": _axis(rng, 64, 1024), "h": _axis(rng, 64, 1024),
                "steps": rng.randint(1, 2), **pre, "stiff": float(round(math.exp(rng.uniform(4.0, 8.0))))}
    if kind == "full":
        return {"kind": "step", "scene": "full", "w": _axis(rng, 64, 1280), "h": _axis(rng, 64, 1280),
                "steps": rng.randint(1, 2), **scheme, **grav, **mg, **rim}
    if kind == "ref":
        return {"kind": "step", "scene": "ref", "w": _axis(rng, 64, 768), "h": _axis(rng, 64, 768),
                "steps": rng.randint(1, 2), "limiter": scheme["limiter"], "edge": scheme["edge"], **grav, **mg}
    if kind == "batch":
        sizes = " ".join("%dx%d" % (_axis(rng, 64, 512), _axis(rng, 64, 512)) for _ in range(rng.randint(2, 6)))
        sizes += " %dx%d" % (2 * (rng.choice([128, 256, 512]),))  # the configured mix's powers of two among them
        return {"kind": "batch", "sizes": sizes, "steps": rng.randint(2, 4)}
    return {"kind": "network", "n": rng.randint(2, 24), "crop": 8 * rng.randint(2, 12)}


# ----------------------------------------------------------------------------------------------- configurations
def _config(c, dt=0.0):
    scene = c["scene"]
    k = dict(width=c["w"], height=c["h"], hydro=scene != "fld", gravity=scene in ("disk", "full", "ref"),
             heat=scene in ("fld", "full", "ref"), opacity_plane=scene in ("fld", "full"))
    for name in ("edge", "limiter", "gamma", "kernel"):
        if name in c:
            k[name] = c[name]
    if k["heat"]:
        k["precond"] = "mg" if c["precond"] == "learned" else c["precond"]
        if "sweeps" in c:
            k["mg_pre"] = k["mg_post"] = c["sweeps"]
    if scene == "disk":
        k["t_floor"] = 1e-6
    if scene == "fld":
        k["gamma"] = 5.0 / 3.0
        k["dt_fixed"] = dt
    if scene == "ref":
        k["channels"] = 14
        k["gamma"] = 2.0
    return Config(**k)


def _worlds(case):
    return [{"kind": "step", "scene": "full", "w": int(w), "h": int(h), "steps": case["steps"], "limiter": "mc",
             "edge": "leave", "gamma": 5.0 / 3.0, "kernel": "softened", "precond": "mg", "sweeps": 4}
            for w, h in (s.split("x") for s in case["sizes"].split())]


# ------------------------------------------------------------------------------------------------------- the inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _grid(w, h):
    y, x = torch.meshgrid(torch.arange(h, device=DEV, dtype=F64), torch.arange(w, device=DEV, dtype=F64), indexing="ij")
    return x, y


def _field(w, h, corr, g):
    """A unit Gaussian random field of correlation length `corr` cells."""
    white = torch.randn((h, w), generator=g, device=DEV, dtype=F64)
    ky = 2 * math.pi * torch.fft.fftfreq(h, device=DEV, dtype=F64)[:, None]
    kx = 2 * math.pi * torch.fft.fftfreq(w, device=DEV, dtype=F64)[None, :]
    f = torch.fft.ifft2(torch.fft.fft2(white) * torch.exp(-0.5 * (kx * kx + ky * ky) * corr * corr)).real
    f = f - f.mean()
    return f / f.std()


def _opacity(w, h, g):
    """Lognormal over six decades (0.1 to 99.9 percent), 32-cell correlation."""
    f = _field(w, h, min(32.0, min(w, h) / 8.0), g)
    s = torch.sort(f.flatten())[0]
    lo, hi = s[int(0.001 * (s.numel() - 1))], s[int(0.999 * (s.numel() - 1))]
    return torch.exp(6.0 * math.log(10.0) / (hi - lo) * f)


def _hot_spots(w, h, g, bg, spot, radius):
    x, y = _grid(w, h)
    T = torch.full((h, w), bg, device=DEV, dtype=F64)
    at = torch.rand((3, 2), generator=g, device=DEV, dtype=F64) * 0.6 + 0.2
    for a, b in at.tolist():
        T += (spot - bg) * torch.exp(-((x - a * w) ** 2 + (y - b * h) ** 2) / (2 * radius * radius))
    return T


def _disk(w, h, g, mass, rim=None):
    """A Gaussian disk with lognormal noise on circular orbits of the mass inside them, in thin gas; with `rim` it
    falls off to vacuum (returned as a mask) around that radius."""
    x, y = _grid(w, h)
    dx, dy = x - (w - 1) / 2, y - (h - 1) / 2
    r = torch.hypot(dx, dy)
    s = 0.15 * min(w, h)
    noise = torch.exp(0.05 * torch.randn((h, w), generator=g, device=DEV, dtype=F64))
    sig = mass * torch.exp(-r * r / (2 * s * s)) * noise
    void = None
    if rim:
        sig = sig * torch.exp(-(r / (rim * min(w, h))) ** 10)
        void = sig < FLOOR_GAS
    sig = torch.clamp(sig, min=FLOOR_GAS)
    order = torch.argsort(r.flatten())
    inside = torch.empty(w * h, device=DEV, dtype=F64)
    inside[order] = torch.cumsum(sig.flatten()[order], 0)
    v = torch.sqrt(inside.reshape(h, w) / torch.clamp(r, min=0.5))
    r = torch.clamp(r, min=1e-12)
    return sig, -v * dy / r, v * dx / r, void


def _planes(sig, u, v, p, gamma):
    return torch.stack([sig, sig * u, sig * v, p / (gamma - 1) + 0.5 * sig * (u * u + v * v)])


def _scene(c, seed):
    """The state, FP32 planes (4 or 14, h, w), the opacity plane or None, and the fixed Δt or 0."""
    g = _gen(seed)
    w, h = c["w"], c["h"]
    x, y = _grid(w, h)
    kappa, dt = None, 0.0
    if c["scene"] == "sod":
        a, b, k = torch.rand(3, generator=g, device=DEV, dtype=F64).tolist()
        edge = w * (0.4 + 0.2 * a) + 0.02 * w * torch.sin(2 * math.pi * y / h * (1 + int(4 * k)))
        left = x < edge
        noise = 1 + 0.02 * _field(w, h, 6.0, g)
        sig = torch.where(left, 1.0, 0.125 * (0.8 + 0.4 * b)) * noise
        P = _planes(sig, 0.1 * noise - 0.1, 0 * x, torch.where(left, 1.0, 0.1), c["gamma"])
    elif c["scene"] == "ref":
        sol = 0.3125 * min(w, h)
        a, b = (torch.rand(2, generator=g, device=DEV, dtype=F64) * 0.1 + 0.42).tolist()
        r = torch.hypot(x - w / 2, y - h / 2)
        core = torch.hypot(x - a * w, y - b * h) < 0.0625 * min(w, h)
        body = (r < sol) & ~core
        noise = 1 + 0.05 * _field(w, h, 4.0, g)
        sig = (2e-3 + torch.exp(-4 * (r / sol) ** 2) + 2.0 * core) * noise
        T = torch.where(core, 400.0, torch.where(body, 40.0, 1.0)).to(F64)
        X = torch.zeros((10, h, w), device=DEV, dtype=F64)
        X[0] = torch.where(core, 0.0, torch.where(body, 0.7346, 1.0))
        X[1] = torch.where(core, 1.0, torch.where(body, 0.2485, 0.0))
        X[2] = torch.where(body, 0.0092, 0.0)
        X[3] = torch.where(body, 0.0077, 0.0)
        u, v = torch.where(body, 0.05, 0.0), torch.where(body, 0.02, 0.0)
        gas = _Gas(_config(c))
        inv_mu, ye = gas.composition(X)
        e = sig * T * inv_mu + gas.cold_energy(sig, ye, X[9]) + 0.5 * sig * (u * u + v * v)
        P = torch.cat([torch.stack([sig, sig * u, sig * v, e]), X])
    elif c["scene"] == "fld":
        kappa = _opacity(w, h, g)
        T = _hot_spots(w, h, g, 1e3, 1e6, min(w, h) / 32.0)
        P = _planes(torch.ones_like(T), 0 * T, 0 * T, T, 5.0 / 3.0)
        # Δt: `stiff` times the explicit diffusion limit, the least C / (4 a_r T³) over a cell's couplings
        er, ar = 6.25e-7 * T ** 4, 6.25e-7
        dsum = torch.zeros_like(T)
        for d in (0, 1):
            lo, hi = [slice(None)] * 2, [slice(None)] * 2
            lo[d], hi[d] = slice(None, -1), slice(1, None)
            ks, fe = 0.5 * (kappa[tuple(lo)] + kappa[tuple(hi)]), 0.5 * (er[tuple(lo)] + er[tuple(hi)])
            R = (er[tuple(hi)] - er[tuple(lo)]).abs() / (ks * fe)
            D = 12800.0 * (2 + R) / (6 + 3 * R + R * R) / ks
            dsum[tuple(lo)] += D
            dsum[tuple(hi)] += D
        dt = c["stiff"] * float((1.5 / (4 * ar * T ** 3) / dsum).min())
    else:
        mass = c.get("mass", 1.0)
        sig, u, v, void = _disk(w, h, g, mass, c.get("rim"))
        if c["scene"] == "full":
            kappa = _opacity(w, h, g)
            p = sig * _hot_spots(w, h, g, 1.0, 100.0, min(w, h) / 64.0)
        else:
            # a warm disk (sound speed about a fifth of the orbital speed): a cold one amplifies the last bit of its state
            p = 0.15 * 0.15 * min(w, h) * sig ** c["gamma"]
        P = _planes(sig, u, v, p, c["gamma"])
        if void is not None:  # the floor state
            t_floor = 1e-6 if c["scene"] == "disk" else 0.05
            z = torch.zeros_like(x)
            P = torch.where(void[None], torch.stack([z + FLOOR, z, z, z + FLOOR * t_floor / (c["gamma"] - 1)]), P)
    return P.to(torch.float32), None if kappa is None else kappa.to(torch.float32), dt


def _batch_scenes(case, seed):
    worlds = _worlds(case)
    for k, c in enumerate(worlds):
        c["mass"] = 0.5 + 1.5 * float(torch.rand(1, generator=_gen(seed * 131 + k), device=DEV))
    return worlds, [_scene(c, seed * 131 + k) for k, c in enumerate(worlds)]


def _host(t):
    """A pinned host array of a device tensor's values."""
    if t is None:
        return None
    pinned = torch.empty(t.shape, dtype=t.dtype, pin_memory=DEV == "cuda")
    pinned.copy_(t)
    return pinned.numpy()


# the network: (cin, cout, input, relu); "skip" adds the encoder layer's output
_LAYERS = [(4, 8, "in", 1), (8, 8, "prev", 1), (8, 16, "pool", 1), (16, 16, "prev", 1), (16, 32, "pool", 1),
           (32, 32, "prev", 1), (32, 64, "pool", 1), (64, 64, "prev", 1), (64, 32, "up", 1), (32, 32, "skip", 1),
           (32, 16, "up", 1), (16, 16, "skip", 1), (16, 8, "up", 1), (8, 8, "skip", 1), (8, 1, "prev", 0)]
_SKIP = {9: 5, 11: 3, 13: 1}


def _network_inputs(case, seed):
    """Weights of a network in training and a batch: unit residuals, scaled couplings, mass shares; smooth errors."""
    g = _gen(seed)
    n, crop = case["n"], case["crop"]
    parts = []
    for ci, co, _, relu in _LAYERS:
        parts.append(math.sqrt((2.0 if relu else 1.0) / (9 * ci))
                     * torch.randn(co * 9 * ci, generator=g, device=DEV, dtype=F64))
        parts.append(0.05 * torch.randn(co, generator=g, device=DEV, dtype=F64))
    feats = torch.empty((n, 4, crop, crop), device=DEV, dtype=F64)
    feats[:, 0] = torch.randn((n, crop, crop), generator=g, device=DEV, dtype=F64)
    feats[:, 1:3] = 0.25 * torch.rand((n, 2, crop, crop), generator=g, device=DEV, dtype=F64)
    feats[:, 3] = torch.rand((n, crop, crop), generator=g, device=DEV, dtype=F64)
    target = torch.stack([_field(crop, crop, 2.0, g) for _ in range(n)])
    f32 = torch.float32
    return torch.cat(parts).to(f32), feats.to(f32), target.to(f32)


# ------------------------------------------------------------------------------------------------------- a program
def prepare(case, seed):
    kind = case["kind"]
    if kind == "gravity":
        w, h = case["w"], case["h"]
        sig = _disk(w, h, _gen(seed), 1.0)[0].to(torch.float32).contiguous()
        cfg = Config(width=w, height=h, gravity=True, kernel=case["kernel"]).to_c()
        return {"lib": load_library(), "cfg": cfg, "sigma": sig, "out": [torch.empty_like(sig) for _ in range(3)]}
    if kind == "network":
        theta, feats, target = (_host(t) for t in _network_inputs(case, seed))
        learner = Learner(crop=case["crop"], capacity=16, seed=0)
        learner.set_params(theta)
        return {"learner": learner, "feats": feats, "target": target}
    if kind == "batch":
        worlds, scenes = _batch_scenes(case, seed)
        batch = Batch([_config(c) for c in worlds])
        return {"batch": batch, "in": [(_host(P), _host(k)) for P, k, _ in scenes], "steps": case["steps"]}
    P, kappa, dt = _scene(case, seed)
    step = Step(_config(case, dt))
    state = {"step": step, "planes": _host(P), "kappa": _host(kappa), "out": _host(torch.zeros_like(P)),
             "steps": case["steps"]}
    if case.get("precond") == "learned":
        # a network trained on the residuals of smaller worlds of the same kind
        small = dict(case, w=256, h=256)
        learner = Learner(crop=64, capacity=512, seed=1)
        for k in range(3):
            tP, tk, tdt = _scene(small, seed + 1 + k)
            with Step(_config(small, tdt)) as t:
                t.upload(_host(tP))
                t.upload_opacity(_host(tk))
                learner.collect(t, tdt, crops=16, seed=k)
        learner.train(TRAIN, batch=8, seed=1)
        step.attach_learner(learner)
        step.set_heat_precond("learned")
        state["learner"] = learner
    return state


def run(state):
    if "sigma" in state:
        phi, gx, gy = state["out"]
        status = state["lib"].sr_gravity_solve_static(
            ctypes.byref(state["cfg"]), state["sigma"].data_ptr(), phi.data_ptr(), gx.data_ptr(), gy.data_ptr(), None)
        if status:
            raise RuntimeError("sr_gravity_solve_static: %d" % status)
        return {"phi": phi, "gx": gx, "gy": gy}
    if "feats" in state:
        loss, grad, out = state["learner"].loss_grad(state["feats"], state["target"])
        return {"loss": loss, "grad": grad, "out": out}
    if "batch" in state:
        batch = state["batch"]
        for k, (planes, kappa) in enumerate(state["in"]):
            batch.upload(k, planes, kappa)
        batch.run(state["steps"])
        return [batch.readback(k) for k in range(len(batch))]
    step = state["step"]
    step.upload(state["planes"])
    if state["kappa"] is not None:
        step.upload_opacity(state["kappa"])
    step.run(state["steps"])
    dt = step.read_dt()
    return {"planes": step.readback(state["out"]), "sim_time": dt.sim_time, "dt_next": dt.dt_next}


# ------------------------------------------------------------------------------------------------------- work, bounds
def work(case):
    kind = case["kind"]
    if kind == "gravity":
        n = case["w"] * case["h"]
        return {"bytes": 16.0 * n, "flops": 5.0 * 4 * n * math.log2(4 * n)}
    if kind == "network":
        pix = case["n"] * case["crop"] ** 2
        level, macs = 0, 0.0
        for ci, co, mode, _ in _LAYERS:
            level += {"pool": 1, "up": -1}.get(mode, 0)
            macs += 9.0 * ci * co * pix / 4 ** level
        return {"bytes": 4.0 * (6 * pix + 2 * 110153), "flops": 6.0 * macs}
    total = {"bytes": 0.0, "flops": 0.0}
    for c in _worlds(case) if kind == "batch" else [case]:
        n, ref = c["w"] * c["h"], c["scene"] == "ref"
        b = 8.0 * (14 if ref else 4) * n if c["scene"] != "fld" else 24.0 * n
        f = 0.0
        if c["scene"] != "fld":
            f += (3000.0 if ref else 1000.0) * n
        if c["scene"] in ("disk", "full", "ref"):
            f += 2 * 5.0 * 4 * n * math.log2(4 * n)  # P2 and the half step's solve
        if c["scene"] in ("fld", "full", "ref"):
            b += (4.0 if not ref else 0.0) * n  # the opacity
            f += 200.0 * n
        total["bytes"] += b * c["steps"]
        total["flops"] += f * c["steps"]
    return total


def tolerance(case):
    kind = case["kind"]
    if kind == "network":
        return {"rel": 2e-2, "max": 0.5}   # BF16 operands in every convolution
    if kind == "gravity":
        return {"rel": 2e-5, "max": 2e-3}  # g differences an FP32 potential two cells apart
    # FP32 states summed in 64 bits over some steps; a cell at a limiter's or a vacuum edge's switch moves the most
    return {"rel": 1e-5, "max": 1e-1}


# ------------------------------------------------------------------------------------------------------- 64 bits
class _Gas:
    """The gas scheme in 64 bits: 4 conserved fields and, in reference mode, ten mass fractions. A state `q` is
    (4 + species, h, w): Σ, u, v, Π, X."""

    ZA = [2.0, 0.75, 7 / 12, 9 / 16, 11 / 20, 13 / 24, 15 / 28, 17 / 32, 27 / 56, 1.0]
    ZE = [1.0, 0.5, 0.5, 0.5, 0.5, 0.5, 0.5, 0.5, 26 / 56, 0.0]

    def __init__(self, cfg):
        self.c = cfg
        self.ref = cfg.channels == 14
        self.gm1 = cfg.gamma - 1
        self.eps_floor = cfg.t_floor / cfg.mu / self.gm1
        if self.ref:
            x = torch.exp(torch.linspace(math.log(1e-8), math.log(1e8), 512, dtype=F64, device=DEV))
            self.lnu = [torch.log(self._cold_closed(x, *k)) for k in ((cfg.k1e, cfg.k2e), (cfg.k1n, cfg.k2n))]
            self.za, self.ze = (torch.tensor(t, dtype=F64, device=DEV)[:, None, None] for t in (self.ZA, self.ZE))

    # ---- the EOS
    @staticmethod
    def _cold_closed(x, k1, k2):
        y = k1 / k2 * torch.sqrt(x)
        series = sum((1.0 if k % 2 == 0 else -1.0) * y ** k / k for k in range(2, 12))
        return x * 2 * k2 * k2 / k1 * torch.where(y < 2e-2, series, y - torch.log1p(y))

    @staticmethod
    def _table(lnu, x):
        """ln u interpolated in ln x on 512 nodes from 1e-8 to 1e8."""
        pos = (torch.log(torch.clamp(x, min=1e-300)) - math.log(1e-8)) * (511 / (math.log(1e8) - math.log(1e-8)))
        i = torch.clamp(torch.floor(pos), 0, 510).long()
        a, b = lnu[i], lnu[i + 1]
        u = torch.where(pos < 0, torch.exp(lnu[0]) * (x / 1e-8) ** 2, torch.exp(a + (pos - i) * (b - a)))
        return torch.where(x > 0, u, 0.0)

    @staticmethod
    def _cold_p(x, k1, k2):
        xs = torch.clamp(x, min=1e-300)
        return torch.where(x > 0, 1 / (1 / (k1 * xs * xs) + 1 / (k2 * xs ** 1.5)), 0.0)

    def composition(self, X):
        return (X * self.za).sum(0), (X * self.ze).sum(0)  # 1/μ, Y_e

    def cold_energy(self, s, ye, xn):
        return self._table(self.lnu[0], ye * s) + self._table(self.lnu[1], xn * s)

    def _sides(self, X):
        """1/(μ(γ-1))'s ε floor, and the cold energy and pressure as functions of Σ."""
        if not self.ref:
            return self.eps_floor, (lambda s: 0.0), (lambda s: 0.0)
        inv_mu, ye = self.composition(X)
        c = self.c
        return (c.t_floor * inv_mu, lambda s: self.cold_energy(s, ye, X[9]) / s,
                lambda s: self._cold_p(ye * s, c.k1e, c.k2e) + self._cold_p(X[9] * s, c.k1n, c.k2n))

    def read(self, U):
        X = U[4:]
        floor, ecold, pcold = self._sides(X)
        vac = U[0] < VAC
        s = torch.where(vac, FLOOR, U[0])
        raw = U[3] / s - 0.5 * (U[1] ** 2 + U[2] ** 2) / (s * s) - ecold(s)
        eps = torch.where(vac, floor + 0 * s, torch.maximum(raw, floor + 0 * s))
        u, v = torch.where(vac, 0.0, U[1] / s), torch.where(vac, 0.0, U[2] / s)
        return torch.cat([torch.stack([s, u, v, self.gm1 * s * eps + pcold(s)]), X])

    def cons(self, q):
        floor, ecold, pcold = self._sides(q[4:])
        s = q[0]
        eps = torch.maximum((q[3] - pcold(s)) / s / self.gm1, floor + 0 * s)
        e = s * (eps + ecold(s)) + 0.5 * s * (q[1] ** 2 + q[2] ** 2)
        return torch.cat([torch.stack([s, s * q[1], s * q[2], e]), s * q[4:]])

    def prim(self, U):
        """(primitives, where the state has a density and thermal energy)."""
        ok = (U[0] > 0) & torch.isfinite(U).all(0)
        s = torch.where(ok, U[0], 1.0)
        X = U[4:] / s
        floor, ecold, pcold = self._sides(X)
        raw = U[3] / s - 0.5 * (U[1] ** 2 + U[2] ** 2) / (s * s) - ecold(s)
        ok = ok & (raw > 0)
        p = self.gm1 * s * torch.maximum(raw, floor + 0 * s) + pcold(s)
        return torch.cat([torch.stack([s, U[1] / s, U[2] / s, p]), X]), ok

    # ---- slopes, prediction, fluxes
    def _limited(self, l, c, r):
        a, b = c - l, r - c
        m = torch.minimum(a.abs(), b.abs())
        if self.c.limiter == "mc":
            m = torch.minimum(0.5 * (a + b).abs(), 2 * m)
        return torch.where(a * b <= 0, 0.0, torch.copysign(m, a))

    def slope(self, l, c, r):
        s = self._limited(l, c, r)
        if self.ref:
            central = 0.5 * (r[4:] - l[4:])
            ratio = torch.where(central != 0, s[4:] / torch.where(central != 0, central, 1.0), 1.0)
            s = torch.cat([s[:4], torch.clamp(ratio.min(0)[0], max=1.0) * central])
        if self.c.thermal_bracket:
            hottest = torch.maximum(torch.maximum(l[3] / l[0], c[3] / c[0]), r[3] / r[0])
            fine = torch.ones_like(hottest, dtype=torch.bool)
            for f in (-0.5, 0.5):
                fine &= c[3] + f * s[3] <= 2 * hottest * (c[0] + f * s[0])
            s[0] = torch.where(fine, s[0], 0.0)
            s[3] = torch.where(fine, s[3], 0.0)
        return s

    @staticmethod
    def flux(q, e, d):
        un, m = q[1 + d], q[0] * q[1 + d]
        f = [m, m * q[1], m * q[2], (e + q[3]) * un]
        f[1 + d] = f[1 + d] + q[3]
        return torch.cat([torch.stack(f), m * q[4:]])

    def predicted(self, Q, half, g):
        """Each cell's four faces (left, right, up, down) as (U, q), and its half-step Σ, Σu, Σv, for the cells one in
        from Q's rim; g (2, ...) there or None."""
        c = Q[:, 1:-1, 1:-1]
        sx = self.slope(Q[:, 1:-1, :-2], c, Q[:, 1:-1, 2:])
        sy = self.slope(Q[:, :-2, 1:-1], c, Q[:, 2:, 1:-1])
        W = [c - 0.5 * sx, c + 0.5 * sx, c - 0.5 * sy, c + 0.5 * sy]
        UW = [self.cons(q) for q in W]
        f = [self.flux(W[k], UW[k][3], k // 2) for k in range(4)]
        delta = half * ((f[0] - f[1]) + (f[2] - f[3]))
        mid = torch.stack([c[0], c[0] * c[1], c[0] * c[2]]) + delta[:3]
        faces = []
        for q, U in zip(W, UW):
            d = delta
            if g is not None:
                d = delta.clone()
                d[1] += half * q[0] * g[0]
                d[2] += half * q[0] * g[1]
                d[3] += half * q[0] * ((q[1] + 0.5 * half * g[0]) * g[0] + (q[2] + 0.5 * half * g[1]) * g[1])
            U1 = U + d
            q1, ok = self.prim(U1)
            faces.append((torch.where(ok, U1, U), torch.where(ok, q1, q)))
        if g is not None:
            mid[1] += half * c[0] * g[0]
            mid[2] += half * c[0] * g[1]
        return faces, mid

    def hll(self, L, R, d):
        (Ul, l), (Ur, r) = L, R
        gamma = 2.0 if self.ref else self.c.gamma
        cl, cr = (torch.sqrt(torch.clamp(gamma * q[3] / q[0], min=0)) for q in (l, r))
        sl = torch.minimum(l[1 + d] - cl, r[1 + d] - cr)
        sr = torch.maximum(l[1 + d] + cl, r[1 + d] + cr)
        fl, fr = self.flux(l, Ul[3], d)[:4], self.flux(r, Ur[3], d)[:4]
        mid = (sr * fl - sl * fr + sl * sr * (Ur[:4] - Ul[:4])) / (sr - sl)
        f = torch.where(sl >= 0, fl, torch.where(sr <= 0, fr, mid))
        return torch.cat([f, f[0] * torch.where(f[0] > 0, l[4:], r[4:])])

    def _ghosted(self, q):
        for axis in (2, 1):  # columns, then rows over the padded width
            n, comp = q.shape[axis], 1 if axis == 2 else 2
            if self.c.edge == "bounce":
                lo, hi = q.narrow(axis, 0, 2).flip(axis).clone(), q.narrow(axis, n - 2, 2).flip(axis).clone()
                lo[comp], hi[comp] = -lo[comp], -hi[comp]
            else:
                lo, hi = (torch.cat([q.narrow(axis, k, 1)] * 2, axis).clone() for k in (0, n - 1))
                lo[comp], hi[comp] = torch.clamp(lo[comp], max=0), torch.clamp(hi[comp], min=0)
            q = torch.cat([lo, q, hi], axis)
        return q

    def _face_fluxes(self, faces, axis):
        """Fluxes at the n + 1 faces of an axis (0 x, 1 y), walls or open edges at its ends."""
        dim = 2 - axis
        n = faces[0][1].shape[dim] - 2
        across = 1 if axis == 0 else 2
        def cut(t):  # drop the other axis's ghost cells
            return t.narrow(across, 1, t.shape[across] - 2)
        low, high = [tuple(cut(t) for t in faces[2 * axis + k]) for k in (0, 1)]
        f = self.hll(tuple(t.narrow(dim, 0, n + 1) for t in high), tuple(t.narrow(dim, 1, n + 1) for t in low), axis)
        for k, own, sign in ((0, low[1].narrow(dim, 1, 1), 1.0), (n, high[1].narrow(dim, n, 1), -1.0)):
            wall = torch.zeros_like(f.narrow(dim, k, 1))
            wall[1 + axis] = own[3]
            at = f.narrow(dim, k, 1)
            inflow = sign * at[0] > 0
            at.copy_(wall if self.c.edge == "bounce" else torch.where(inflow, wall, at))
        return f

    def step(self, U, dt, gravity=None, rad=None):
        """P4; `gravity`: the solver of Σ -> φ, gx, gy, run on the start state and the half step."""
        q = self.read(U)
        g = None if gravity is None else torch.stack(gravity(U[0])[1:])
        gp = None if g is None else F.pad(g[None], (1, 1, 1, 1), mode="replicate")[0]
        faces, mid = self.predicted(self._ghosted(q), 0.5 * dt, gp)
        fx, fy = self._face_fluxes(faces, 0), self._face_fluxes(faces, 1)
        mid = mid[:, 1:-1, 1:-1]
        vac = U[0] < VAC
        pv = F.pad(vac, (1, 1, 1, 1), value=True)
        empty = vac & pv[1:-1, :-2] & pv[1:-1, 2:] & pv[:-2, 1:-1] & pv[2:, 1:-1]
        start = torch.cat([U[:4], U[0] * U[4:]])
        start = torch.where(vac, self.cons(q), start)
        new = start - dt * ((fx[:, :, 1:] - fx[:, :, :-1]) + (fy[:, 1:] - fy[:, :-1]))
        if gravity is not None:
            src = torch.where(empty, 0.0, 0.5 * (U[0] + new[0]))
            src = torch.where(src >= VAC, src, 0.0)
            phi, gx, gy = gravity(src)
            kick = torch.stack([dt * src * gx, dt * src * gy])
            net = torch.where(empty, 0.0, kick).sum((1, 2))
            energy = torch.zeros_like(phi)
            for axis, f in ((0, fx), (1, fy)):
                d = 1 - axis
                n = phi.shape[d]
                pad = (1, 1, 0, 0) if axis == 0 else (0, 0, 1, 1)
                P = F.pad(phi[None, None], pad, mode="replicate")[0, 0]
                M = F.pad(mid[None], pad, mode="replicate")[0]
                k, e_low, e_high = self._face_work(f[0], *(M[0].narrow(d, i, n + 1) for i in (0, 1)),
                                                   *(M[1 + axis].narrow(d, i, n + 1) for i in (0, 1)),
                                                   P.narrow(d, 0, n + 1) - P.narrow(d, 1, n + 1), dt)
                kick[axis] += k.narrow(d, 1, n) - k.narrow(d, 0, n)
                energy += e_low.narrow(d, 1, n) + e_high.narrow(d, 0, n)
            new[1:3] += kick
            new[3] += energy
        push = None
        if rad is not None:
            d = dt * self.c.kappa0 * (1 + U[4]) * U[0] * rad / self.c.c_sb
            d = torch.where(vac | empty, 0.0, d)
            push = self._push_share(new, d) * d
            new[1:3] += push
        new = torch.cat([new[:4], new[4:] / new[0]])
        new = torch.where(empty, U, new)
        if push is not None:
            size = torch.hypot(push[0], push[1])
            if float(size.sum()) > 0:
                new[1:3] -= size * (push.sum((1, 2)) / size.sum())[:, None, None]
        if gravity is not None and float(src.max()) > 0:
            at = int(torch.argmax(src))
            new[1].view(-1)[at] -= net[0]
            new[2].view(-1)[at] -= net[1]
        return new, g

    def _push_share(self, U, d):
        d2 = (d * d).sum(0)
        s = U[0]
        floor, ecold, _ = self._sides(U[4:] / s)
        a = s * (U[3] / s - 0.5 * (U[1] ** 2 + U[2] ** 2) / (s * s) - ecold(s) - floor)
        q = U[1] * d[0] + U[2] * d[1]
        disc = torch.sqrt(torch.clamp(q * q + 2 * s * a * d2, min=0))
        root = torch.where(q >= 0, 2 * s * a / torch.clamp(q + disc, min=1e-300),
                           (disc - q) / torch.clamp(d2, min=1e-300))
        return torch.where(d2 == 0, 1.0, torch.where(a > 0, torch.clamp(root, max=1.0), 0.0))

    @staticmethod
    def _face_work(q, sl, sh, pl, ph, d, dt):
        a, b = torch.clamp(sl, min=0), torch.clamp(sh, min=0)
        w = torch.where(a + b > 0, a / torch.where(a + b > 0, a + b, 1.0), 0.5)
        extra = dt * (q - 0.5 * (pl + ph)) * d
        both = (a > 0) & (b > 0)
        a1, b1 = torch.where(both, a, 1.0), torch.where(both, b, 1.0)
        ul, uh, inv = pl / a1, ph / b1, 1 / a1 + 1 / b1
        du = ul - uh
        c = torch.where((extra < 0) & both, torch.minimum(-extra, 0.25 * du * du / inv), 0.0)
        on = c > 0
        den = du + torch.copysign(torch.sqrt(torch.clamp(du * du - 2 * inv * c, min=0)), du)
        kick = torch.where(on, -2 * c / torch.where(on, den, 1.0), 0.0)
        el, eh = ul * kick + 0.5 * kick * kick / a1, -uh * kick + 0.5 * kick * kick / b1
        rest = extra + c
        return kick, 0.5 * dt * pl * d + w * rest + el, 0.5 * dt * ph * d + (1 - w) * rest + eh

    def floors(self, U):
        X = U[4:]
        if self.ref:
            X = torch.clamp(X, min=0)
            X = X / X.sum(0)
        floor, ecold, _ = self._sides(X)
        floor = floor + 0 * U[0]
        vac = U[0] < VAC
        s = torch.where(vac, FLOOR, U[0])
        raw = U[3] / s - 0.5 * (U[1] ** 2 + U[2] ** 2) / (s * s) - ecold(s)
        e = torch.where(vac, FLOOR * (floor + ecold(s)), U[3] + s * torch.clamp(floor - raw, min=0))
        return torch.cat([torch.stack([s, torch.where(vac, 0.0, U[1]), torch.where(vac, 0.0, U[2]), e]), X])

    def dt(self, U, g):
        if self.c.dt_fixed > 0:
            return self.c.dt_fixed
        q = self.read(U)
        c = torch.sqrt(torch.clamp((2.0 if self.ref else self.c.gamma) * q[3] / q[0], min=0))
        dt = self.c.cfl / float((q[1].abs() + q[2].abs() + 2 * c).max())
        top = 0.0 if g is None else float(torch.hypot(g[0], g[1]).max())
        return min(dt, self.c.eta_g / math.sqrt(top)) if top > 0 else dt


class _Gravity:
    """φ and g = -∇φ (central differences of φ on the box and one ring) of Σ by the zero-padded FFT convolution."""

    def __init__(self, cfg):
        w, h = cfg.width, cfg.height
        self.w, self.h = w, h
        self.px, self.py = (1 << (2 * n + 1).bit_length() for n in (w, h))
        dx, dy = (torch.arange(p, device=DEV, dtype=F64) for p in (self.px, self.py))
        dx, dy = torch.minimum(dx, self.px - dx), torch.minimum(dy, self.py - dy)
        r2 = dx[None, :] ** 2 + dy[:, None] ** 2
        if cfg.kernel == "softened":
            k = 1 / torch.sqrt(r2 + cfg.softening ** 2)
        else:
            r2[0, 0] = 1.0
            k = 1 / torch.sqrt(r2)
            k[0, 0] = 4 * math.log(1 + math.sqrt(2))
        self.k = torch.fft.rfft2(-cfg.G * k)

    def __call__(self, sigma):
        src = torch.where(sigma >= VAC, sigma, 0.0)
        f = torch.fft.irfft2(torch.fft.rfft2(F.pad(src, (1, self.px - self.w - 1, 1, self.py - self.h - 1))) * self.k,
                             s=(self.py, self.px))[: self.h + 2, : self.w + 2]
        return (f[1:-1, 1:-1].contiguous(), -0.5 * (f[1:-1, 2:] - f[1:-1, :-2]), -0.5 * (f[2:, 1:-1] - f[:-2, 1:-1]))


def _heat_step(gas, U, kappa, dt):
    """P5: one backward-Euler step of u = a_r T⁴ with the flux law frozen at its start; (U, the mean face flux per axis)."""
    c = gas.c
    ref = gas.ref
    w, h = c.width, c.height
    is_gas = U[0] >= VAC
    s = torch.where(is_gas, U[0], FLOOR)
    inv_c = gas.composition(U[4:])[0] if ref else torch.full_like(s, 1 / (c.mu * gas.gm1))
    floor, ecold, _ = gas._sides(U[4:])
    eps = torch.maximum(U[3] / s - 0.5 * (U[1] ** 2 + U[2] ** 2) / (s * s) - ecold(s), floor + 0 * s)
    t0 = torch.where(is_gas, eps / inv_c, c.t_floor)
    kap = c.kappa0 * (1 + U[4]) if ref else (kappa if kappa is not None else torch.full_like(s, c.kappa0))
    cap = s * inv_c
    u_vac = c.a_r * c.t_floor ** 4
    K, nb = [], []
    for axis in (0, 1):
        d = 1 - axis
        pad = (1, 1, 0, 0) if axis == 0 else (0, 0, 1, 1)
        n = s.shape[d]

        def ends(t, value):
            p = F.pad(t, pad, value=value)
            return p.narrow(d, 0, n + 1), p.narrow(d, 1, n + 1)
        ga, gb = ends(is_gas, False)
        ta, tb = ends(torch.where(is_gas, t0, c.t_floor), c.t_floor)
        sa, sb = ends(s, FLOOR)
        ka, kb = ends(kap, 0.0)
        ka, kb = torch.where(ga, ka, kb), torch.where(gb, kb, ka)  # a vacuum side takes the gas side's κ
        era, erb = c.a_r * ta ** 4, c.a_r * tb ** 4
        ks, fe = 0.5 * (ka * sa + kb * sb), 0.5 * (era + erb)
        on = ga | gb
        ks = torch.where(on, ks, 1.0)
        R = (erb - era).abs() / (ks * fe)
        K.append(torch.where(on, c.c_sb * (2 + R) / (6 + 3 * R + R * R) / ks, 0.0))
        nb.append(ga & gb)
    inner = [torch.where(b, k, 0.0) for k, b in zip(K, nb)]

    def over(x, y):
        return (x[:, :-1] + x[:, 1:]) + (y[:-1] + y[1:])
    kvac = torch.where(is_gas, over(*K) - over(*inner), 0.0)
    ksum = torch.where(is_gas, over(*inner), 0.0)
    kx, ky = inner[0][:, 1:-1], inner[1][1:-1]

    def coupled(x):  # Σ_f D (x_i - x_j)
        out = torch.zeros_like(x)
        f = kx * (x[:, 1:] - x[:, :-1])
        out[:, 1:] += f
        out[:, :-1] -= f
        f = ky * (x[1:] - x[:-1])
        out[1:] += f
        out[:-1] -= f
        return out
    heat = torch.where(is_gas, cap / dt, 0.0)
    t, u = t0.clone(), c.a_r * t0 ** 4
    heat0 = float((cap * t0)[is_gas].sum())
    for _ in range(60):
        slope = 1 / (4 * c.a_r * t ** 3)
        mass = torch.where(is_gas, heat * slope + kvac, 1.0)
        diag = mass + ksum
        b = torch.where(is_gas, heat * slope * u - heat * (t - t0) + kvac * u_vac, 0.0)
        x = torch.where(is_gas, u, 0.0)
        r = b - mass * x - coupled(x)
        z = r / diag
        p, rz = z.clone(), (r * z).sum()
        stop = 1e-22 * float((heat * slope * u * u).sum())
        for it in range(20000):
            if it % 8 == 0 and float(rz) <= stop:
                break
            q = mass * p + coupled(p)
            alpha = rz / torch.clamp((p * q).sum(), min=1e-300)
            x += alpha * p
            r -= alpha * q
            z = r / diag
            new = (r * z).sum()
            p = z + new / torch.clamp(rz, min=1e-300) * p
            rz = new
        nt = torch.sqrt(torch.sqrt(torch.clamp(x, min=u_vac) / c.a_r))
        nt = torch.where(is_gas, torch.minimum(torch.maximum(nt, 0.5 * t), 2 * t), t)
        moved = float((cap * (nt - t).abs())[is_gas].sum())
        step = float(((nt - t).abs() / t).max())
        t, u = nt, c.a_r * nt ** 4
        if moved <= 1e-11 * heat0 and step <= 1e-9:
            break
    radiated = float((dt * kvac * (u - u_vac)).sum())
    gained, held = float((cap * (t - t0))[is_gas].sum()), float((cap * t)[is_gas].sum())
    delta = -(gained + radiated) / held
    U = U.clone()
    U[3] = torch.where(is_gas, U[3] + cap * ((1 + delta) * t - t0), U[3])
    v = torch.where(is_gas, u, u_vac)
    px, py = F.pad(v, (1, 1, 0, 0), value=u_vac), F.pad(v, (0, 0, 1, 1), value=u_vac)
    fx, fy = -K[0] * (px[:, 1:] - px[:, :-1]), -K[1] * (py[1:] - py[:-1])
    return U, torch.stack([0.5 * (fx[:, :-1] + fx[:, 1:]), 0.5 * (fy[:-1] + fy[1:])])


def _exact_world(case, P, kappa, dt_fixed):
    cfg = _config(case, dt_fixed)
    gas = _Gas(cfg)
    gravity = _Gravity(cfg) if cfg.gravity else None
    U = P.to(F64)
    kappa = None if kappa is None else kappa.to(F64)
    g = None if gravity is None else torch.stack(gravity(U[0])[1:])
    dt, time, rad = gas.dt(U, g), 0.0, None
    for _ in range(case["steps"]):
        time += dt
        if cfg.hydro:
            U, g = gas.step(U, dt, gravity, rad)
        if cfg.heat:
            U, flux = _heat_step(gas, U, kappa, dt)
            rad = flux if gas.ref else None
        U = gas.floors(U)
        dt = gas.dt(U, g)
    return {"planes": U, "sim_time": time, "dt_next": dt}


def _exact_network(case, seed):
    theta, feats, target = (t.to(F64) for t in _network_inputs(case, seed))
    theta.requires_grad_(True)
    outs, at, x = [], 0, feats
    for k, (ci, co, mode, relu) in enumerate(_LAYERS):
        wgt = theta[at:at + co * 9 * ci].reshape(co, 3, 3, ci).permute(0, 3, 1, 2)
        bias = theta[at + co * 9 * ci:at + co * 9 * ci + co]
        at += co * 9 * ci + co
        if mode == "pool":
            hh, ww = x.shape[2:]
            pad = (0, ww % 2, 0, hh % 2)
            x = F.avg_pool2d(F.pad(x, pad), 2) / F.avg_pool2d(F.pad(torch.ones_like(x[:1, :1]), pad), 2)
        elif mode == "up":
            hh, ww = outs[_SKIP[k + 1]].shape[2:]
            x = x.repeat_interleave(2, 2).repeat_interleave(2, 3)[:, :, :hh, :ww]
        elif mode == "skip":
            x = x + outs[_SKIP[k]]
        x = F.conv2d(x, wgt, bias, padding=1)
        x = F.relu(x) if relu else x
        outs.append(x)
    y = x[:, 0]

    def op(v):  # the crop's Jacobi-scaled operator
        dx, dy = feats[:, 1, :, :-1], feats[:, 2, :-1]
        out = v - F.pad(dx * v[:, :, 1:], (0, 1)) - F.pad(dx * v[:, :, :-1], (1, 0))
        return out - F.pad(dy * v[:, 1:], (0, 0, 0, 1)) - F.pad(dy * v[:, :-1], (0, 0, 1, 0))
    energy = (target * op(target)).sum((1, 2))
    d = target - y
    loss = ((d * op(d)).sum((1, 2)) / (energy + 1e-3 * energy.mean())).mean()
    loss.backward()
    return {"loss": float(loss), "grad": theta.grad, "out": y.detach()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "gravity":
        sig = _disk(case["w"], case["h"], _gen(seed), 1.0)[0].to(torch.float32).to(F64)
        cfg = Config(width=case["w"], height=case["h"], gravity=True, kernel=case["kernel"])
        return dict(zip(("phi", "gx", "gy"), (t.contiguous() for t in _Gravity(cfg)(sig))))
    if kind == "network":
        return _exact_network(case, seed)
    if kind == "batch":
        worlds, scenes = _batch_scenes(case, seed)
        return [_exact_world(c, *s)["planes"] for c, s in zip(worlds, scenes)]
    return _exact_world(case, *_scene(case, seed))
