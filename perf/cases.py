"""The work a user of this framework has it do, as cases that can be timed.

Every case is one pass through the public entry points: a simulation loaded with
particles and advanced some steps, an ensemble advanced, forces on a particle
set, an offload step on host buffers, a training step of the learned correction.
``exact`` restates each of them in 64-bit torch, without this repository's code.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from stardust_b200 import _lib as L
from stardust_b200.ensemble import Ensemble, member_config
from stardust_b200.learned import LAYOUT, N_PARAMS, Correction, PMField, init_params
from stardust_b200.sim import Sim, SimConfig

DEV = "cuda"
ORDERS = {"tiled": L.SD_ORDER_TILED, "rowmajor": L.SD_ORDER_ROWMAJOR, "morton": L.SD_ORDER_MORTON}
BATCHES = 4  # optimiser steps of one training pass


def _steps(name, scene, n, grid, steps, dt, order="tiled", boundary="periodic", integrator="kd", units="newton",
           soft=1.0, learned=False, hydro=False, diagnostics=False):
    c = {"kind": "steps", "scene": scene, "n": n, "grid": grid, "steps": steps, "dt": dt, "order": order,
         "boundary": boundary, "integrator": integrator, "units": units, "soft": soft, "learned": learned,
         "hydro": hydro, "diagnostics": diagnostics}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one step of a tiny scene, called on its own: a caller's own loop with work between
        # steps. Launches and latency are all of it.
        {"name": "step_16k_32", "kind": "step", "scene": "disk", "n": 16384, "grid": 32, "dt": 1e-3, "order": "tiled"},
        # the single disk galaxy: 262,144 particles on 64^3, ten steps of 1e-3
        _steps("disk_262k_64", "disk", 262144, 64, 10, 1e-3),
        # the two-galaxy encounter: 4M particles on 256^3, strongly clustered, many keys change
        _steps("pair_4m_256", "pair", 4194304, 256, 10, 5e-4),
        # the cosmic web, the headline workload and the largest: 16M particles on 512^3 with
        # energies and momentum recorded every step
        _steps("web_16m_512", "web", 16777216, 512, 10, 1e-3, diagnostics=True),
        # the coarse grid with the learned correction in every step: 2M particles on 128^3
        _steps("learned_2m_128", "web", 2097152, 128, 10, 1e-3, learned=True),
        # the default configuration (row-major order, reference units, 2,000,000 particles on
        # 128^3), stepped by the CFL-clamped step() as an interactive program does
        {"name": "default_2m_128", "kind": "auto", "scene": "ball", "n": 2000000, "grid": 128, "steps": 4,
         "order": "rowmajor", "soft": 3.0},
        # the reference's own order for a larger scene of odd size, many steps in one call
        _steps("rowmajor_8m_256", "web", 8000003, 256, 10, 1e-3, order="rowmajor", soft=2.0),
        # a galaxy in an isolated box: the reference's default boundary, 2 x 128 = 256^3 transforms
        _steps("isolated_1m_128", "disk", 1000003, 128, 8, 1e-3, order="rowmajor", boundary="isolated"),
        # 64 independent scenes of uneven sizes advanced together
        {"name": "ensemble_64", "kind": "ensemble", "count": 64, "n_min": 16384, "n_max": 1048576, "steps": 5,
         "dt": 5e-4},
        # forces of a particle set on a fine grid: what training pairs and force checks are made of
        {"name": "accel_2m_512", "kind": "accel", "scene": "web", "n": 2097152, "grid": 512, "soft": 4.0},
        # a program with its particles in host memory: four pipelined offload steps
        {"name": "offload_1m_128", "kind": "offload", "scene": "pair", "n": 1048576, "grid": 128, "calls": 4,
         "dt": 5e-4},
        # training the correction: gradients and Adam steps on batches of 16,384 rows
        {"name": "train_16384", "kind": "train", "rows": 16384},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tiled", "tiled", "tiled", "learned", "order", "order", "isolated", "isolated", "step", "auto",
                       "ensemble", "accel", "offload", "train"])
    scene = rng.choice(["disk", "pair", "web", "web", "ball"])
    soft = rng.choice([1.0, 1.5, 2.0, 3.0])
    if kind == "tiled":
        g = rng.choice([16, 32, 64, 128, 256, 512])
        n = _log(rng, max(1000, g ** 3 // 64), min(16000000, 4 * g ** 3))
        return _steps(None, scene, n, g, 10 if g < 512 else 6, rng.choice([1e-3, 5e-4]), soft=soft,
                      integrator=rng.choice(["kd", "kd", "kdk"]), units=rng.choice(["newton", "newton", "reference"]),
                      diagnostics=rng.random() < 0.3)
    if kind == "learned":
        g = rng.choice([64, 128, 256])
        return _steps(None, scene, _log(rng, g ** 3 // 8, min(4000000, 2 * g ** 3)), g, 10, 1e-3, soft=soft, learned=True)
    if kind == "order":
        g = rng.choice([32, 64, 128, 256, 512])
        n = _log(rng, max(4000, g ** 3 // 32), min(8000000, 4 * g ** 3))
        return _steps(None, scene, n, g, 10 if g < 512 else 4, 1e-3, soft=soft,
                      order=rng.choice(["rowmajor", "rowmajor", "morton"]), units=rng.choice(["newton", "reference"]))
    if kind == "isolated":
        g = rng.choice([16, 32, 64, 128, 256])
        n = _log(rng, max(1000, g ** 3 // 32), min(4000000, 4 * g ** 3))
        return _steps(None, rng.choice(["disk", "pair", "ball"]), n, g, 8 if g < 256 else 4, 1e-3, soft=soft,
                      order=rng.choice(["rowmajor", "tiled"]), boundary="isolated", hydro=rng.random() < 0.4)
    if kind == "step":
        g = rng.choice([16, 32, 64])
        return {"kind": "step", "scene": scene, "n": _log(rng, 2000, 2 * g ** 3), "grid": g, "dt": 1e-3,
                "order": rng.choice(["tiled", "rowmajor"])}
    if kind == "auto":
        g = rng.choice([32, 64, 128, 256])
        return {"kind": "auto", "scene": scene, "n": _log(rng, g ** 3 // 8, min(8000000, 2 * g ** 3)), "grid": g,
                "steps": 4, "order": rng.choice(["rowmajor", "rowmajor", "tiled"]), "soft": soft}
    if kind == "ensemble":
        lo = _log(rng, 4096, 65536)
        return {"kind": "ensemble", "count": rng.randint(4, 64), "n_min": lo, "n_max": lo * rng.randint(2, 16),
                "steps": 5, "dt": 5e-4}
    if kind == "accel":
        g = rng.choice([64, 128, 256, 512])
        return {"kind": "accel", "scene": scene, "n": _log(rng, 50000, 4000000), "grid": g, "soft": g / 128.0}
    if kind == "offload":
        g = rng.choice([64, 128, 256])
        return {"kind": "offload", "scene": scene, "n": _log(rng, 50000, 4000000), "grid": g, "calls": 3, "dt": 5e-4}
    return {"kind": "train", "rows": 16 * _log(rng, 64, 4096)}


# ---- scenes (made on the GPU from the seed) --------------------------------------------


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 13)
    return g


def _galaxy(n, g, mass=1.0):
    """Exponential disk (80 %) and Plummer bulge (20 %), circular velocities with 5 % dispersion."""
    nd = int(round(0.8 * n))
    nb = n - nd
    u = torch.rand(3, nd, generator=g, device=DEV).clamp_min_(1e-7)
    R = -0.08 * (u[0].log() + u[1].log())
    R = torch.where(R > 0.3, 0.3 * torch.sqrt(u[2]), R)
    th = 2 * math.pi * torch.rand(nd, generator=g, device=DEV)
    z = 0.008 * torch.atanh((2 * torch.rand(nd, generator=g, device=DEV) - 1).clamp_(-0.99999, 0.99999))
    disk = torch.stack([R * th.cos(), R * th.sin(), z], 1)
    ub = torch.rand(nb, generator=g, device=DEV).clamp_(1e-5, 0.99)
    rb = 0.03 / torch.sqrt(ub.pow(-2.0 / 3.0) - 1.0)
    d = torch.randn(nb, 3, generator=g, device=DEV)
    bulge = d / d.norm(dim=1, keepdim=True).clamp_min(1e-6) * rb.clamp_max(0.3)[:, None]
    x = torch.cat([disk, bulge])
    r = x.norm(dim=1)
    menc = torch.empty_like(r)
    menc[r.argsort()] = torch.arange(1, n + 1, device=DEV, dtype=torch.float32) * (mass / n)
    v = torch.randn(n, 3, generator=g, device=DEV)
    vc = torch.sqrt(menc[:nd] / r[:nd].clamp_min(1e-4))
    v[:nd] = torch.stack([-th.sin(), th.cos(), torch.zeros_like(th)], 1) * vc[:, None] + 0.05 * vc[:, None] * v[:nd]
    v[nd:] *= torch.sqrt(menc[nd:] / (3.0 * r[nd:].clamp_min(0.03)))[:, None]
    return x, v


def _scene(kind, n, seed):
    """float32 (n, 4) positions in [0, 1) and velocities; vel.w carries the particle's number."""
    g = _gen(seed)
    if kind == "disk":
        x, v = _galaxy(n, g)
        x = x + 0.5
    elif kind == "pair":
        n1 = n // 2
        a, va = _galaxy(n1, g, 0.5)
        b, vb = _galaxy(n - n1, g, 0.5)
        parts = []
        for (y, w), inc, s in (((a, va), 30.0, 0.5), ((b, vb), -60.0, -0.5)):
            c, q = math.cos(math.radians(inc)), math.sin(math.radians(inc))
            m = torch.tensor([[1.0, 0, 0], [0, c, q], [0, -q, c]], device=DEV)
            parts.append((y @ m + 0.5 + torch.tensor([0.4 * s, 0, 0], device=DEV),
                          w @ m + torch.tensor([-1.936 * s, 1.118 * s, 0], device=DEV)))
        x, v = torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts])
    elif kind == "ball":
        d = torch.randn(n, 3, generator=g, device=DEV)
        r = 0.45 * torch.rand(n, generator=g, device=DEV).pow(1.0 / 3.0)
        x = d / d.norm(dim=1, keepdim=True).clamp_min(1e-6) * r[:, None]
        x = 0.5 + x + 0.04 * torch.sin(12.566 * x.roll(1, 1))
        v = 0.02 * torch.randn(n, 3, generator=g, device=DEV)
    else:  # web: a lattice displaced by a Gaussian field with P(k) ~ k^-2, 0.5 lattice cells rms
        s = max(4, int(math.ceil(n ** (1.0 / 3.0) - 1e-9)))
        k = torch.fft.fftfreq(s, 1.0 / s, device=DEV)
        kr = torch.arange(s // 2 + 1, device=DEV, dtype=torch.float32)
        kz, ky, kx = k[:, None, None], k[None, :, None], kr[None, None, :]
        k2 = kz * kz + ky * ky + kx * kx
        k2[0, 0, 0] = 1.0
        delta = torch.fft.rfftn(torch.randn(s, s, s, generator=g, device=DEV)) / k2.pow(1.5)
        delta[0, 0, 0] = 0.0
        psi = torch.stack([torch.fft.irfftn(1j * kk * delta, s=(s, s, s)) for kk in (kx, ky, kz)], -1).reshape(-1, 3)
        del delta, k2
        psi *= 0.5 / s / psi.square().sum(1).mean().sqrt()
        q = (torch.arange(s, device=DEV, dtype=torch.float32) + 0.5) / s
        zz, yy, xx = torch.meshgrid(q, q, q, indexing="ij")
        x = torch.stack([xx, yy, zz], -1).reshape(-1, 3) + psi
        v = psi * math.sqrt(4.0 * math.pi)
        if s ** 3 > n:
            keep = torch.div(torch.arange(n, device=DEV) * s ** 3, n, rounding_mode="floor")
            x, v = x[keep], v[keep]
    pos = torch.zeros(n, 4, device=DEV)
    vel = torch.zeros(n, 4, device=DEV)
    pos[:, :3] = x - x.floor()
    pos[:, :3][pos[:, :3] >= 1.0] = 0.0
    vel[:, :3] = v - v.mean(0)
    vel[:, 3] = torch.arange(n, device=DEV, dtype=torch.float32)
    return pos, vel


def _members(case):
    """The recipes of an ensemble: sizes spread over their logarithm, the grid matched to the size."""
    out = []
    for i in range(case["count"]):
        t = (i * 0.61803398875 + 0.5) % 1.0
        n = int(case["n_min"] * (case["n_max"] / case["n_min"]) ** t) | 1
        out.append(("disk" if i % 2 else "web", n, 32 if n < 65536 else (64 if n < 524288 else 128)))
    return out


def _config(case):
    k = case["kind"]
    newton = case.get("units", "reference" if k == "auto" else "newton") == "newton"
    hydro = 1 if case.get("hydro") else 0
    return SimConfig(particle_count=case["n"], grid_size=case["grid"], softening_cells=case.get("soft", 1.0),
                     units=L.SD_UNITS_NEWTON if newton else L.SD_UNITS_REFERENCE, order=ORDERS[case.get("order", "tiled")],
                     boundary=L.SD_BOUNDARY_ISOLATED if case.get("boundary") == "isolated" else L.SD_BOUNDARY_PERIODIC,
                     integrator=L.SD_INT_KDK if case.get("integrator") == "kdk" else L.SD_INT_KD,
                     sort_interval=1, keep_density=1 if k == "auto" else 0, preset=L.SD_PRESET_EMPTY,
                     diagnostics=1 if case.get("diagnostics") else 0, pressure_enabled=hydro, cooling_enabled=hydro)


def _correction(case, seed):
    return Correction(init_params(int(seed) % 1000003), 1e-2, case["soft"] / case["grid"], case["grid"], 4 * case["grid"])


# ---- preparation and passes ------------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _prepare_train(case, seed)
    if kind == "ensemble":
        return _prepare_ensemble(case, seed)
    pos, vel = _scene(case["scene"], case["n"], seed)
    if kind == "accel":
        return {"kind": kind, "field": PMField(pos, case["grid"], case["soft"] / case["grid"])}
    stream = torch.cuda.Stream()
    sim = Sim(0)
    sim.set_stream(stream)
    sim.init(_config(case))
    if case.get("learned"):
        sim.set_correction(_correction(case, seed))
    st = {"kind": kind, "case": case, "sim": sim, "stream": stream, "pos": pos, "vel": vel}
    if kind == "offload":
        st["pos"], st["vel"] = pos.cpu().pin_memory(), vel.cpu().pin_memory()
        st["out"] = [(torch.empty_like(st["pos"]).pin_memory(), torch.empty_like(st["vel"]).pin_memory())
                     for _ in range(case["calls"])]
        return st
    st["slots"] = (torch.empty_like(pos), torch.empty_like(vel))
    if kind != "step":
        st["by_id"] = (torch.zeros_like(pos), torch.zeros_like(vel))
    torch.cuda.synchronize()
    return st


def _prepare_ensemble(case, seed):
    ens = Ensemble(0)
    base, total = [], 0
    for i, (scene, n, grid) in enumerate(_members(case)):
        pos, vel = _scene(scene, n, int(seed) * 101 + i)
        torch.cuda.synchronize()
        ens.add(member_config({"n": n, "grid": grid}), pos, vel)
        base.append(torch.full((n,), total, dtype=torch.int64, device=DEV))
        total += n
    ens.synchronize()
    slots = [torch.empty(total, 4, device=DEV) for _ in range(2)]
    views, at = [], 0
    for i, (_, n, _) in enumerate(_members(case)):
        views.append((ens.scene(i), slots[0][at:at + n], slots[1][at:at + n]))
        at += n
    return {"kind": "ensemble", "case": case, "ens": ens, "views": views, "slots": slots, "base": torch.cat(base),
            "by_id": [torch.zeros(total, 4, device=DEV) for _ in range(2)]}


def _prepare_train(case, seed):
    g = _gen(seed)
    n = case["rows"] * BATCHES
    x = torch.zeros(n, 32, device=DEV)
    x[:, :27] = 0.7 * torch.randn(n, 1, generator=g, device=DEV) - 0.3 + 0.4 * torch.randn(n, 27, generator=g, device=DEV)
    x[:, 27:30] = torch.rand(n, 3, generator=g, device=DEV) - 0.5
    x = x.bfloat16()
    a = 0.3 * torch.randn(32, 3, generator=g, device=DEV)
    t = (torch.tanh(x.float() @ a) + 0.5 * torch.randn(n, 3, generator=g, device=DEV)).contiguous()
    p0 = torch.from_numpy(init_params(int(seed) % 1000003)).to(DEV)
    ws = torch.empty(int(L.lib().sd_mlp_train_workspace_bytes(case["rows"])), dtype=torch.uint8, device=DEV)
    z = lambda k: torch.zeros(k, device=DEV)  # noqa: E731
    return {"kind": "train", "rows": case["rows"], "x": x, "t": t, "p0": p0, "p": p0.clone(), "m": z(N_PARAMS),
            "v": z(N_PARAMS), "g": z(N_PARAMS), "sse": z(BATCHES), "ws": ws}


def _run_train(st):
    lib, rows = L.lib(), st["rows"]
    p, m, v, g, ws = st["p"], st["m"], st["v"], st["g"], st["ws"]
    p.copy_(st["p0"])
    m.zero_()
    v.zero_()
    for b in range(BATCHES):
        xb, tb = st["x"][b * rows:(b + 1) * rows], st["t"][b * rows:(b + 1) * rows]
        L.check(lib.sd_mlp_loss_grad(p.data_ptr(), xb.data_ptr(), tb.data_ptr(), rows, g.data_ptr(),
                                     st["sse"][b:].data_ptr(), ws.data_ptr(), ws.numel(), None), "sd_mlp_loss_grad")
        L.check(lib.sd_mlp_adam(p.data_ptr(), m.data_ptr(), v.data_ptr(), g.data_ptr(), b + 1, ctypes.c_float(2e-3),
                                ctypes.c_float(0.9), ctypes.c_float(0.999), ctypes.c_float(1e-8), None), "sd_mlp_adam")
    return {"grad": g, "params": p, "m": m, "v": v, "sse": st["sse"]}


def _read_by_id(st, base=None):
    """The particles by their numbers: the order a program that follows particles wants."""
    pos, vel = st["slots"]
    ids = vel[:, 3].to(torch.int64)
    if base is not None:
        ids += base
    st["by_id"][0].index_copy_(0, ids, pos)
    st["by_id"][1].index_copy_(0, ids, vel)
    return {"pos": st["by_id"][0], "vel": st["by_id"][1][:, :3]}


def _by_slot(pos, vel):
    return {"pos": pos, "vel": vel[:, :3], "id": vel[:, 3]}


def run(st):
    kind = st["kind"]
    if kind == "train":
        return _run_train(st)
    if kind == "accel":
        return st["field"].accel()
    if kind == "ensemble":
        st["ens"].steps(st["case"]["dt"], st["case"]["steps"])
        for view, p, v in st["views"]:
            view.get_particles_into(p, v)
        st["ens"].synchronize()
        return _read_by_id(st, st["base"])
    case, sim = st["case"], st["sim"]
    if kind == "offload":
        for out in st["out"]:
            sim.step_host_async(st["pos"], st["vel"], case["dt"], out)
        sim.step_host_wait()
        return [_by_slot(*out) for out in st["out"]]
    here = torch.cuda.current_stream()
    st["stream"].wait_stream(here)
    with torch.cuda.stream(st["stream"]):
        sim.set_particles(st["pos"], st["vel"])
        if kind == "step":
            sim.step(case["dt"])
        elif kind == "auto":
            for _ in range(case["steps"]):
                sim.step()
        else:
            sim.steps(case["dt"], case["steps"])
            if case["integrator"] == "kdk":
                sim.synchronize()
        sim.get_particles_into(*st["slots"])
        out = _by_slot(*st["slots"]) if kind == "step" else _read_by_id(st)
    here.wait_stream(st["stream"])
    return out


# ---- what a pass cannot do without -----------------------------------------------------


def _step_work(n, grid, box, learned=False):
    """A step reads and writes every particle once and makes the density and the potential
    once; deposit, kick and interpolation are about 250 operations a particle, the two
    transforms 2.5 M log2 M each, the correction 13,000 operations a particle."""
    m = float(box) ** 3
    return 64.0 * n + 8.0 * float(grid) ** 3, 250.0 * n + 5.0 * m * math.log2(m) + (13000.0 * n if learned else 0.0)


def work(case):
    kind = case["kind"]
    if kind == "train":
        r = case["rows"] * BATCHES
        return {"bytes": r * (64.0 + 12.0) + BATCHES * 20.0 * N_PARAMS, "flops": 6.0 * r * 6656}
    if kind == "ensemble":
        w = [_step_work(n, g, g) for _, n, g in _members(case)]
        return {"bytes": case["steps"] * sum(b for b, _ in w), "flops": case["steps"] * sum(f for _, f in w)}
    n, g = case["n"], case["grid"]
    b, f = _step_work(n, g, 2 * g if case.get("boundary") == "isolated" else g, case.get("learned", False))
    if kind == "accel":
        return {"bytes": 32.0 * n + 8.0 * g ** 3, "flops": f}
    k = {"step": 1, "auto": case.get("steps"), "offload": case.get("calls")}.get(kind, case.get("steps"))
    return {"bytes": k * b, "flops": k * f}


# ---- 64-bit restatement ----------------------------------------------------------------


def _corners(x, G, periodic):
    g = x * G - 0.5
    i = g.floor()
    f = g - i
    i = i.to(torch.int64)
    for c in range(8):
        o = [c & 1, (c >> 1) & 1, c >> 2]
        w = 1.0
        j = []
        for d in range(3):
            w = w * (f[:, d] if o[d] else 1.0 - f[:, d])
            q = i[:, d] + o[d]
            j.append(q & (G - 1) if periodic else q.clamp(0, G - 1))
        yield w, (j[2] * G + j[1]) * G + j[0]


CHUNK = 1 << 21


def _deposit(x, G, periodic):
    rho = torch.zeros(G ** 3, dtype=torch.float64, device=DEV)
    for a in range(0, len(x), CHUNK):
        for w, c in _corners(x[a:a + CHUNK], G, periodic):
            rho.index_add_(0, c, w)
    return rho


def _sample(field, x, G, periodic):
    out = torch.zeros(len(x), field.shape[1], dtype=torch.float64, device=DEV)
    for a in range(0, len(x), CHUNK):
        for w, c in _corners(x[a:a + CHUNK], G, periodic):
            out[a:a + CHUNK] += w[:, None] * field[c]
    return out


def _shift(a, dim, s, periodic):
    """a at the neighbour s (+1 or -1) cells on; past the edge of an isolated grid its own value."""
    if periodic:
        return a.roll(-s, dim)
    n = a.shape[dim]
    if s > 0:
        return torch.cat([a.narrow(dim, 1, n - 1), a.narrow(dim, n - 1, 1)], dim)
    return torch.cat([a.narrow(dim, 0, 1), a.narrow(dim, 0, n - 1)], dim)


def _potential(rho, G, soft, periodic):
    if periodic:
        k = torch.fft.fftfreq(G, 1.0 / G, device=DEV, dtype=torch.float64)
        kr = torch.arange(G // 2 + 1, device=DEV, dtype=torch.float64)
        k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + kr[None, None, :] ** 2
        k2[0, 0, 0] = 1.0
        s = 2.0 * math.pi * soft / G
        green = -torch.exp(-0.5 * s * s * k2) / (4.0 * math.pi ** 2 * k2)
        green[0, 0, 0] = 0.0
        return torch.fft.irfftn(torch.fft.rfftn(rho.view(G, G, G)) * green, s=(G, G, G))
    S = 2 * G
    i = torch.arange(S, device=DEV, dtype=torch.float64)
    d2 = torch.minimum(i, S - i) ** 2
    r = torch.sqrt(d2[:, None, None] + d2[None, :, None] + d2[None, None, :])
    spec = torch.fft.rfftn(-1.0 / (r + max(soft, 0.5)))
    del r
    spec *= torch.fft.rfftn(rho.view(G, G, G), s=(S, S, S))
    return torch.fft.irfftn(spec, s=(S, S, S))[:G, :G, :G]


def _gradient_force(phi, G, scale, periodic):
    h = 0.5 * G * scale
    return torch.stack([-(_shift(phi, d, 1, periodic) - _shift(phi, d, -1, periodic)) * h for d in (2, 1, 0)],
                       -1).reshape(-1, 3)


def _cell(x, G):
    return (x * G).to(torch.int64).clamp(0, G - 1)


def _mlp_force(x, rho, G, corr):
    """The correction's network on the density stencil and the sub-cell offset, its weights the
    16-bit ones it is defined with, everything else in 64 bits."""
    W = {}
    for k, (o, sh) in LAYOUT.items():
        t = torch.from_numpy(np.ascontiguousarray(corr.params[o:o + int(np.prod(sh))])).to(DEV).reshape(sh)
        W[k] = (t.bfloat16() if k[0] == "W" else t).double()
    feat = torch.log1p(rho * (float(G) ** 3 / len(x))) - math.log(2.0)
    out = torch.empty(len(x), 3, dtype=torch.float64, device=DEV)
    for a in range(0, len(x), CHUNK // 4):
        p = x[a:a + CHUNK // 4]
        c = _cell(p, G)
        f = torch.zeros(len(p), 32, dtype=torch.float64, device=DEV)
        for j in range(27):
            d = [j % 3 - 1, j // 3 % 3 - 1, j // 9 - 1]
            q = [(c[:, e] + d[e]) & (G - 1) for e in range(3)]
            f[:, j] = feat[(q[2] * G + q[1]) * G + q[0]]
        f[:, 27:30] = p * G - c - 0.5
        h = torch.nn.functional.silu(f @ W["W1"] + W["b1"])
        h = torch.nn.functional.silu(h @ W["W2"] + W["b2"])
        out[a:a + CHUNK // 4] = (h @ W["W3"] + W["b3"])[:, :3]
    return out * corr.out_scale


class _Exact:
    """The step in 64 bits: deposit, potential, central differences, kick, drift, and the
    removal of the mean velocity."""

    def __init__(self, pos, vel, G, soft=1.0, units="newton", periodic=True, corr=None, hydro=False):
        self.x, self.v = pos[:, :3].double(), vel[:, :3].double()
        self.G, self.soft, self.periodic, self.corr, self.hydro = G, soft, periodic, corr, hydro
        n = len(pos)
        f = {True: 4.0 * math.pi * float(G) ** 3, False: float(G)}[periodic] if units == "newton" else 1.0
        self.scale = f / n
        self.disp = torch.zeros(G ** 3, 3, dtype=torch.float64, device=DEV) if hydro else None
        self.dcnt = torch.zeros(G ** 3, dtype=torch.float64, device=DEV) if hydro else None
        self.count = 0

    def accel(self):
        rho = _deposit(self.x, self.G, self.periodic)
        phi = _potential(rho, self.G, self.soft, self.periodic)
        a = _sample(_gradient_force(phi, self.G, self.scale, self.periodic), self.x, self.G, self.periodic)
        if self.corr is not None:
            a += _mlp_force(self.x, rho, self.G, self.corr)
        return a

    def _pressure(self):
        G = self.G
        h = 0.5 * G * 0.45 / self.dcnt.clamp_min(1.0)
        f = []
        for e, d in enumerate((2, 1, 0)):
            q = self.disp[:, e].view(G, G, G)
            df = (_shift(q, d, 1, self.periodic) - _shift(q, d, -1, self.periodic)).reshape(-1)
            f.append((-df * h).clamp(-5.0, 5.0) * (self.dcnt > 0))
        return _sample(torch.stack(f, 1), self.x, G, self.periodic)

    def _cool(self, dt):
        c = _cell(self.x, self.G)
        c = (c[:, 2] * self.G + c[:, 1]) * self.G + c[:, 0]
        cnt = torch.zeros_like(self.dcnt).index_add_(0, c, torch.ones_like(self.x[:, 0]))
        s = torch.zeros_like(self.disp).index_add_(0, c, self.v)
        many = cnt[c] >= 2
        dv = (s[c] / cnt[c][:, None] - self.v) * many[:, None]
        self.disp = torch.zeros_like(self.disp).index_add_(0, c, dv * dv)
        self.dcnt = torch.zeros_like(self.dcnt).index_add_(0, c, many.double())
        self.v = self.v + min(0.08 * dt * 60.0, 0.5) * dv

    def step(self, kick, drift=None):
        drift = kick if drift is None else drift
        a = self.accel()
        if self.hydro:
            a += self._pressure()
            if self.count % 2 == 0:
                self._cool(2 * drift)
        self.v = self.v + a * kick
        self.x = self.x + self.v * drift
        if self.periodic:
            self.x = self.x - self.x.floor()
        else:
            lo, hi = self.x < 0.002, self.x > 0.998
            self.v = torch.where(lo, 0.25 * self.v.abs(), torch.where(hi, -0.25 * self.v.abs(), self.v))
            self.x = self.x.clamp(0.002, 0.998)
        self.v = self.v - self.v.mean(0)
        self.count += 1

    def out(self, pos, vel, perm=None):
        r = {"pos": torch.cat([self.x, pos[:, 3:].double()], 1), "vel": self.v}
        return r if perm is None else dict({k: t[perm] for k, t in r.items()}, id=vel[perm, 3].double())


def _f32(v):
    return float(np.float32(v))


def _sorted_by(pos, G, order):
    """The stable sort's permutation of the particles in the given order."""
    p = pos[:, :3]
    if order == "tiled":
        i = (p * G - 0.5).floor().to(torch.int64) & (G - 1)
        key = (((i[:, 2] >> 2) * (G // 4) + (i[:, 1] >> 2)) * 16) + (i[:, 2] & 3) * 4 + (i[:, 1] & 3)
    else:
        i = (p * G).to(torch.int64).clamp(0, G - 1)
        key = (i[:, 2] * G + i[:, 1]) * G + i[:, 0]
    return torch.sort(key, stable=True)[1]


def _exact_train(case, seed):
    st = _prepare_train(case, seed)
    rows = case["rows"]
    p, m, v = st["p0"].double(), st["m"].double(), st["v"].double()
    sse = []
    for b in range(BATCHES):
        x, t = st["x"][b * rows:(b + 1) * rows].double(), st["t"][b * rows:(b + 1) * rows].double()
        q = p.clone().requires_grad_(True)
        W = {}
        for k, (o, sh) in LAYOUT.items():
            w = q[o:o + int(np.prod(sh))].reshape(sh)
            # the weights enter rounded to 16 bits; the gradient is the rounded weights' one
            W[k] = w + (w.detach().float().bfloat16().double() - w.detach()) if k[0] == "W" else w
        h = torch.nn.functional.silu(x @ W["W1"] + W["b1"])
        h = torch.nn.functional.silu(h @ W["W2"] + W["b2"])
        e = ((h @ W["W3"] + W["b3"])[:, :3] - t).square().sum()
        sse.append(float(e))
        (g,) = torch.autograd.grad(e / (3.0 * rows), q)
        m = 0.9 * m + 0.1 * g
        v = 0.999 * v + 0.001 * g * g
        s = b + 1
        p = p - 2e-3 * (m / (1 - 0.9 ** s)) / ((v / (1 - 0.999 ** s)).sqrt() + 1e-8)
    return {"grad": g, "params": p, "m": m, "v": v, "sse": torch.tensor(sse, dtype=torch.float64)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "ensemble":
        pos, vel = [], []
        for i, (scene, n, grid) in enumerate(_members(case)):
            p, v = _scene(scene, n, int(seed) * 101 + i)
            e = _Exact(p, v, grid)
            for _ in range(case["steps"]):
                e.step(_f32(case["dt"]))
            r = e.out(p, v)
            pos.append(r["pos"])
            vel.append(r["vel"])
        return {"pos": torch.cat(pos), "vel": torch.cat(vel)}
    pos, vel = _scene(case["scene"], case["n"], seed)
    corr = _correction(case, seed) if case.get("learned") else None
    e = _Exact(pos, vel, case["grid"], case.get("soft", 1.0), case.get("units", "reference" if kind == "auto" else "newton"),
               case.get("boundary") != "isolated", corr, case.get("hydro", False))
    if kind == "accel":
        a = e.accel()
        return torch.cat([a, torch.zeros_like(a[:, :1])], 1)
    dt = _f32(case.get("dt", 0.0016))
    if kind in ("step", "offload"):
        e.step(dt)
        r = e.out(pos, vel, _sorted_by(pos, case["grid"], case.get("order", "tiled")))
        if kind == "step":
            return r
        return [{k: t.cpu() for k, t in r.items()}] * case["calls"]
    if kind == "auto":
        for _ in range(case["steps"]):
            vmax = float(e.v.norm(dim=1).max())
            e.step(min(_f32(0.0016), 0.8 / (case["grid"] * vmax)) if vmax > 1e-6 else _f32(0.0016))
        return e.out(pos, vel)
    kdk = case["integrator"] == "kdk"
    for k in range(case["steps"]):
        e.step(0.5 * dt if kdk and k == 0 else dt, dt)
    if kdk:
        e.step(0.5 * dt, 0.0)
    return e.out(pos, vel)
