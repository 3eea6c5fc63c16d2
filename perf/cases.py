"""The workloads whose time is measured: seeded inputs, one pass through the public API, the work a pass cannot do
without, and what it returns in 64-bit arithmetic.

A scene pass is one simulation job: the particle state in, a number of substeps, the particle state out (x, v, C, F and
damage, in pinned host buffers a program keeps). A batch pass advances resident scenes together and reads their state; a
serving pass submits requests of uneven length and ticks until the last one has finished; a stream pass runs a list of
independent one-substep jobs. Sizes are those of the repository's own configurations: the 32,768-particle elastic cube,
the 0.5 x 0.1 x 0.5 m AnisoMPM slab at dx = 1/128 (425,984 particles) and 1/256 (3,407,872), boxes of 5k-400k particles
in a batch and serving requests from 10k particles on.

Slabs start in the middle of a tear: stretched along the fibres, with a damaged band across the middle and their ends held
by sticky grips that shear them apart (the grips move along their own planes, so a repeated job meets the same ones).
Boxes start slightly deformed on the sticky ground.
"""
import math

import numpy as np
import torch

import ziran2020_gb300 as zr

DT = {"box": 1e-4, "slab": 5e-5, "cloud": 5e-5}
MODEL = {"corotated": zr.COROTATED, "borden": zr.NEOHOOKEAN_BORDEN, "qr": zr.QR_STABLE_NEOHOOKEAN}
DAMAGE = dict(alpha=-1.0, eta=0.1, zeta=1.0, residual=0.01)
GRIP_CELLS, GRIP_SPEED, GROUND = 2, 0.5, 0.05


# --------------------------------------------------------------------------------------------------------- the cases
def _scene(name, shape, material, damage, bits, cells, nx, ny, nz, ppc, substeps):
    return {"name": name, "kind": "scene", "shape": shape, "material": material, "damage": damage, "bits": bits, "cells": cells,
            "nx": nx, "ny": ny, "nz": nz, "ppc": ppc, "substeps": substeps}


def listed():
    return [
        # the smallest call: a preview box advanced by a few substeps between two looks at it
        _scene("preview box f32", "box", "corotated", "none", 32, 64, 8, 8, 8, 2, 4),
        # the elastic cube of side 0.25 at dx = 1/64, in both precisions
        _scene("elastic cube f32", "box", "corotated", "none", 32, 64, 16, 16, 16, 2, 50),
        _scene("elastic cube f64", "box", "corotated", "none", 64, 64, 16, 16, 16, 2, 20),
        # the AnisoMPM slab at dx = 1/128, in both precisions
        _scene("slab f32", "slab", "borden", "explicit", 32, 128, 64, 13, 64, 2, 20),
        _scene("slab f64", "slab", "borden", "explicit", 64, 128, 64, 13, 64, 2, 6),
        # the slab at dx = 1/256, the size the throughput metric is quoted on
        _scene("large slab f32", "slab", "borden", "explicit", 32, 256, 128, 26, 128, 2, 20),
        # the implicit damage solve
        _scene("implicit slab f32", "slab", "borden", "implicit", 32, 128, 64, 13, 64, 2, 10),
        # the fibre-reinforced QR-stable model of the AnisoMPM demos, odd sizes, 27 particles per cell
        _scene("fibre slab f32", "slab", "qr", "explicit", 32, 160, 61, 11, 59, 3, 12),
        # a splash of uneven blobs: three models in one scene, 1 to ~100 particles per cell, slip and separating walls
        {"name": "blobs f32", "kind": "cloud", "particles": 100003, "blobs": 37, "bits": 32, "cells": 64, "substeps": 20},
        # boxes of uneven sizes advanced together
        {"name": "batch f32", "kind": "batch", "scenes": 12, "least": 5000, "most": 200000, "bits": 32, "substeps": 40},
        # served requests of uneven sizes and lengths
        {"name": "serve f32", "kind": "serve", "scenes": 6, "least": 10000, "most": 60000, "bits": 32, "substeps": 60},
        # independent one-substep jobs on full states, pipelined
        {"name": "stream f32", "kind": "stream", "jobs": 8, "bits": 32, "cells": 128, "nx": 64, "ny": 13, "nz": 64},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["scene"] * 8 + ["cloud", "batch", "serve", "stream"])
    if kind == "cloud":
        return {"kind": kind, "particles": int(_log_uniform(rng, 3000, 400000)), "blobs": rng.randint(5, 60), "bits": 32,
                "cells": rng.choice([48, 64, 96]), "substeps": rng.randint(5, 25)}
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(3, 12), "least": 5000, "most": int(_log_uniform(rng, 20000, 200000)), "bits": 32,
                "substeps": rng.randint(20, 40)}
    if kind == "serve":
        return {"kind": kind, "scenes": rng.randint(2, 6), "least": 10000, "most": int(_log_uniform(rng, 15000, 60000)), "bits": 32,
                "substeps": rng.randint(20, 60)}
    if kind == "stream":
        return {"kind": kind, "jobs": rng.randint(3, 8), "bits": 32, "cells": 128, "nx": rng.randint(20, 64), "ny": rng.randint(5, 13),
                "nz": rng.randint(20, 64)}
    bits = rng.choice([32, 32, 64])
    shape = rng.choice(["box", "slab", "slab"])
    ppc = rng.choice([1, 2, 2, 2, 3])
    cells = rng.choice([64, 96, 128, 160, 256]) if shape == "slab" else rng.choice([64, 64, 96])
    n = _log_uniform(rng, 4000, 2.0e6 if bits == 32 else 4.0e5)
    filled = n / ppc**3
    if shape == "box":
        side = max(4, min(int(0.5 * cells), round(filled ** (1 / 3))))
        nx, ny, nz = (max(4, min(int(0.6 * cells), side + rng.randint(-2, 2))) for _ in range(3))
        material, damage = "corotated", "none"
    else:
        side = max(4, min(int(0.55 * cells), round((5 * filled) ** (1 / 3))))
        nx, nz = (max(4, min(int(0.6 * cells), side + rng.randint(-3, 3))) for _ in range(2))
        ny = max(3, side // 5 + rng.randint(-1, 1))
        material = rng.choice(["borden", "borden", "qr"])
        damage = rng.choice(["explicit", "explicit", "implicit"])
    n = nx * ny * nz * ppc**3
    substeps = max(2, min(rng.randint(4, 40), int((4.0e7 if bits == 32 else 2.0e6) / n)))
    case = _scene("", shape, material, damage, bits, cells, nx, ny, nz, ppc, substeps)
    del case["name"]
    return case


def work(case):
    """Bytes and floating-point operations of one pass: every substep reads each particle's state (x, v, C, F, mass, volume;
    damage and critical stress where there is damage) and writes what it changes; a job's state also crosses the host link."""
    s = case["bits"] // 8
    bytes_, flops = 0.0, 0.0
    for n, substeps, damaged, in_out in _parts(case):
        bytes_ += n * substeps * s * (26 + 24 + (3 if damaged else 0)) + n * s * 25 * in_out
        # per particle and substep: 27 nodes of scatter and of gather (weights, affine momentum and force; v, C, grad v),
        # stress and, where there is damage, the phase field on both sides
        flops += n * substeps * (27 * (2 * 16 + (8 if damaged else 0)) + 350)
    return {"bytes": float(bytes_), "flops": float(flops)}


def _parts(case):
    """(particles, substeps, has damage, state transfers) of the scenes of a pass"""
    if case["kind"] == "scene":
        return [(case["nx"] * case["ny"] * case["nz"] * case["ppc"] ** 3, case["substeps"], case["damage"] != "none", 2)]
    if case["kind"] == "cloud":
        return [(case["particles"], case["substeps"], True, 2)]
    if case["kind"] == "stream":
        return [(case["jobs"] * case["nx"] * case["ny"] * case["nz"] * 8, 1, True, 2)]
    if case["kind"] == "batch":
        return [(_box_cells(n) ** 3 * 8, case["substeps"], False, 1) for n in _sizes(case)]
    return [(_box_cells(n) ** 3 * 8, k, False, 2) for n, k in zip(_sizes(case), _lengths(case))]


def _sizes(case):
    """particle counts of a batch's or a server's scenes, spread over the logarithm of their range"""
    k = case["scenes"]
    return [case["least"] * (case["most"] / case["least"]) ** (i / max(1, k - 1)) for i in range(k)]


def _lengths(case):
    return [max(4, case["substeps"] - 7 * i) for i in range(case["scenes"])]


def _box_cells(n):
    return max(2, round((n / 8) ** (1 / 3)))


# ------------------------------------------------------------------------------------------------------------ inputs
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Draws:
    """seeded uniforms and normals on the device"""

    def __init__(self, seed):
        self.dev = _device()
        self.g = torch.Generator(device=self.dev)
        self.g.manual_seed(seed)

    def uniform(self, *shape):
        return torch.rand(*shape, generator=self.g, device=self.dev, dtype=torch.float64)

    def normal(self, *shape):
        return torch.randn(*shape, generator=self.g, device=self.dev, dtype=torch.float64)


def _lattice(r, nx, ny, nz, ppc, dx, lo):
    """jittered positions, ppc^3 per cell, in cell order"""
    ax = [torch.arange(k * ppc, device=r.dev, dtype=torch.float64) for k in (nx, ny, nz)]
    grid = torch.stack(torch.meshgrid(*ax, indexing="ij"), dim=-1)
    grid = grid.reshape(nx, ppc, ny, ppc, nz, ppc, 3).permute(0, 2, 4, 1, 3, 5, 6).reshape(-1, 3)
    return (grid + r.uniform(*grid.shape)) * (dx / ppc) + torch.tensor(lo, device=r.dev, dtype=torch.float64)


def _fibre_frames(r, n, kappa=20.0):
    """F0 = (a, a_perp, a x a_perp) with the fibre a from a von Mises-Fisher law about +x"""
    u, ph = r.uniform(n), 2 * math.pi * r.uniform(n)
    w = (1 + torch.log(u + (1 - u) * math.exp(-2 * kappa)) / kappa).clamp(-1, 1)
    s = (1 - w * w).clamp_min(0).sqrt()
    a = torch.stack([w, s * ph.cos(), s * ph.sin()], dim=1)
    b = torch.stack([-a[:, 1], a[:, 0], torch.zeros_like(w)], dim=1)
    b = b / b.norm(dim=1, keepdim=True).clamp_min(1e-12)
    return torch.stack([a, b, torch.linalg.cross(a, b)], dim=2)


def _box_inputs(r, cells, nx, ny, nz, ppc, centre=None, v0=(0.0, -1.0, 0.0), E=1e4):
    dx = 1.0 / cells
    lo = [0.5 - 0.5 * nx * dx, GROUND + 0.5 * dx, 0.5 - 0.5 * nz * dx]
    if centre is not None:
        lo = [c - 0.5 * k * dx for c, k in zip(centre, (nx, ny, nz))]
    x = _lattice(r, nx, ny, nz, ppc, dx, lo)
    n = x.shape[0]
    V0 = torch.full((n,), dx**3 / ppc**3, device=r.dev, dtype=torch.float64)
    F = torch.eye(3, device=r.dev, dtype=torch.float64) + 0.02 * r.normal(n, 3, 3).clamp(-3, 3)
    v = torch.tensor(v0, device=r.dev, dtype=torch.float64) + 0.05 * r.normal(n, 3)
    return dict(x=x, v=v, C=r.normal(n, 3, 3), F=F, d=torch.zeros(n, device=r.dev, dtype=torch.float64), m=1000.0 * V0, V0=V0,
                sigma_c=torch.ones_like(V0), dx=dx, dt=DT["box"], gravity=(0.0, -9.8, 0.0), apic=1.0, domain=cells + 4, implicit=False,
                ranges=[(0, n, "corotated", E, 0.3, 0.0, False)],
                objects=[((0, GROUND, 0), (0, 1, 0), zr.STICKY, 0.0, (0, 0, 0))])


def _slab_inputs(r, cells, nx, ny, nz, ppc, material, damage):
    dx = 1.0 / cells
    lo = [0.5 - 0.5 * k * dx for k in (nx, ny, nz)]
    x = _lattice(r, nx, ny, nz, ppc, dx, lo) - 0.5
    n = x.shape[0]
    V0 = torch.full((n,), dx**3 / ppc**3, device=r.dev, dtype=torch.float64)
    stretch = torch.tensor([1.03, 0.995, 0.995], device=r.dev, dtype=torch.float64)
    x = x * stretch
    F = torch.diag(stretch) @ _fibre_frames(r, n) @ (torch.eye(3, device=r.dev, dtype=torch.float64) + 0.004 * r.normal(n, 3, 3).clamp(-3, 3))
    half = 0.5 * nx * dx * float(stretch[0])
    v = torch.stack([0.3 * x[:, 0] / half, torch.zeros(n, device=r.dev, dtype=torch.float64), GRIP_SPEED * x[:, 0] / half], dim=1) + 0.02 * r.normal(n, 3)
    W = 2.0 * r.normal(n, 3, 3)
    band = 0.9 * torch.exp(-((x[:, 0] / (4 * dx)) ** 2))
    d = (band * r.uniform(n) + 0.02 * r.uniform(n)).clamp(0, 0.95)
    grip = half - GRIP_CELLS * dx
    return dict(x=x + 0.5, v=v, C=W - W.transpose(1, 2), F=F, d=d, m=800.0 * V0, V0=V0, sigma_c=(400.0 + 40.0 * r.normal(n)).clamp_min(100.0),
                dx=dx, dt=DT["slab"], gravity=(0.0, 0.0, 0.0), apic=0.0, domain=cells + 4, implicit=damage == "implicit",
                ranges=[(0, n, material, 5e4, 0.25, 10.0 if material == "qr" else 0.0, True)],
                objects=[((0.5 - grip, 0, 0), (1, 0, 0), zr.STICKY, 0.0, (0, 0, -GRIP_SPEED)),
                         ((0.5 + grip, 0, 0), (-1, 0, 0), zr.STICKY, 0.0, (0, 0, GRIP_SPEED))])


def _cloud_inputs(r, case):
    dx, n, k = 1.0 / case["cells"], case["particles"], case["blobs"]
    centre = 0.25 + 0.5 * r.uniform(k, 3)
    centre[:, 1] = centre[:, 1].clamp_min(0.3)
    radius = dx * torch.exp(math.log(1.0) + r.uniform(k) * math.log(6.0))
    owner = torch.sort((r.uniform(n) * k).long()).values
    x = (centre[owner] + radius[owner, None] * r.normal(n, 3).clamp(-2.5, 2.5)).clamp(0.1, 0.9)
    V0 = torch.full((n,), dx**3 / 8, device=r.dev, dtype=torch.float64)
    F = torch.eye(3, device=r.dev, dtype=torch.float64) + 0.01 * r.normal(n, 3, 3).clamp(-3, 3)
    speed = 0.6 * r.normal(k, 3).clamp(-1.5, 1.5)
    v = speed[owner] + 0.02 * r.normal(n, 3)
    a, b = n // 3, 2 * n // 3
    d = torch.zeros(n, device=r.dev, dtype=torch.float64)
    d[a:b] = 0.3 * r.uniform(b - a)
    d[b:] = 0.1 * r.uniform(n - b)
    tilt = 1 / math.sqrt(2.0)
    return dict(x=x, v=v, C=r.normal(n, 3, 3), F=F, d=d, m=1000.0 * V0, V0=V0, sigma_c=(200.0 + 20.0 * r.normal(n)).clamp_min(50.0), dx=dx,
                dt=DT["cloud"], gravity=(0.0, -9.8, 0.0), apic=1.0, domain=case["cells"] + 4, implicit=False,
                ranges=[(0, a, "corotated", 1e4, 0.3, 0.0, False), (a, b - a, "borden", 2e4, 0.25, 0.0, True), (b, n - b, "qr", 2e4, 0.25, 5.0, True)],
                objects=[((0.3, 0.3, 0.5), (tilt, tilt, 0), zr.SLIP, 0.3, (0, 0, 0.25)), ((0, 0.28, 0), (0, 1, 0), zr.SEPARATE, 0.4, (0, 0, 0)),
                         ((0.8, 0, 0), (-1, 0, 0), zr.SEPARATE, 0.0, (0, 0, 0))])


def _rounded(sc, bits):
    """the inputs as the engine's precision holds them"""
    if bits == 32:
        for k in ("x", "v", "C", "F", "d", "m", "V0", "sigma_c"):
            sc[k] = sc[k].float().double()
    return sc


def _scenes(case, seed):
    """the scenes of a case's pass, as tensors on the device"""
    r = _Draws(seed)
    kind, bits = case["kind"], case["bits"]
    if kind == "scene":
        args = (r, case["cells"], case["nx"], case["ny"], case["nz"], case["ppc"])
        sc = [_box_inputs(*args) if case["shape"] == "box" else _slab_inputs(*args, case["material"], case["damage"])]
    elif kind == "cloud":
        sc = [_cloud_inputs(r, case)]
    elif kind == "stream":
        sc = [_slab_inputs(r, case["cells"], case["nx"], case["ny"], case["nz"], 2, "borden", "explicit")]
    else:
        sc = []
        for n in _sizes(case):
            side = _box_cells(n)
            cells = max(64, 2 * side)
            u = r.uniform(7).tolist()
            centre = [0.35 + 0.3 * t for t in u[:3]]
            sc.append(_box_inputs(r, cells, side, side, side, 2, centre, [0.2 * (2 * u[3] - 1), 2 * u[4] - 1, 0.2 * (2 * u[5] - 1)], 5e3 + 4.5e4 * u[6]))
    return [_rounded(s, bits) for s in sc]


def _rows(sc, bits):
    """state rows (x, v, C, F, d) in pinned host memory"""
    n = sc["x"].shape[0]
    t = torch.cat([sc["x"], sc["v"], sc["C"].reshape(n, 9), sc["F"].reshape(n, 9), sc["d"][:, None]], dim=1)
    return _pinned(t.to(torch.float32 if bits == 32 else torch.float64))


def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=torch.cuda.is_available())
    h.copy_(t)
    return h


def _host(t):
    return np.ascontiguousarray(t.cpu().numpy())


def _build(sc, bits):
    s = zr.Scene(zr.F32 if bits == 32 else zr.F64)
    _fill(s, _host_arrays(sc), sc)
    return s


def _host_arrays(sc):
    return {k: _host(sc[k]) for k in ("x", "v", "F", "m", "V0", "sigma_c")}


def _fill(s, a, sc):
    s.set_params(sc["dx"], sc["dt"], sc["gravity"], sc["apic"], 0.6, sc["domain"])
    s.add_particles(a["x"], a["m"], a["V0"], v=a["v"], F=a["F"])
    for first, count, material, E, nu, fibre, damaged in sc["ranges"]:
        if material == "corotated":
            s.add_corotated(first, count, E, nu)
        elif material == "borden":
            s.add_neohookean_borden(first, count, E, nu)
        else:
            s.add_qr_stable_neohookean(first, count, E, nu, fibre)
        if damaged:
            s.add_aniso_damage(first, count, DAMAGE["alpha"], 0.5 * sc["dx"], DAMAGE["eta"], DAMAGE["zeta"], DAMAGE["residual"], a["sigma_c"][first:first + count])
    for origin, normal, kind, friction, velocity in sc["objects"]:
        s.add_halfspace(origin, normal, kind, friction, velocity)
    if sc["implicit"]:
        s.set_implicit_damage(True)


# ------------------------------------------------------------------------------------------------------------ passes
WARM = 2  # substeps a batch has run before its first pass (they choose its schedule)


def prepare(case, seed):
    kind, bits = case["kind"], case["bits"]
    scenes = _scenes(case, seed)
    state = {"case": case}
    if kind in ("scene", "cloud", "stream"):
        sc = scenes[0]
        state["scene"] = _build(sc, bits)
        rows = _rows(sc, bits)
        if kind == "stream":
            jobs = [rows] + [_pinned(_job_rows(rows, seed, j)) for j in range(1, case["jobs"])]
            state["keep"] = jobs, [torch.empty(rows.shape, dtype=rows.dtype, pin_memory=torch.cuda.is_available()) for _ in jobs]
            state["in"], state["out"] = [t.numpy() for t in state["keep"][0]], [t.numpy() for t in state["keep"][1]]
        else:
            out = torch.empty(rows.shape, dtype=rows.dtype, pin_memory=torch.cuda.is_available())
            history = _pinned(torch.zeros(rows.shape[0], dtype=rows.dtype)) if sc["implicit"] else None
            state["keep"] = rows, out, history
            state["in"], state["out"] = rows.numpy(), out.numpy()
            state["history"] = None if history is None else history.numpy()
        run(state)  # the program's warm-up: buffers, schedule, graphs
    elif kind == "batch":
        state["batch"] = zr.Batch(zr.F32)
        for sc in scenes:
            s = _build(sc, bits)
            state["batch"].add_scene(s)
            s.close()
        state["batch"].step(WARM)
    else:
        state["server"] = zr.Server(zr.F32, budget_bytes=60e9, tick_substeps=10, max_scenes=256)
        state["requests"] = [({**sc, "x": None}, _host_arrays(sc), k) for sc, k in zip(scenes, _lengths(case))]
        for sc, _, _ in state["requests"]:
            for k in ("v", "C", "F", "d", "m", "V0", "sigma_c"):
                sc[k] = None
    return state


def _job_rows(rows, seed, j):
    """a stream's later jobs: the same particles with other velocities"""
    r = _Draws(seed * 1000003 + j)
    t = rows.clone()
    t[:, 3:6] += (0.1 * r.normal(rows.shape[0], 3)).to(rows.dtype).cpu()
    return t


def _fields(rows):
    return {"x": rows[:, 0:3], "v": rows[:, 3:6], "C": rows[:, 6:15], "F": rows[:, 15:24], "d": rows[:, 24]}


def run(state):
    case = state["case"]
    if case["kind"] in ("scene", "cloud"):
        s = state["scene"]
        s.set_state(state["in"])
        if state["history"] is not None:
            s.set("dtilde_max", state["history"])
        s.step(case["substeps"])
        return _fields(s.get_state(state["out"]))
    if case["kind"] == "stream":
        return [_fields(o) for o in state["scene"].step_stream(state["in"], state["out"])]
    if case["kind"] == "batch":
        b = state["batch"]
        b.step(case["substeps"])
        return [{f: b.get(i, f, np.float32) for f in ("x", "v", "C", "F")} for i in range(case["scenes"])]
    sv = state["server"]
    ids = []
    for sc, arrays, substeps in state["requests"]:
        s = zr.Scene(zr.F32)
        _fill(s, arrays, sc)
        ids.append(sv.submit_scene(s, substeps))
        s.close()
    running, queued = 1, 1
    while running or queued:
        running, queued, _ = sv.tick()
    out = []
    for i in ids:
        out.append({f: sv.result(i, f, np.float32) for f in ("x", "v", "C", "F")})
        sv.release(i)
    return out


# ------------------------------------------------------------------------- the same passes in 64 bits, in plain torch
def exact(case, seed):
    kind = case["kind"]
    scenes = _scenes(case, seed)
    if kind in ("scene", "cloud"):
        return _rows_exact(_advance(scenes[0], case["substeps"]))
    if kind == "stream":
        sc = scenes[0]
        rows = _rows(sc, case["bits"])
        out = []
        for j in range(case["jobs"]):
            job = dict(sc)
            if j:
                job["v"] = _job_rows(rows, seed, j)[:, 3:6].to(sc["x"].device).double()
            out.append(_rows_exact(_advance(job, 1)))
        return out
    steps = [WARM + case["substeps"]] * len(scenes) if kind == "batch" else _lengths(case)
    got = []
    for sc, k in zip(scenes, steps):
        sc["C"] = torch.zeros_like(sc["C"])  # scenes built from particles start with C = 0
        f = _rows_exact(_advance(sc, k))
        got.append({q: f[q].reshape(-1, 3) if q in "xv" else f[q].reshape(-1, 9) for q in ("x", "v", "C", "F")})
    return got


def _rows_exact(sc):
    n = sc["x"].shape[0]
    return {"x": sc["x"].cpu().numpy(), "v": sc["v"].cpu().numpy(), "C": sc["C"].reshape(n, 9).cpu().numpy(), "F": sc["F"].reshape(n, 9).cpu().numpy(),
            "d": sc["d"].cpu().numpy()}


def _det(F):
    return (F[:, 0] * torch.linalg.cross(F[:, 1], F[:, 2])).sum(1)


def _polar(F):
    X = F
    for _ in range(9):
        cof = torch.stack([torch.linalg.cross(X[:, 1], X[:, 2]), torch.linalg.cross(X[:, 2], X[:, 0]), torch.linalg.cross(X[:, 0], X[:, 1])], dim=1)
        X = 0.5 * (X + cof / (X[:, 0] * cof[:, 0]).sum(1)[:, None, None])
    return X


def _eye(F):
    return torch.eye(3, device=F.device, dtype=F.dtype)


def _lame(E, nu):
    return E * nu / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))


def _tau_corotated(F, E, nu):
    lam, mu = _lame(E, nu)
    cof = torch.stack([torch.linalg.cross(F[:, 1], F[:, 2]), torch.linalg.cross(F[:, 2], F[:, 0]), torch.linalg.cross(F[:, 0], F[:, 1])], dim=1)
    P = 2 * mu * (F - _polar(F)) + (lam * (_det(F) - 1))[:, None, None] * cof
    return P @ F.transpose(1, 2)


def _tau_borden(F, E, nu, g):
    lam, mu = _lame(E, nu)
    kappa = 0.666666 * mu + lam
    B, J = F @ F.transpose(1, 2), _det(F)
    tr3 = B.diagonal(dim1=1, dim2=2).sum(1) / 3
    vol = J * kappa * 0.5 * (J - 1 / J)
    dev = (g * mu * J ** (-2.0 / 3))[:, None, None] * (B - tr3[:, None, None] * _eye(F))
    return dev + torch.where(J >= 1, g * vol, vol)[:, None, None] * _eye(F)


def _tau_qr(F, E, nu, fibre, g):
    """Kirchhoff stress Q A Q^T of the QR-stable Neo-Hookean energy, F = Q R with a positive diagonal"""
    lam, mu = _lame(E, nu)
    a, b, c = F[:, :, 0], F[:, :, 1], F[:, :, 2]
    dot = lambda p, q: (p * q).sum(1)  # noqa: E731
    r00 = dot(a, a).sqrt()
    q0 = a / r00[:, None]
    r01 = dot(q0, b)
    b = b - r01[:, None] * q0
    r11 = dot(b, b).sqrt()
    q1 = b / r11[:, None]
    q2 = torch.linalg.cross(q0, q1)
    r02, r12, r22 = dot(q0, c), dot(q1, c), dot(q2, c)
    z = torch.zeros_like(r00)
    R = torch.stack([r00, r01, r02, z, r11, r12, z, z, r22], dim=1).reshape(-1, 3, 3)
    J = r00 * r11 * r22
    vol = torch.where(J >= 1, g, torch.ones_like(g)) * lam * (J - 1) * J - g * mu * J
    D = (g * mu)[:, None, None] * R + torch.diag_embed(vol[:, None] / torch.stack([r00, r11, r22], dim=1))
    D[:, 0, 0] += fibre * mu * (r00 - 1)
    A = D @ R.transpose(1, 2)
    A = torch.triu(A) + torch.triu(A, 1).transpose(1, 2)
    Q = torch.stack([q0, q1, q2], dim=2)
    return Q @ A @ Q.transpose(1, 2), J


def _tension(S):
    """sum of the positive principal values times their projectors (cyclic Jacobi)"""
    A = {(i, j): S[:, i, j].clone() for i in range(3) for j in range(3)}
    V = {(i, j): torch.full_like(S[:, 0, 0], float(i == j)) for i in range(3) for j in range(3)}
    for _ in range(7):
        for p, q in ((0, 1), (0, 2), (1, 2)):
            apq = A[p, q]
            safe = torch.where(apq == 0, torch.ones_like(apq), apq)
            th = (A[q, q] - A[p, p]) / (2 * safe)
            t = torch.where(apq == 0, torch.zeros_like(th), torch.where(th >= 0, 1.0, -1.0) / (th.abs() + (th * th + 1).sqrt()))
            c = 1 / (t * t + 1).sqrt()
            s = t * c
            o = 3 - p - q
            A[p, p], A[q, q] = A[p, p] - t * apq, A[q, q] + t * apq
            A[p, o], A[q, o] = c * A[o, p] - s * A[o, q], s * A[o, p] + c * A[o, q]
            A[o, p], A[o, q] = A[p, o], A[q, o]
            A[p, q] = A[q, p] = torch.zeros_like(apq)
            for i in range(3):
                V[i, p], V[i, q] = c * V[i, p] - s * V[i, q], s * V[i, p] + c * V[i, q]
    out = torch.empty_like(S)
    for i in range(3):
        for j in range(3):
            out[:, i, j] = sum(A[k, k].clamp_min(0) * V[i, k] * V[j, k] for k in range(3))
    return out


def _drive(F, material, E, nu, sigma_c):
    """damage drive zeta <phi - 1> with phi from the tensile part of the undegraded Cauchy stress"""
    one = torch.ones_like(sigma_c)
    if material == "qr":
        tau, J = _tau_qr(F, E, nu, 0.0, one)
    else:
        tau, J = _tau_borden(F, E, nu, one), _det(F)
    sp = _tension(tau / J[:, None, None])
    a = _polar(F)[:, :, 0]
    M = sp + DAMAGE["alpha"] * a[:, :, None] * (a[:, None, :] @ sp)
    phi = (M * M.transpose(1, 2)).sum((1, 2)) / sigma_c**2
    return DAMAGE["zeta"] * (phi - 1).clamp_min(0)


def _collide(sc, xi, v):
    alive = torch.ones(xi.shape[0], dtype=torch.bool, device=xi.device)
    for origin, normal, kind, friction, velocity in sc["objects"]:
        o, nrm, vel = (torch.tensor(t, device=xi.device, dtype=torch.float64) for t in (origin, normal, velocity))
        hit = alive & (((xi - o) @ nrm) <= 0)
        if kind == zr.STICKY:
            v = torch.where(hit[:, None], vel, v)
            alive = alive & ~hit
            continue
        r = v - vel
        dot = r @ nrm
        act = hit if kind == zr.SLIP else hit & (dot < 0)
        rt = r - dot[:, None] * nrm
        if friction:
            vn = rt.norm(dim=1)
            keep = torch.where(-dot * friction < vn, 1 + dot * friction / vn.clamp_min(1e-300), torch.zeros_like(vn))
            rt = torch.where((dot < 0)[:, None], rt * keep[:, None], rt)
        v = torch.where(act[:, None], rt + vel, v)
    return v


def _advance(sc, substeps):
    sc = dict(sc)
    damaged_ranges = [q for q in sc["ranges"] if q[6]]
    history = torch.zeros_like(sc["d"])
    for _ in range(substeps):
        history = _substep(sc, damaged_ranges, history)
    return sc


def _substep(sc, damaged_ranges, history):
    x, v, C, F, d, m, V0, dx, dt = (sc[k] for k in ("x", "v", "C", "F", "d", "m", "V0", "dx", "dt"))
    n, dev = x.shape[0], x.device
    base = torch.floor(x / dx - 0.5)
    f = x / dx - base
    lo = base.min(0).values
    dims = [int(t) for t in (base.max(0).values - lo + 3).tolist()]
    b = (base - lo).long()
    first = (b[:, 0] * dims[1] + b[:, 1]) * dims[2] + b[:, 2]
    w = torch.stack([0.5 * (1.5 - f) ** 2, 0.75 - (f - 1) ** 2, 0.5 * (f - 0.5) ** 2], dim=0)
    dw = torch.stack([f - 1.5, 2 * (1 - f), f - 0.5], dim=0)
    offsets = [(i, j, k) for i in range(3) for j in range(3) for k in range(3)]

    def at(i, j, k):
        return first + (i * dims[1] + j) * dims[2] + k

    def weight(i, j, k):
        return w[i, :, 0] * w[j, :, 1] * w[k, :, 2]

    def gradient(i, j, k):
        return torch.stack([dw[i, :, 0] * w[j, :, 1] * w[k, :, 2], w[i, :, 0] * dw[j, :, 1] * w[k, :, 2], w[i, :, 0] * w[j, :, 1] * dw[k, :, 2]], dim=1)

    tau = torch.empty_like(F)
    for q0, cnt, material, E, nu, fibre, damaged in sc["ranges"]:
        r = slice(q0, q0 + cnt)
        g = (1 - d[r]) ** 2 * (1 - DAMAGE["residual"]) + DAMAGE["residual"] if damaged else torch.ones_like(d[r])
        if material == "corotated":
            tau[r] = _tau_corotated(F[r], E, nu)
        elif material == "borden":
            tau[r] = _tau_borden(F[r], E, nu, g)
        else:
            tau[r] = _tau_qr(F[r], E, nu, fibre, g)[0]
    K = (-dt / dx) * V0[:, None, None] * tau
    nodes = dims[0] * dims[1] * dims[2]
    G = torch.zeros(nodes, 6, device=dev, dtype=torch.float64)
    for i, j, k in offsets:
        wt = weight(i, j, k)
        rel = (torch.tensor([i, j, k], device=dev, dtype=torch.float64) - f) * dx
        mom = (wt * m)[:, None] * (v + (C @ rel[:, :, None])[:, :, 0]) + (K @ gradient(i, j, k)[:, :, None])[:, :, 0]
        G.index_add_(0, at(i, j, k), torch.cat([(wt * m)[:, None], mom, (wt * d)[:, None], wt[:, None]], dim=1))
    mass, wsum = G[:, 0], G[:, 5]
    full = mass != 0
    vi = torch.where(full[:, None], G[:, 1:4] / torch.where(full, mass, torch.ones_like(mass))[:, None], torch.zeros_like(G[:, 1:4]))
    vi = vi + dt * torch.tensor(sc["gravity"], device=dev, dtype=torch.float64)
    ids = torch.arange(nodes, device=dev)
    xi = (torch.stack([ids // (dims[1] * dims[2]), (ids // dims[2]) % dims[1], ids % dims[2]], dim=1) + lo) * dx
    vi = torch.where(full[:, None], _collide(sc, xi, vi), torch.zeros_like(vi))
    pf = torch.where(wsum != 0, G[:, 4] / torch.where(wsum != 0, wsum, torch.ones_like(wsum)), torch.zeros_like(wsum))
    if sc["implicit"]:
        history, pf = _solve_damage(sc, damaged_ranges, history, pf, offsets, at, weight, gradient)

    node = torch.cat([vi, pf[:, None]], dim=1)
    pv = torch.zeros_like(v)
    B, gv = torch.zeros_like(C), torch.zeros_like(C)
    lap, pw = torch.zeros_like(d), torch.zeros_like(d)
    second = (1.0, -2.0, 1.0)
    for i, j, k in offsets:
        wt = weight(i, j, k)
        u = node[at(i, j, k)]
        wv = wt[:, None] * u[:, :3]
        pv += wv
        rel = (torch.tensor([i, j, k], device=dev, dtype=torch.float64) - f) * dx
        B += wv[:, :, None] * rel[:, None, :]
        gv += u[:, :3, None] * gradient(i, j, k)[:, None, :]
        if damaged_ranges:
            lap += second[i] * u[:, 3] * (w[j, :, 1] * w[k, :, 2] + w[i, :, 0] * w[k, :, 2] + w[i, :, 0] * w[j, :, 1])
            pw += wt * u[:, 3]
    gv, lap = gv / dx, lap / dx**2
    ca, cb = (sc["apic"] + 1) / 2, (sc["apic"] - 1) / 2
    new_d = d.clone()
    for q0, cnt, material, E, nu, _, _ in damaged_ranges:
        r = slice(q0, q0 + cnt)
        if sc["implicit"]:
            new_d[r] = torch.maximum(d[r], d[r] + pw[r]).clamp_max(1)
        else:
            geo = d[r] - (0.5 * dx) ** 2 * lap[r]
            diff = (1 - d[r]) * _drive(F[r], material, E, nu, sc["sigma_c"][r]) - geo
            new_d[r] = (d[r] + dt / DAMAGE["eta"] * diff.clamp_min(0)).clamp_max(1)
    sc.update(x=x + dt * pv, v=pv, C=(ca * B + cb * B.transpose(1, 2)) * (4 / dx**2), F=F + dt * (gv @ F), d=new_d)
    return history


def _solve_damage(sc, damaged_ranges, history, pf, offsets, at, weight, gradient):
    """the nodal change of the phase field: Jacobi-preconditioned conjugate gradients from zero"""
    dx, dt, F = sc["dx"], sc["dt"], sc["F"]
    eta, l0 = DAMAGE["eta"], 0.5 * dx
    on = torch.zeros_like(history)
    history = history.clone()
    for q0, cnt, material, E, nu, _, _ in damaged_ranges:
        r = slice(q0, q0 + cnt)
        on[r] = 1
        history[r] = torch.maximum(history[r], _drive(F[r], material, E, nu, sc["sigma_c"][r]))
    vol = on * sc["V0"] * _det(F)
    c, e = vol * (1 + dt / eta * (history + 1)), vol * (dt / eta) * l0**2 / dx**2

    def gather(u):
        return sum(u[at(*o)][:, None] * gradient(*o) for o in offsets)

    def scatter(value):
        out = torch.zeros_like(pf)
        for o in offsets:
            out.index_add_(0, at(*o), value(o))
        return out

    diag = scatter(lambda o: weight(*o) * c)
    rhs = scatter(lambda o: weight(*o) * vol * history * (dt / eta)) + pf * scatter(lambda o: weight(*o) * vol)
    inside = diag > 0
    inv = torch.where(inside, 1 / torch.where(inside, diag, torch.ones_like(diag)), torch.zeros_like(diag))

    def apply(u):
        g = e[:, None] * gather(u)
        return torch.where(inside, diag * u + scatter(lambda o: (g * gradient(*o)).sum(1)), torch.zeros_like(u))

    u, res = torch.zeros_like(rhs), torch.where(inside, rhs, torch.zeros_like(rhs))
    z = inv * res
    p, zr_ = z, float((res * z).sum())
    tol, it = min(math.sqrt(zr_), 1e-6), 0
    while math.sqrt(zr_) > tol and it < 100:
        Ap = apply(p)
        a = zr_ / float((p * Ap).sum())
        u, res = u + a * p, res - a * Ap
        z = inv * res
        last, zr_ = zr_, float((res * z).sum())
        p = z + (zr_ / last) * p
        it += 1
    return history, torch.where(inside, u - pf, torch.zeros_like(pf))
