"""Performance cases of the library: the calls its users make, at their sizes.

A case is one call sequence through the public Python entry points
(``tam_gb300.Context`` and the batch functions) on the geometries of
``tam_gb300.workloads``:

  heat    a grid of heat steps: upload a temperature field, take ``steps``
          fused steps, download temperature and damage
  mc      one Monte Carlo pass with its normalised tally brought to the host
  ref     the reference's coupled loop (reference mode) from its initial
          state: ``iters`` outer iterations, then the fields a run writes out
  batch   many uneven instances: one batched MC pass, then batched heat steps

``exact`` restates the heat step in plain torch FP64; the Monte Carlo walks
have no such value (a pass is a sample).
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("tissue-ablation-mc_gb300"))
import tam_gb300 as tam  # noqa: E402
from tam_gb300 import workloads as wl  # noqa: E402

T0 = 310.15
FOREVER = 1.0e9  # mJ per W: a source that stays on for the whole of every run


def listed():
    return [
        # a host loop that takes one step per call on a small grid and reads the
        # temperature back: launches and call overhead
        {"name": "heat call 64", "kind": "heat", "geometry": "cube", "nx": 64, "ny": 64, "nz": 64, "steps": 1, "fp32": True, "on": True},
        # the benchmark cube: 2 s of heating at its stable step
        {"name": "heat cube 200", "kind": "heat", "geometry": "cube", "nx": 200, "ny": 200, "nz": 200, "steps": 821, "fp32": True, "on": True},
        # a grid cut to the tissue at hand: rows of odd length
        {"name": "heat ragged 151", "kind": "heat", "geometry": "cube", "nx": 151, "ny": 150, "nz": 149, "steps": 400, "fp32": True, "on": True},
        # the plain FP64 form on the small configuration: 1 s of heating
        {"name": "heat cube 100 fp64", "kind": "heat", "geometry": "cube", "nx": 100, "ny": 100, "nz": 100, "steps": 103, "fp32": False, "on": True},
        # the vessel grid between two laser pulses (most of a pulsed run)
        {"name": "heat vessels 384", "kind": "heat", "geometry": "vessels", "nx": 384, "ny": 384, "nz": 384, "steps": 400, "fp32": True, "on": False},
        # a quick look: few packets, where one packet's walk is the time
        {"name": "mc call 100", "kind": "mc", "geometry": "cube", "nx": 100, "ny": 100, "nz": 100, "packets": 10_000, "fp32": True},
        # the benchmark pass
        {"name": "mc cube 200", "kind": "mc", "geometry": "cube", "nx": 200, "ny": 200, "nz": 200, "packets": 100_000_000, "fp32": True},
        # the plain FP64 form on the small configuration
        {"name": "mc cube 100 fp64", "kind": "mc", "geometry": "cube", "nx": 100, "ny": 100, "nz": 100, "packets": 1_000_000, "fp32": False},
        # a pass through vessels and inclusions on a grid whose tally exceeds L2
        {"name": "mc vessels 384", "kind": "mc", "geometry": "vessels", "nx": 384, "ny": 384, "nz": 384, "packets": 10_000_000, "fp32": True},
        # the Fortran program's own loop and grid, in its precision ...
        {"name": "ref loop 80 fp64", "kind": "ref", "n": 80, "iters": 96, "power": 2.0, "fp32": False},
        # ... and in the precision form
        {"name": "ref loop 80 fp32", "kind": "ref", "n": 80, "iters": 96, "power": 2.0, "fp32": True},
        # a parameter study: uneven instances side by side
        {"name": "batch 16", "kind": "batch", "instances": 16, "layout": 4, "lo": 64, "hi": 192, "packets": 300_000, "steps": 256},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("heat", "heat", "heat", "mc", "mc", "mc", "ref", "batch"))
    if kind == "heat":
        fp32 = rng.random() < 0.75
        geometry = rng.choice(("cube", "layers", "vessels"))
        hi = 256 if fp32 else 112
        nx, ny, nz = (rng.randint(48, hi) for _ in range(3))
        if rng.random() < 0.5:
            nx = nx // 4 * 4
        steps = _log(rng, 1, 800)
        return {"kind": kind, "geometry": geometry, "nx": nx, "ny": ny, "nz": nz, "steps": steps if fp32 else min(steps, 200), "fp32": fp32,
                "on": rng.random() < 0.6}
    if kind == "mc":
        fp32 = rng.random() < 0.75
        geometry = rng.choice(("cube", "cube", "layers", "vessels"))
        nx, ny, nz = (rng.randint(60, 360 if fp32 else 128) for _ in range(3))
        return {"kind": kind, "geometry": geometry, "nx": nx, "ny": ny, "nz": nz, "packets": _log(rng, 1_000, 20_000_000 if fp32 else 1_000_000), "fp32": fp32}
    if kind == "ref":
        n, power = rng.randint(40, 96), round(rng.uniform(0.5, 3.0), 2)
        # up to ~150 K of heating at the beam: evaporation, no ablation
        most = max(1, min(160, int(200 / (power * (80.0 / n) ** 2))))
        return {"kind": kind, "n": n, "iters": _log(rng, 1, most), "power": power, "fp32": rng.random() < 0.5}
    return {"kind": kind, "instances": rng.randint(3, 24), "layout": rng.randint(1, 10_000), "lo": 48, "hi": rng.randint(96, 192),
            "packets": _log(rng, 10_000, 500_000), "steps": _log(rng, 1, 300)}


# ------------------------------------------------------------ geometries --
def _half(case):
    """Half-widths (cm): the 1 cm cube, the 1 x 1 x 0.5 cm slab or the 2 cm vessel block, the longest grid edge setting the voxel size."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    edge = {"cube": 1.0, "layers": 1.0, "vessels": 2.0}[case["geometry"]] / max(nx, ny, nz)
    return nx * edge / 2, ny * edge / 2, nz * edge / 2


def _grid(case):
    """Material ids (u8, torch on the GPU, [z, y, x]) and the materials of the geometry."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    hx, hy, hz = _half(case)
    if case["geometry"] == "cube":
        return None, [wl.AIR, wl.TISSUE]
    if case["geometry"] == "layers":
        depth = 2 * hz - (torch.arange(nz, device="cuda", dtype=torch.float64) + 0.5) * (2 * hz / nz)
        ids = torch.full((nz,), 3, dtype=torch.uint8, device="cuda")
        ids[depth < 0.21] = 2
        ids[depth < 0.01] = 1
        ids[nz - 1] = 1
        return ids[:, None, None].expand(nz, ny, nx).contiguous(), [wl.AIR, wl.EPIDERMIS, wl.DERMIS, wl.SUBCUTIS]
    rng = np.random.Generator(np.random.Philox(5))  # the same vessels at every size
    L = np.array([2 * hx, 2 * hy, 2 * hz])
    grid = torch.ones((nz, ny, nx), dtype=torch.uint8, device="cuda")
    x, y, z = ((torch.arange(n, device="cuda", dtype=torch.float32) + 0.5) * float(w / n) for n, w in zip((nx, ny, nz), L))
    X, Y, Z = x[None, None, :], y[None, :, None], z[:, None, None]
    for _ in range(20):
        v = rng.normal(size=3)
        v /= np.linalg.norm(v)
        p, r = rng.uniform(0.0, 1.0, size=3) * L, float(rng.uniform(0.01, 0.05))
        dx, dy, dz = X - float(p[0]), Y - float(p[1]), Z - float(p[2])
        t = dx * float(v[0]) + dy * float(v[1]) + dz * float(v[2])
        grid[dx * dx + dy * dy + dz * dz - t * t <= r * r] = 2
    for _ in range(5):
        p = rng.uniform(0.05, 0.95, size=3) * L
        grid[(X - float(p[0])) ** 2 + (Y - float(p[1])) ** 2 + (Z - float(p[2])) ** 2 <= 0.1 ** 2] = 3
    return grid, [wl.AIR, wl.DERMIS, wl.BLOOD, wl.INCLUSION]


def _host(t):
    """A [z, y, x] tensor as the library's (x, y, z) Fortran-ordered array."""
    return t.cpu().numpy().transpose(2, 1, 0)


def _context(case, packets=1, power=2.0, on=True):
    hx, hy, hz = _half(case)
    grid, mats = _grid(case)
    p = tam.default_params(nxg=case["nx"], nyg=case["ny"], nzg=case["nz"], xmax=hx, ymax=hy, zmax=hz, mode=1, precision=1 if case["fp32"] else 0,
                           nphotons=packets, pulse_type=1, power=power, energy_per_pixel=power * (FOREVER if on else 1e-9), total_time=1e9, loops=1,
                           repetition_rate_1=1e9, pulses_to_do=1)
    c = tam.default_config(nmat=len(mats), retrace_fraction=0.0)
    for i, m in enumerate(mats):
        tam.set_material(c, i, *m)
    ctx = tam.Context(p, c)
    if grid is not None:
        ctx.upload(tam.TAM_F_MATERIAL, _host(grid))
    return ctx


def _fields(case, seed):
    """The heat inputs: a temperature with the beam's hot core (up to the damage window, below boiling) and an absorbed
    power per W that falls off around the beam and with depth; both as FP32 values, [z, y, x] FP64 on the GPU."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    hx, hy, hz = _half(case)
    rng = np.random.Generator(np.random.Philox(int(seed)))
    cx, cy = hx * rng.uniform(0.85, 1.15), hy * rng.uniform(0.85, 1.15)
    rise, wide, deep = rng.uniform(15.0, 24.0), rng.uniform(0.12, 0.2), rng.uniform(0.2, 0.35)
    x, y, z = ((torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) * (2 * h / n) for n, h in ((nx, hx), (ny, hy), (nz, hz)))
    r2 = (x[None, None, :] - cx) ** 2 + (y[None, :, None] - cy) ** 2
    d = (2 * hz - z)[:, None, None]
    J = 2.0e7 * rng.uniform(0.8, 1.2) * torch.exp(-r2 / 0.02 - d / 0.33)
    temp = T0 + rise * torch.exp(-r2 / (2 * wide * wide) - d / deep)
    return temp.float().double(), J.float().double()


def _halo(t):
    out = torch.full(tuple(n + 2 for n in t.shape), T0, dtype=torch.float64, device="cuda")
    out[1:-1, 1:-1, 1:-1] = t
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "heat":
        ctx = _context(case, on=case["on"])
        temp, J = _fields(case, seed)
        ctx.upload(tam.TAM_F_JMEAN_GLOBAL, _host(J))
        if not case["on"]:
            ctx.heat_steps(2)  # the pulse ends here: the steps that follow have no source
            ctx.upload(tam.TAM_F_TISSUE, np.zeros((case["nx"], case["ny"], case["nz"]), order="F"))
        return {"case": case, "ctx": ctx, "temp": _host(_halo(temp))}
    if kind == "mc":
        return {"case": case, "ctx": _context(case, packets=case["packets"]), "seed": int(seed)}
    if kind == "ref":
        p = tam.default_params(nxg=case["n"], nyg=case["n"], nzg=case["n"], power=case["power"], pulse_type=tam._abi.TAM_PULSE_TOPHAT,
                               precision=1 if case["fp32"] else 0)
        return {"case": case, "ctx": tam.Context(p), "seed": int(seed)}
    ws = wl.c4(n=case["instances"], seed=case["layout"], packets=case["packets"], edge_range=(case["lo"], case["hi"]))
    return {"case": case, "ctxs": [w.context() for w in ws], "seeds": [int(seed) * 64 + k for k in range(len(ws))]}


def run(state):
    case = state["case"]
    if case["kind"] == "heat":
        ctx = state["ctx"]
        ctx.upload(tam.TAM_F_TEMP, state["temp"])
        return {"temp": ctx.heat_steps(case["steps"], want=True), "omega": ctx.download(tam.TAM_F_TISSUE)}
    if case["kind"] == "mc":
        ctx = state["ctx"]
        return {"jmean": ctx.mc_pass(case["packets"], seed=state["seed"], want=True), "tallies": ctx.tallies()}
    if case["kind"] == "ref":
        ctx = state["ctx"]
        ctx.init_thermal()
        ctx.step_coupled(case["iters"], seed=state["seed"])
        return {"temp": ctx.download(tam.TAM_F_TEMP), "omega": ctx.download(tam.TAM_F_TISSUE), "rhokap": ctx.download(tam.TAM_F_RHOKAP),
                "jmean": ctx.download(tam.TAM_F_JMEAN_GLOBAL)}
    ctxs = state["ctxs"]
    for c in ctxs:
        c.init_thermal()
    n = len(ctxs)
    tam.batch_mc_pass(ctxs, state["seeds"], nphotons=[case["packets"]] * n, streams=[0] * n)
    tam.batch_heat_steps(ctxs, case["steps"])
    return {"temp": [c.download(tam.TAM_F_TEMP) for c in ctxs], "omega": [c.download(tam.TAM_F_TISSUE) for c in ctxs]}


# ------------------------------------------------------------------ work --
def _heat_work(voxels, steps, fp32, on):
    # per step and voxel: T read and written (in FP64, or in FP32 with its compensation term) and the source read while it is on
    per = 16 + ((4 if fp32 else 8) if on else 0)
    return voxels * steps * per, voxels * steps * 28.0


def _mc_work(path, mus, h, packets, voxels, fp32):
    # mean path per packet (cm): 1.5 / h face crossings and mus scatters per cm
    # (12 and 120 operations each); the tally and its normalised copy written once
    return voxels * (8 + (4 if fp32 else 8)), packets * path * (12 * 1.5 / h + 120 * mus)


def work(case):
    kind = case["kind"]
    if kind == "heat":
        b, f = _heat_work(case["nx"] * case["ny"] * case["nz"], case["steps"], case["fp32"], case["on"])
    elif kind == "mc":
        path, mus = {"cube": (1.9, 100.0), "layers": (1.6, 100.0), "vessels": (4.0, 120.0)}[case["geometry"]]
        h = 2 * _half(case)[0] / case["nx"]
        b, f = _mc_work(path, mus, h, case["packets"], case["nx"] * case["ny"] * case["nz"], case["fp32"])
    elif kind == "ref":
        # per iteration and voxel: T, rhokap, J read, T, rhokap, J written; 125,000 packets of a few steps
        v = case["n"] ** 3
        b, f = case["iters"] * v * 48.0, case["iters"] * (v * 40.0 + 125_000 * 60.0)
    else:
        b = f = 0.0
        for q in wl.c4_instances(case["instances"], case["layout"], case["packets"], edge_range=(case["lo"], case["hi"])):
            v = q["edges"][0] * q["edges"][1] * q["edges"][2]
            for w in (_heat_work(v, case["steps"], True, True), _mc_work(0.8, q["mus"], 0.005, case["packets"], v, True)):
                b, f = b + w[0], f + w[1]
    return {"bytes": float(b), "flops": float(f)}


# ----------------------------------------------------------------- exact --
def exact(case, seed):
    """The heat cases in torch FP64: the 7-point step with face diffusivities from arithmetic means of k, rho, c, fixed
    faces at 310.15 K and a convective top face, the source, and Arrhenius damage between 43 and 100 C."""
    if case["kind"] != "heat" or case["nx"] * case["ny"] * case["nz"] * case["steps"] > 30e9:
        return None
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    hx, hy, hz = _half(case)
    temp, J = _fields(case, seed)
    grid, mats = _grid(case)
    k, rho, c = (torch.tensor([m[i] for m in mats], dtype=torch.float64, device="cuda") for i in (4, 5, 6))
    ids = torch.ones_like(temp, dtype=torch.long) if grid is None else grid.long()
    k, rho, c = k[ids], rho[ids], c[ids]
    del ids, grid
    d = [2e-2 * h / n for h, n in ((hx, nx), (hy, ny), (hz, nz))]
    dt = 0.9 / (2.0 * max(m[4] / (m[5] * m[6]) for m in mats[1:]) * sum(1.0 / (q * q) for q in d))
    inv = 1.0 / (rho * c)
    src = 2.0 * dt * J * inv if case["on"] else None
    own = k * inv

    def face(axis):
        a, b = [slice(None)] * 3, [slice(None)] * 3
        a[axis], b[axis] = slice(None, -1), slice(1, None)
        a, b = tuple(a), tuple(b)
        return a, b, dt / d[2 - axis] ** 2 * (0.5 * (k[a] + k[b])) / ((0.5 * (rho[a] + rho[b])) * (0.5 * (c[a] + c[b])))

    faces = [face(axis) for axis in range(3)]
    edges = [(axis, side, dt / d[2 - axis] ** 2 * own.select(axis, side)) for axis in range(3) for side in (0, -1)]
    robin = 10.0 * d[2] / k[-1]
    del inv, own, rho, c
    omega = torch.zeros_like(temp)
    lnA, EaR = math.log(3.1e98), 6.28e5 / 8.314
    for _ in range(case["steps"]):
        new = temp.clone()
        for a, b, w in faces:
            flux = w * (temp[b] - temp[a])
            new[a] += flux
            new[b] -= flux
        for axis, side, w in edges:
            t = temp.select(axis, side)
            top = axis == 0 and side == -1
            new.select(axis, side).add_(w * (-robin * (t - 298.15) if top else T0 - t))
        if src is not None:
            new += src
        temp = new
        hot = (temp >= 316.15) & (temp < 373.15)
        omega += torch.where(hot, dt * torch.exp(lnA - EaR / temp), 0.0)
    out = _halo(temp)
    # the written halo: the face's temperature (z faces over y faces over x faces), the convective face's ghost on top
    ghost = temp[-1] - robin * (temp[-1] - 298.15)
    ghost = torch.nn.functional.pad(ghost[None, None], (1, 1, 1, 1), mode="replicate")[0, 0]
    out[-1] = ghost
    return {"temp": _host(out), "omega": _host(omega)}
