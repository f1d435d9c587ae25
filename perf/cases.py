"""Performance cases of the time-step engine: what its users run, through the public Python entry points.

A case is a whole call of a user's program on a simulation that it keeps: a forward run of a shot (reset, run,
seismograms and, where a program looks at it, the final wavefield), a streamed run (one call a step, a source row in and
a seismogram row out), a batch of shots, or a misfit gradient.  Meshes are rectangular grids, straight or with relief
(topography and bent layers), of 4- or 9-node quadrilaterals and 8-node hexahedra; models are constant layers or one
value per GLL point.  ``exact`` restates the discretisation (degree-4 spectral elements, Newmark time stepping, Stacey
edges, fluid-solid coupling) in plain 64-bit torch.
"""
import math
from types import SimpleNamespace

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from specfempp_b200 import adjoint
from specfempp_b200.sfg import Simulation2D
from specfempp_b200.sfg3d import Simulation3D

BOTTOM, RIGHT, TOP, LEFT = 0, 1, 2, 3
# saturated sandstone: rho_s, rho_f, phi, tortuosity, kxx, kxz, kzz, kappa_s, kappa_f, kappa_fr, eta_f, mu_fr, Q_mu
SANDSTONE = (2650.0, 880.0, 0.1, 2.0, 1e-9, 0.0, 1e-9, 12.2e9, 1.985e9, 9.6e9, 1e-3, 5.1e9, 9999.0)


def _case2d(kind, nx, nz, steps, nrec, relief=0.0, grf=False, nodes=4, shots=1, types="displacement", field=True,
            interval=0, nsrc=1):
    return {"kind": kind, "nx": nx, "nz": nz, "steps": steps, "nrec": nrec, "relief": relief, "grf": grf,
            "nodes": nodes, "shots": shots, "types": types, "field": field, "interval": interval, "nsrc": nsrc}


def _case3d(nx, ny, nz, steps, nrec, relief=0.0, types="displacement"):
    return {"kind": "elastic3d", "nx": nx, "ny": ny, "nz": nz, "steps": steps, "nrec": nrec, "relief": relief,
            "types": types}


def listed():
    named = {
        # a host program that streams source values in and samples out, one call a step, on a small mesh: latency
        "stream_psv_80x60": dict(_case2d("psv", 80, 60, 40, 5, field=False), stream=True),
        # the small elastic model of the configurations: a step is a few microseconds of work
        "psv_80x60": _case2d("psv", 80, 60, 800, 5),
        # the fluid-solid model of the configurations: water over four layers, receivers along the seafloor
        "coupled_400x200": _case2d("coupled", 400, 200, 800, 200),
        # a survey mesh with topography and a velocity model given per GLL point, odd sizes, two seismogram types
        "psv_relief_301x177": _case2d("psv", 301, 177, 600, 61, relief=0.3, grf=True, types="displacement,velocity"),
        # SH waves on curved 9-node elements
        "sh_curved_257x130": _case2d("sh", 257, 130, 600, 33, relief=0.3, nodes=9),
        # a water tank, pressure records
        "acoustic_500x250": _case2d("acoustic", 500, 250, 600, 100, types="pressure"),
        # fluid-saturated rock, viscous, four components a point
        "poro_150x150": _case2d("poro", 150, 150, 400, 6),
        # a 32-shot batch on one point model (a sixth of the configurations' mesh)
        "batch32_400x200": _case2d("psv", 400, 200, 120, 64, grf=True, shots=32, field=False),
        # waveform misfit and its gradient for one source of an inversion on the initial (constant) model
        "gradient_250x125": _case2d("psv", 250, 125, 600, 50, grf=False, interval=100),
        # a fluid-solid mesh with relief: nothing in it is straight
        "coupled_relief_181x121": _case2d("coupled", 181, 121, 800, 100, relief=0.25),
        # 3D: a small box and a layered model with heterogeneity per GLL point, free top and Stacey elsewhere
        "elastic3d_13x11x9": _case3d(13, 11, 9, 300, 20, types="displacement,velocity"),
        "elastic3d_48x48x32": _case3d(48, 48, 32, 150, 200),
    }
    return [dict(case, name=name) for name, case in named.items()]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["psv", "psv", "sh", "acoustic", "coupled", "coupled", "poro", "batch", "gradient", "stream",
                       "elastic3d", "elastic3d"])
    relief = rng.choice([0.0, round(rng.uniform(0.1, 0.35), 3)])
    if kind == "elastic3d":
        nx, ny = _log(rng, 8, 48), _log(rng, 8, 48)
        nz = _log(rng, 6, min(32, 70000 // (nx * ny)))
        return _case3d(nx, ny, nz, rng.randint(40, 150), rng.randint(3, 200), relief=relief,
                       types=rng.choice(["displacement", "displacement,velocity"]))
    if kind == "batch":
        shots = rng.choice([2, 4, 6, 8, 12, 16, 20, 32])
        nx = _log(rng, 40, 320)
        return _case2d(rng.choice(["psv", "psv", "sh"]), nx, _log(rng, 30, 160), rng.randint(40, 120), rng.randint(5, 80),
                       relief=relief, grf=rng.random() < 0.5, shots=shots, field=False)
    nx = _log(rng, 40, 400)
    nz = _log(rng, 30, 200)
    if kind == "gradient":
        nx, nz = min(nx, 230), min(nz, 120)
        return _case2d(rng.choice(["psv", "psv", "sh"]), nx, nz, rng.randint(120, 600), rng.randint(5, 60), relief=relief,
                       grf=rng.random() < 0.5, interval=rng.randint(20, 90))
    if kind == "stream":
        return dict(_case2d(rng.choice(["psv", "sh", "acoustic"]), nx, nz, rng.randint(20, 80), rng.randint(1, 100),
                            relief=relief, field=False), stream=True)
    if kind == "poro":
        return _case2d("poro", min(nx, 160), min(nz, 150), rng.randint(100, 400), rng.randint(1, 20), relief=relief)
    types = {"acoustic": ["pressure", "displacement"], "coupled": ["displacement"]}.get(
        kind, ["displacement", "displacement,velocity", "acceleration"])
    nodes = rng.choice([4, 4, 9]) if kind != "coupled" else 4
    return _case2d(kind, nx, nz, rng.randint(100, 800), rng.randint(1, 200), relief=relief,
                   grf=kind in ("psv", "sh") and rng.random() < 0.4, nodes=nodes, types=rng.choice(types),
                   nsrc=rng.randint(1, 3) if kind != "coupled" else 1)


# ------------------------------------------------------------------------------------------------------- inputs ---

H = 50.0            # element width in metres
NODES = np.array([-1.0, -math.sqrt(3 / 7), 0.0, math.sqrt(3 / 7), 1.0])
WEIGHTS = np.array([0.1, 49 / 90, 32 / 45, 49 / 90, 0.1])


def _smooth(rng, n, shape, coords):
    """A smooth field of unit size: a few plane waves of seeded direction and phase."""
    out = np.zeros(shape, np.float32)
    for _ in range(n):
        k = rng.normal(size=len(coords)) * 2 * math.pi / (14 * H)
        p = np.float32(rng.uniform(0, 2 * math.pi))
        for c, kc in zip(coords, k):
            p = p + c.astype(np.float32) * np.float32(kc)
        out += np.sin(p, dtype=np.float32)
    return out / np.float32(math.sqrt(n / 2))


def _relief(x, width, z, height, amp):
    return z + amp * H * np.sin(2 * math.pi * 3 * x / width + 0.7) * (z / height) + \
        0.5 * amp * H * np.sin(2 * math.pi * 7 * x / width) * np.sin(math.pi * z / height)


def _grid2d(case):
    """Control nodes and elements of an nx x nz grid (bottom row first)."""
    nx, nz, m = case["nx"], case["nz"], 2 if case["nodes"] == 9 else 1
    width, height = nx * H, nz * H
    xs, zs = np.linspace(0.0, width, m * nx + 1), np.linspace(0.0, height, m * nz + 1)
    Z, X = np.meshgrid(zs, xs, indexing="ij")
    if case["relief"]:
        Z = _relief(X, width, Z, height, case["relief"])
    iz, ix = np.divmod(np.arange(nx * nz), nx)
    at = lambda dx, dz: (m * iz + dz) * (m * nx + 1) + m * ix + dx  # noqa: E731
    order = [(0, 0), (m, 0), (m, m), (0, m)]
    if m == 2:
        order += [(1, 0), (2, 1), (1, 2), (0, 1), (1, 1)]
    knods = np.stack([at(dx, dz) for dx, dz in order], 1).astype(np.int32)
    return np.stack([X.ravel(), Z.ravel()], 1), knods, ix, iz


def _shape(nodes, xi, ga):
    """Shape functions and their xi / gamma derivatives, [..., nodes]."""
    if nodes == 4:
        fx, fg = [(1 - xi) / 2, (1 + xi) / 2], [(1 - ga) / 2, (1 + ga) / 2]
        dx, dg = [-0.5 + 0 * xi, 0.5 + 0 * xi], [-0.5 + 0 * ga, 0.5 + 0 * ga]
        pairs = [(0, 0), (1, 0), (1, 1), (0, 1)]
    else:
        q = lambda t: [t * (t - 1) / 2, 1 - t * t, t * (t + 1) / 2]  # noqa: E731
        d = lambda t: [t - 0.5, -2 * t, t + 0.5]  # noqa: E731
        fx, fg, dx, dg = q(xi), q(ga), d(xi), d(ga)
        pairs = [(0, 0), (2, 0), (2, 2), (0, 2), (1, 0), (2, 1), (1, 2), (0, 1), (1, 1)]
    return (np.stack([fx[a] * fg[b] for a, b in pairs], -1), np.stack([dx[a] * fg[b] for a, b in pairs], -1),
            np.stack([fx[a] * dg[b] for a, b in pairs], -1))


def _inside(p):
    """The points, moved to at least a twentieth of an element from every element edge."""
    k = np.floor(p / H)
    return (k + np.clip(p / H - k, 0.05, 0.95)) * H


def _inputs2d(case, seed):
    """Mesh, model, sources and receivers: what a user's program hands over."""
    rng = np.random.default_rng(seed)
    kind, nx, nz = case["kind"], case["nx"], case["nz"]
    coorg, knods, ix, iz = _grid2d(case)
    kmato = np.zeros(nx * nz, np.int32)
    vp = float(rng.uniform(2400.0, 2900.0))
    mats = [(1, 2200.0, vp, vp / 1.73)]
    mat_poro = None
    n_el = nz
    if kind == "acoustic":
        mats = [(0, 1020.0, 1500.0, 0.0)]
    elif kind == "coupled":
        n_el = nz - max(2, round(0.15 * nz))
        mats = [(1, 1700.0 + 0.2 * v, v, v / 1.73) for v in rng.uniform(2500.0, 4500.0, 4)] + [(0, 1020.0, 1500.0, 0.0)]
        kmato = np.where(iz >= n_el, 4, np.minimum(3, iz * 4 // n_el)).astype(np.int32)
    elif kind == "poro":
        mat_poro = np.array([SANDSTONE], np.float64) * (1 + 0.02 * rng.uniform(-1, 1, 13))
        mat_poro[0, 5], mat_poro[0, 12] = 0.0, 9999.0
        mats = [(1, 2400.0, 0.0, 0.0)]
    med = np.array([m[0] for m in mats], np.int32)
    sides = [] if kind == "poro" else [(iz == 0, BOTTOM), (ix == nx - 1, RIGHT), (ix == 0, LEFT)]
    none = np.zeros(0, np.int32)
    abs_i = np.concatenate([np.nonzero(s)[0] for s, _ in sides]).astype(np.int32) if sides else none
    abs_t = np.concatenate([np.full(s.sum(), t) for s, t in sides]).astype(np.int32) if sides else none
    free = np.nonzero((iz == nz - 1) & (med[kmato] == 0))[0].astype(np.int32)
    mesh = SimpleNamespace(
        nspec=nx * nz, npgeo=len(coorg), ngnod=case["nodes"], coorg=coorg, knods=knods, kmato=kmato, mat_medium=med,
        mat_rho=np.array([m[1] for m in mats]), mat_vp=np.array([m[2] for m in mats]),
        mat_vs=np.array([m[3] for m in mats]), abs_ispec=abs_i, abs_type=abs_t, free_ispec=free,
        free_type=np.full(len(free), TOP, np.int32), mat_poro=mat_poro)
    point = {}
    vmax, vmin = max(m[2] for m in mats), min(m[3] or m[2] for m in mats)
    if kind == "poro":
        vmax, vmin = 3300.0, 1000.0
    if kind == "sh":
        vmax = mats[0][3]
    if case["grf"] or case["interval"]:
        g = NODES * 0.5 + 0.5
        gx = (ix[:, None] * H + np.tile(g, 5)[None] * H)
        gz = (iz[:, None] * H + np.repeat(g, 5)[None] * H)
        f = 1 + (0.05 * _smooth(rng, 6, gx.shape, (gx, gz)) if case["grf"] else np.zeros(gx.shape, np.float32))
        vpp = (vp * f).astype(np.float32)
        point = {"vp": vpp, "vs": (vpp / np.float32(1.73)).astype(np.float32),
                 "rho": (2200.0 * (0.5 + 0.5 * f)).astype(np.float32)}
        vmax = float(point["vs" if kind == "sh" else "vp"].max())
        vmin = float(point["vs"].min())
    thin = 1.0 - 2.5 * case["relief"] * max(1.0 / nz, 0.04)
    dt = (0.16 if case["relief"] or kind == "poro" else 0.25) * 0.1727 * H * thin / vmax
    # two elements a wavelength, or a shorter wavelet where the run is too short for its peak to leave the source
    f0 = max(vmin / (2.0 * H), 2.6 / (case["steps"] * dt)) * float(rng.uniform(1.0, 1.2))
    # sources in the middle part (in the water of a fluid-solid model), receivers around them
    nsrc = max(case["shots"], case["nsrc"])
    width, height = nx * H, nz * H
    zs = (n_el + min(2.5, 0.5 * (nz - n_el))) * H if kind == "coupled" else None
    src = [{"x": float(rng.uniform(0.35, 0.65) * width + 3.1), "z": float(zs + 1.7 if zs else rng.uniform(0.4, 0.7) * height),
            "f0": f0 * float(rng.uniform(0.8, 1.0)), "angle": float(rng.uniform(0, 180)),
            "shot": i if case["shots"] > 1 else 0} for i in range(nsrc)]
    nrec = case["nrec"]
    near = np.array([[s["x"], s["z"]] for s in src])[np.arange(nrec) % nsrc]
    off = np.stack([np.linspace(-1, 1, nrec) * min(10 * H, 0.3 * width), np.full(nrec, 0.6 * H)], 1)
    if case["shots"] > 1:
        off[:, 0] = rng.uniform(-0.9, 0.9, nrec) * H
    rec = near + off
    if kind == "coupled":       # along the seafloor, on the solid's side
        rec[:, 1] = (n_el - 0.3) * H
    # points in grid coordinates, off the element edges (where either element may hold them), then moved with the relief
    rec = _inside(rec)
    for s in src:
        s["x"], s["z"] = _inside(np.array([s["x"], s["z"]])).tolist()
    move = lambda p: (p[0], _relief(p[0], width, p[1], height, case["relief"]) if case["relief"] else p[1])  # noqa: E731
    for s in src:
        s["x"], s["z"] = move((s["x"], s["z"]))
    rec = np.array([move(p) for p in rec])
    return SimpleNamespace(mesh=mesh, point=point, dt=dt, src=src, rec=rec, factor=1e10, knods=knods, ix=ix, iz=iz,
                           types=case["types"].split(","))


def _source_values(inp, steps):
    """Ricker values [steps, sources]: a shot starts 1.2 periods before its lowest source's peak, and the others are
    shifted by the difference of their own starts."""
    start = {}
    for s in inp.src:
        start[s["shot"]] = min(start.get(s["shot"], math.inf), -1.2 / s["f0"])
    out = []
    for s in inp.src:
        t0 = start[s["shot"]]
        a = (math.pi * s["f0"] * (np.arange(steps) * inp.dt + t0 - (-1.2 / s["f0"] - t0))) ** 2
        out.append(inp.factor * (1 - 2 * a) * np.exp(-a))
    return np.stack(out, 1)


def _observed(inp, steps):
    """Recorded data of an inversion: a wavelet that arrives at each receiver with the distance, [steps, nrec, 2]."""
    s = inp.src[0]
    d = np.hypot(inp.rec[:, 0] - s["x"], inp.rec[:, 1] - s["z"])
    t = np.arange(steps)[:, None] * inp.dt - 1.2 / s["f0"] - d[None] / 2000.0
    a = (math.pi * s["f0"] * t) ** 2
    w = (1 - 2 * a) * np.exp(-a) * 1e10 / (2200.0 * 2000.0 ** 2) * 0.05
    return np.stack([w, -0.5 * w], -1).astype(np.float32)


def _inputs3d(case, seed):
    rng = np.random.default_rng(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    X, Y, Z = nx * H, ny * H, nz * H
    z, y, x = np.meshgrid(np.linspace(-Z, 0, nz + 1), np.linspace(0, Y, ny + 1), np.linspace(0, X, nx + 1), indexing="ij")
    if case["relief"]:
        z = z + case["relief"] * H * np.sin(2 * math.pi * 2 * x / X) * np.cos(2 * math.pi * y / Y) * (1 + z / Z)
    nodes = np.stack([x, y, z], -1).reshape(-1, 3)
    e = np.arange(nx * ny * nz)
    ex, ey, ez = e % nx, e // nx % ny, e // (nx * ny)
    g = NODES * 0.5 + 0.5
    gx = (ex[:, None] + np.tile(g, 25)[None]).astype(np.float32) * np.float32(H)
    gy = (ey[:, None] + np.tile(np.repeat(g, 5), 5)[None]).astype(np.float32) * np.float32(H)
    gz = (ez[:, None] + np.repeat(g, 25)[None]).astype(np.float32) * np.float32(H)
    vp = (3000 + 800 * (1 - gz / Z)) * (1 + np.float32(0.03) * _smooth(rng, 3, gx.shape, (gx, gy, gz)))
    vp = vp.astype(np.float32)
    vs = (vp / np.float32(1.73)).astype(np.float32)
    rho = (np.float32(1700) + np.float32(0.2) * vp).astype(np.float32)
    thin = 1.0 - 4 * case["relief"] / max(nz, 6)
    dt = 0.2 * 0.1727 * H * thin / float(vp.max())
    mesh = SimpleNamespace(nex=nx, ney=ny, nez=nz, nodes=nodes, rho=rho, vp=vp, vs=vs, absorbing=(1, 1, 1, 1, 1, 0))
    src = SimpleNamespace(x=0.5 * X + 7.0, y=0.5 * Y - 3.0, z=-0.45 * Z + 2.0, f0=max(float(vs.min()) / (2 * H), 2.6 / (case["steps"] * dt)), factor=1e15,
                          kind="moment_tensor", comp=tuple(float(c) for c in rng.normal(size=6)), tshift=0.0)
    n = case["nrec"]
    rec = np.stack([src.x + rng.uniform(-1, 1, n) * min(4 * H, 0.4 * X), src.y + rng.uniform(-1, 1, n) * min(4 * H, 0.4 * Y),
                    src.z + rng.uniform(-1, 1, n) * min(3 * H, 0.3 * Z)], -1)
    return SimpleNamespace(mesh=mesh, dt=dt, src=src, rec=_inside(rec), types=case["types"].split(","))


# ------------------------------------------------------------------------------------------------- prepare, run ---

def prepare(case, seed):
    """The simulation that a program keeps: mesh and model uploaded, sources and receivers placed."""
    if case["kind"] == "elastic3d":
        inp = _inputs3d(case, seed)
        sim = Simulation3D(inp.mesh, dt=inp.dt, nstep=case["steps"])
        sim.set_sources([inp.src])
        sim.set_receivers(inp.rec, inp.types)
        sim.initialize()
        return {"case": case, "sim": sim}
    inp = _inputs2d(case, seed)
    p = inp.point
    sim = Simulation2D(inp.mesh, dt=inp.dt, nstep=case["steps"], nshots=case["shots"],
                       elastic_wave="sh" if case["kind"] == "sh" else "psv",
                       point_rho=p.get("rho"), point_vp=p.get("vp"), point_vs=p.get("vs"))
    sources = [SimpleNamespace(x=s["x"], z=s["z"], f0=s["f0"], factor=inp.factor, angle=s["angle"], shot=s["shot"])
               for s in inp.src]
    sim.set_sources(sources)
    sim.set_receivers(inp.rec[:, 0], inp.rec[:, 1], types=inp.types)
    sim.initialize()
    state = {"case": case, "sim": sim}
    if case["interval"]:
        kappa, mu = adjoint.moduli(*(p[k].astype(np.float64) for k in ("rho", "vp", "vs")))
        state.update(sources=sources, rho=p["rho"], kappa=kappa.astype(np.float32), mu=mu.astype(np.float32),
                     observed=_observed(inp, case["steps"])[None])
    if case.get("stream"):
        rows = _source_values(inp, case["steps"]).astype(np.float32)
        state["rows"] = torch.from_numpy(rows).pin_memory().numpy() if torch.cuda.is_available() else rows
        state["out"] = np.zeros((case["steps"], len(inp.types), case["nrec"], 2), np.float32)
    return state


def run(state):
    case, sim = state["case"], state["sim"]
    if case.get("interval"):
        misfit, grads = adjoint.l2_misfit_gradient(sim, state["sources"], state["rho"], state["kappa"], state["mu"],
                                                   state["observed"], case["steps"], case["interval"])
        return {"misfit": misfit, "rho": grads[0], "kappa": grads[1], "mu": grads[2]}
    sim.reset()
    if case.get("stream"):
        rows, out = state["rows"], state["out"]
        for k in range(case["steps"]):
            sim.step_io(rows[k], out[k])
        return {"seismograms": out}
    sim.run(case["steps"])
    out = {"seismograms": sim.seismograms()}
    if case["kind"] == "elastic3d":
        out["u"] = sim.field("displacement")
    elif case["field"]:
        if case["kind"] != "acoustic":
            out["u"] = sim.field("elastic")
        if case["kind"] in ("acoustic", "coupled"):
            out["chi"] = sim.field("acoustic")
    return out


def work(case):
    """Per step: displacement and velocity read and written, the inverse mass and the model's words read (one set a GLL
    point of the mesh where the model is given per point, none where it is constant in layers); a gradient takes two
    forward sweeps' worth of state, its two sums and the recorded state both ways."""
    if case["kind"] == "elastic3d":
        loc = 125 * case["nx"] * case["ny"] * case["nz"]
        pts = (4 * case["nx"] + 1) * (4 * case["ny"] + 1) * (4 * case["nz"] + 1)
        return {"bytes": case["steps"] * (pts * 4.0 * (4 * 3 + 1) + loc * 8.0), "flops": case["steps"] * loc * 260.0}
    loc, pts = 25 * case["nx"] * case["nz"], (4 * case["nx"] + 1) * (4 * case["nz"] + 1)
    nc = {"psv": 2, "sh": 1, "acoustic": 1, "coupled": 2, "poro": 4}[case["kind"]]
    s = case["shots"]
    step = pts * 4.0 * (4 * nc * s + 1) + loc * (8.0 if case["grf"] else 0.0)
    flops = loc * s * (60.0 * nc)
    if case["interval"]:
        step = 2 * step + pts * 4.0 * (4 * nc) + loc * 16.0 + loc * 8.0
        flops *= 3
    return {"bytes": case["steps"] * step, "flops": case["steps"] * flops}


def tolerance(case):
    """32-bit fields over hundreds of steps: measured against the 64-bit restatement, times about four (accelerations and
    the pressure, second derivatives in time, carry the most rounding; of a gradient the bulk modulus does)."""
    if case.get("interval"):
        return {"rel": 1e-4, "max": 1e-2}
    if "acceleration" in case["types"] or "pressure" in case["types"]:
        return {"rel": 2e-4, "max": 1e-2}
    return {"rel": 2e-5, "max": 1e-3}


# -------------------------------------------------------------------------------------------------------- exact ---

def _gll():
    """The 5x5 derivative matrix D[i, j] = l_j'(x_i)."""
    D = np.zeros((5, 5))
    for j in range(5):
        for i in range(5):
            for k in range(5):
                if k != j:
                    D[i, j] += np.prod([(NODES[i] - NODES[m]) if m not in (j, k) else 1.0 for m in range(5)]) / \
                        np.prod([NODES[j] - NODES[m] for m in range(5) if m != j])
    return D


def _lag(x):
    h = np.array([np.prod([(x - NODES[m]) / (NODES[j] - NODES[m]) for m in range(5) if m != j]) for j in range(5)])
    return h, h @ _gll_cache


_gll_cache = _gll()


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _locate(coorg, knods, nodes, ix, iz, nx, nz, p):
    """Element and local coordinates of a point: the grid cell by x, then the row by Newton."""
    best = None
    col = min(nx - 1, max(0, int(p[0] // H)))
    row0 = min(nz - 1, max(0, int(p[1] // H)))
    for row in sorted(range(max(0, row0 - 12), min(nz, row0 + 13)), key=lambda r: abs(r - row0)):
        e = row * nx + col
        c = coorg[knods[e]]
        xi = ga = 0.0
        for _ in range(12):
            s, dx, dg = _shape(nodes, np.float64(xi), np.float64(ga))
            r = p - s @ c
            J = np.stack([dx @ c, dg @ c], 1)
            d = np.linalg.solve(J, r)
            xi, ga = xi + d[0], ga + d[1]
        m = max(abs(xi), abs(ga))
        if best is None or m < best[0]:
            best = (m, e, min(1.0, max(-1.0, xi)), min(1.0, max(-1.0, ga)))
        if m <= 1.0:
            break
    return best[1:]


class _Grid2D:
    """The discretisation of one case in 64 bits."""

    def __init__(self, case, seed, inp):
        self.case, self.inp = case, inp
        self.nx, self.nz = nx, nz = case["nx"], case["nz"]
        m, dev = inp.mesh, _dev()
        self.T = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)
        ga, xi = np.meshgrid(NODES, NODES, indexing="ij")
        s, dx, dg = (a.reshape(25, -1) for a in _shape(m.ngnod, xi, ga))
        c = m.coorg[m.knods]
        xx, zx = c[:, :, 0] @ dx.T, c[:, :, 1] @ dx.T
        xg, zg = c[:, :, 0] @ dg.T, c[:, :, 1] @ dg.T
        J = xx * zg - xg * zx
        self.J = self.T(J)
        # J times d xi / d x, d xi / d z, d gamma / d x, d gamma / d z
        self.A = [self.T(a) for a in (zg, -xg, -zx, xx)]
        gi = (4 * inp.iz[:, None] + np.repeat(np.arange(5), 5)[None]) * (4 * nx + 1) + 4 * inp.ix[:, None] + \
            np.tile(np.arange(5), 5)[None]
        self.ib = self.T(gi)
        self.npts = (4 * nx + 1) * (4 * nz + 1)
        self.W = self.T(np.outer(WEIGHTS, WEIGHTS).ravel())
        self.D = self.T(_gll_cache)
        self.w = self.T(WEIGHTS)
        med = m.mat_medium[m.kmato]
        self.el = self.T(np.nonzero(med == 1)[0])
        self.ac = self.T(np.nonzero(med == 0)[0])
        # Stacey: per element point weight and unnormalised normal, later edges win
        st = {}
        for e, t in zip(m.abs_ispec, m.abs_type):
            d = st.setdefault(int(e), {})
            for i in range(5):
                q = {BOTTOM: i, TOP: 20 + i, LEFT: 5 * i, RIGHT: 5 * i + 4}[int(t)]
                sg = -1.0 if t in (BOTTOM, LEFT) else 1.0
                n = (-zx[e, q], xx[e, q]) if t in (BOTTOM, TOP) else (zg[e, q], -xg[e, q])
                d[q] = (WEIGHTS[i], sg * n[0], sg * n[1])
        rows = [(e, q, *v) for e, d in st.items() for q, v in d.items()]
        rows = np.array(rows).reshape(-1, 5)
        e, q = rows[:, 0].astype(np.int64), rows[:, 1].astype(np.int64)
        self.st = {}
        for name, sel in (("el", med[e] == 1), ("ac", med[e] == 0)):
            r = rows[sel]
            self.st[name] = SimpleNamespace(e=self.T(e[sel]), q=self.T(q[sel]), g=self.T(gi[e[sel], q[sel]]),
                                            w=self.T(r[:, 2].copy()), nx=self.T(r[:, 3].copy()), nz=self.T(r[:, 4].copy()))
        keep = np.ones((m.nspec, 25))
        keep[m.free_ispec, 20:] = 0.0
        self.keep = self.T(keep)
        # model per GLL point
        p = inp.point
        per = lambda k, v: self.T(p[k].astype(np.float64)) if k in p else self.T(np.repeat(v[m.kmato][:, None], 25, 1))  # noqa: E731
        self.rho, vp, vs = per("rho", m.mat_rho), per("vp", m.mat_vp), per("vs", m.mat_vs)
        self.mu = self.rho * vs ** 2
        self.kappa = torch.where(self.T(med == 1)[:, None], self.rho * (vp ** 2 - 4 / 3 * vs ** 2), self.rho * vp ** 2)
        if m.mat_poro is not None:
            v = m.mat_poro[0]
            Db = v[7] * (1 + v[2] * (v[7] / v[8] - 1))
            f = 1 / (Db - v[9])
            rb = (1 - v[2]) * v[0] + v[2] * v[1]
            self.poro = SimpleNamespace(H=(v[7] - v[9]) ** 2 * f + v[9] + 4 / 3 * v[11], C=v[7] * (v[7] - v[9]) * f,
                                        M=v[7] ** 2 * f, mu=v[11], pt=v[2] / v[3], rr=v[1] / rb, ex=v[10] / v[4],
                                        ez=v[10] / v[6], ms=rb - v[2] * v[1] / v[3],
                                        mf=(v[1] * v[3] * rb - v[2] * v[1] ** 2) / (v[2] * rb))
        # fluid-solid interface: horizontal edges between a solid element and the water element above it
        below = np.nonzero((med[:-nx] == 1) & (med[nx:] == 0))[0]
        self.cp = None
        if len(below):
            g = gi[below][:, 20:].ravel()
            nxx, nzz = (-zx[below][:, 20:] * WEIGHTS).ravel(), (xx[below][:, 20:] * WEIGHTS).ravel()
            self.cp = SimpleNamespace(g=self.T(g), nx=self.T(nxx), nz=self.T(nzz))
        # sources and receivers
        loc = lambda pt: _locate(m.coorg, m.knods, m.ngnod, inp.ix, inp.iz, nx, nz, np.asarray(pt))  # noqa: E731
        self.med = med
        self.src = []
        stf = _source_values(inp, case["steps"])
        for i, sc in enumerate(inp.src):
            e, x, g = loc((sc["x"], sc["z"]))
            h = np.outer(_lag(g)[0], _lag(x)[0]).ravel()
            self.src.append((e, self.T(gi[e]), self.T(h), self.T(stf[:, i]), sc["angle"] * math.pi / 180, sc["shot"]))
        R = [loc(pt) for pt in inp.rec]
        self.rec_e = self.T(np.array([r[0] for r in R]))
        self.rec_h = self.T(np.array([np.outer(_lag(r[2])[0], _lag(r[1])[0]).ravel() for r in R]))
        self.rec_ac = med[np.array([r[0] for r in R])] == 0

    def grad(self, U, e):
        """J times the physical derivatives (d/dx, d/dz) of U [ne, 25, ...]."""
        V = U.reshape(U.shape[0], 5, 5, -1)
        dx = torch.einsum("ij,ezjc->ezic", self.D, V).reshape(U.shape)
        dg = torch.einsum("ij,ejxc->eixc", self.D, V).reshape(U.shape)
        sh = (-1, 25) + (1,) * (U.dim() - 2)
        A = [a[e].reshape(sh) for a in self.A]
        return A[0] * dx + A[2] * dg, A[1] * dx + A[3] * dg

    def div(self, Sx, Sz, e):
        """Minus the weak divergence of the flux (Sx, Sz) [ne, 25, ...]."""
        sh = (-1, 25) + (1,) * (Sx.dim() - 2)
        A = [a[e].reshape(sh) for a in self.A]
        W = self.W.reshape((1, 25) + (1,) * (Sx.dim() - 2))
        F0 = (W * (A[0] * Sx + A[1] * Sz)).reshape(Sx.shape[0], 5, 5, -1)
        F1 = (W * (A[2] * Sx + A[3] * Sz)).reshape(Sx.shape[0], 5, 5, -1)
        r = torch.einsum("ji,ezjc->ezic", self.D, F0) + torch.einsum("ji,ejxc->eixc", self.D, F1)
        return -r.reshape(Sx.shape)

    def assemble(self, r, e, like):
        return torch.zeros_like(like).index_add(0, self.ib[e].reshape(-1), r.reshape((-1,) + r.shape[2:]))

    def model(self, rho, kappa, mu):
        """Everything that depends on the model: differentiable in rho, kappa, mu."""
        dt, m = self.inp.dt, SimpleNamespace()
        kind = self.case["kind"]
        m.mu, m.l2m, m.rho, m.kappa = mu, kappa + 4 / 3 * mu, rho, kappa
        m.nc = {"sh": 1, "acoustic": 1, "poro": 4}.get(kind, 2)
        zero = torch.zeros(self.npts, dtype=torch.float64, device=rho.device)
        if len(self.el):
            e, s = self.el, self.st["el"]
            mass = torch.index_add(zero, 0, self.ib[e].reshape(-1), (rho * self.W * self.J)[e].reshape(-1))
            m.minv_el = torch.stack([mass] * m.nc, 1)
            if kind == "poro":
                one = torch.index_add(zero, 0, self.ib.reshape(-1), (self.W * self.J).reshape(-1))
                P = self.poro
                m.minv_el = torch.stack([P.ms * one] * 2 + [P.mf * one] * 2, 1)
            j1 = torch.sqrt(s.nx ** 2 + s.nz ** 2)
            rr, rm, rl = rho[s.e, s.q], mu[s.e, s.q], m.l2m[s.e, s.q]
            m.rvp, m.rvs = torch.sqrt(rl * rr), torch.sqrt(rm * rr)
            if m.nc == 1:
                m.minv_el = m.minv_el.index_add(0, s.g, (dt / 2 * s.w * j1 * m.rvs)[:, None])
            elif kind != "poro":
                f = torch.stack([((s.nx + s.nz) * n / j1 ** 2) * (m.rvp - m.rvs) + m.rvs for n in (s.nx, s.nz)], 1)
                m.minv_el = m.minv_el.index_add(0, s.g, dt / 2 * (s.w * j1)[:, None] * f)
            m.minv_el = 1 / m.minv_el
        if len(self.ac):
            e, s = self.ac, self.st["ac"]
            mass = torch.index_add(zero, 0, self.ib[e].reshape(-1), (self.W * self.J / kappa)[e].reshape(-1))
            m.imp = 1 / torch.sqrt(rho[s.e, s.q] * kappa[s.e, s.q])
            j1 = torch.sqrt(s.nx ** 2 + s.nz ** 2)
            m.minv_ac = 1 / mass.index_add(0, s.g, dt / 2 * s.w * j1 * m.imp)
        return m

    def elastic(self, m, u, v):
        """Forces on the solid, u and v [npts, nc, shots]."""
        e, s, kind = self.el, self.st["el"], self.case["kind"]
        gx, gz = self.grad(u[self.ib[e]], e)
        iJ = (1 / self.J[e])[..., None]
        if kind == "poro":
            P = self.poro
            gx, gz = gx * iJ[..., None], gz * iJ[..., None]
            lam, dv, dw = P.H - 2 * P.mu, gx[:, :, 0] + gz[:, :, 1], gx[:, :, 2] + gz[:, :, 3]
            sxx = P.H * gx[:, :, 0] + lam * gz[:, :, 1] + P.C * dw
            szz = P.H * gz[:, :, 1] + lam * gx[:, :, 0] + P.C * dw
            sxz = P.mu * (gz[:, :, 0] + gx[:, :, 1])
            sp = P.C * dv + P.M * dw
            Sx = torch.stack([sxx - P.pt * sp, sxz, sp - P.rr * sxx, -P.rr * sxz], 2)
            Sz = torch.stack([sxz, szz - P.pt * sp, -P.rr * sxz, sp - P.rr * szz], 2)
            r = self.div(Sx, Sz, e)
            vv = v[self.ib[e]]
            f = (self.W * self.J[e])[..., None]
            dx, dz = f * P.ex * vv[:, :, 2], f * P.ez * vv[:, :, 3]
            return self.assemble(r + torch.stack([P.pt * dx, P.pt * dz, -dx, -dz], 2), e, u)
        mu, l2m = m.mu[e][..., None] * iJ, m.l2m[e][..., None] * iJ
        if m.nc == 1:
            r = self.div(mu[:, :, None] * gx, mu[:, :, None] * gz, e)
        else:
            lam = l2m - 2 * mu
            sxx = l2m * gx[:, :, 0] + lam * gz[:, :, 1]
            szz = l2m * gz[:, :, 1] + lam * gx[:, :, 0]
            sxz = mu * (gz[:, :, 0] + gx[:, :, 1])
            r = self.div(torch.stack([sxx, sxz], 2), torch.stack([sxz, szz], 2), e)
        out = self.assemble(r, e, u)
        j1 = torch.sqrt(s.nx ** 2 + s.nz ** 2)
        vs = v[s.g]
        if m.nc == 1:
            t = (s.w * j1 * m.rvs)[:, None, None] * vs
        else:
            n = torch.stack([s.nx, s.nz], 1)[..., None]
            vn = (vs * n).sum(1, keepdim=True)
            t = (s.w * j1)[:, None, None] * (vn * n / (j1 ** 2)[:, None, None] * (m.rvp - m.rvs)[:, None, None] +
                                             m.rvs[:, None, None] * vs)
        return out.index_add(0, s.g, -t)

    def acoustic(self, m, u, v):
        e, s = self.ac, self.st["ac"]
        gx, gz = self.grad(u[self.ib[e]], e)
        k = 1 / (self.J[e] * m.rho[e])
        r = self.div(k * gx, k * gz, e)
        j1 = torch.sqrt(s.nx ** 2 + s.nz ** 2)
        pos = torch.full((self.inp.mesh.nspec,), -1, dtype=torch.int64, device=u.device)
        pos[e] = torch.arange(len(e), device=u.device)
        r = r.index_put((pos[s.e], s.q), -s.w * j1 * m.imp * v[s.g], accumulate=True) * self.keep[e]
        return self.assemble(r, e, u)

    def sources(self, m, step, kind, f_el, f_ac):
        for e, g, h, f, ang, shot in self.src:
            if self.med[e] == 0:
                f_ac = f_ac.index_add(0, g, -f[step] * h / m.kappa[e])
                continue
            if kind == "sh":
                d = [1.0]
            elif kind == "poro":
                fs, ff = 1 - self.poro.pt, 1 - self.poro.rr
                d = [math.sin(ang) * fs, math.cos(ang) * fs, math.sin(ang) * ff, math.cos(ang) * ff]
            else:
                d = [math.sin(ang), math.cos(ang)]
            t = torch.zeros((25,) + f_el.shape[1:], dtype=torch.float64, device=h.device)
            t[:, :, shot] = f[step] * h[:, None] * torch.tensor(d, dtype=torch.float64, device=h.device)
            f_el = f_el.index_add(0, g, t)
        return f_el, f_ac

    def step(self, m, k, ue, ve, ae, ua, va, aa):
        dt, kind = self.inp.dt, self.case["kind"]
        if ue is not None:
            ue, ve = ue + dt * ve + dt * dt / 2 * ae, ve + dt / 2 * ae
        if ua is not None:
            ua, va = ua + dt * va + dt * dt / 2 * aa, va + dt / 2 * aa
        fe = self.elastic(m, ue, ve) if ue is not None else None
        fa = self.acoustic(m, ua, va) if ua is not None else None
        fe, fa = self.sources(m, k, kind, fe, fa)
        if ua is not None:
            if self.cp:
                u = ue[self.cp.g, :, 0]
                fa = fa.index_add(0, self.cp.g, -(self.cp.nx * u[:, 0] + self.cp.nz * u[:, 1]))
            aa = fa * m.minv_ac
            aa = torch.where(torch.isfinite(aa), aa, torch.zeros_like(aa)) if self.cp else aa
            va = va + dt / 2 * aa
        if ue is not None:
            if self.cp:
                x = aa[self.cp.g]
                fe = fe.index_add(0, self.cp.g, torch.stack([self.cp.nx * x, self.cp.nz * x], 1)[..., None])
            ae = fe * m.minv_el[..., None]
            ae = torch.where(torch.isfinite(ae), ae, torch.zeros_like(ae)) if self.cp else ae
            ve = ve + dt / 2 * ae
        return ue, ve, ae, ua, va, aa

    def record(self, m, st):
        """[types, nrec, 2, shots]"""
        ue, ve, ae, ua, va, aa = st
        out = []
        for t in self.inp.types:
            k = {"displacement": 0, "velocity": 1, "acceleration": 2, "pressure": 2}[t]
            o = torch.zeros((len(self.rec_e), 2, self.case["shots"]), dtype=torch.float64, device=self.rec_h.device)
            if ue is not None:
                f = (ue, ve, ae)[k][self.ib[self.rec_e]]
                r = torch.einsum("rq,rqcs->rcs", self.rec_h, f[:, :, :2])
                o = torch.cat([r, torch.zeros_like(r)], 1) if r.shape[1] == 1 else r
            elif t == "pressure":
                p = -(self.rec_h * aa[self.ib[self.rec_e]]).sum(1)
                o = torch.stack([p, torch.zeros_like(p)], 1)[..., None]
            else:
                f = (ua, va, aa)[k][self.ib[self.rec_e]]
                gx, gz = self.grad(f, self.rec_e)
                s = self.rec_h / (self.J * m.rho)[self.rec_e]
                o = torch.stack([(s * gx).sum(1), (s * gz).sum(1)], 1)[..., None]
            out.append(o)
        return torch.stack(out)

    def zero(self, m):
        z = lambda *n: torch.zeros(n, dtype=torch.float64, device=self.rec_h.device)  # noqa: E731
        e = [z(self.npts, m.nc, self.case["shots"]) for _ in range(3)] if len(self.el) else [None] * 3
        a = [z(self.npts) for _ in range(3)] if len(self.ac) else [None] * 3
        return (*e, *a)


def _exact2d(case, seed):
    inp = _inputs2d(case, seed)
    G = _Grid2D(case, seed, inp)
    steps = case["steps"]
    if not case["interval"]:
        with torch.no_grad():
            m = G.model(G.rho, G.kappa, G.mu)
            st, rec = G.zero(m), []
            for k in range(steps):
                st = G.step(m, k, *st)
                rec.append(G.record(m, st))
        seis = torch.stack(rec).permute(4, 0, 1, 2, 3)        # [shots, steps, types, nrec, 2]
        if case.get("stream"):
            return {"seismograms": seis[0]}
        out = {"seismograms": seis}
        if case["field"]:                                     # the handle numbers its points as it likes
            out.update({k: None for k in ("u", "chi")
                        if (k == "u" and case["kind"] != "acoustic") or (k == "chi" and case["kind"] in ("acoustic", "coupled"))})
        return out
    par = [G.rho.clone()] + [G.T(a) for a in _moduli(inp)]
    obs = G.T(_observed(inp, steps).astype(np.float64))
    for p in par:
        p.requires_grad_(True)
    n = 15                                                    # steps kept at once

    def chunk(k0, k1, rho, kappa, mu, *st):
        m = G.model(rho, kappa, mu)
        st = (*st, None, None, None)
        L = 0.0
        for k in range(k0, k1):
            st = G.step(m, k, *st)
            L = L + 0.5 * ((G.record(m, st)[0, :, :, 0] - obs[k]) ** 2).sum()
        return (L, *st[:3])

    st, L = G.zero(G.model(*par))[:3], 0.0
    for k0 in range(0, steps, n):
        dL, *st = checkpoint(chunk, k0, min(k0 + n, steps), *par, *st, use_reentrant=False)
        L = L + dL
    L.backward()
    return {"misfit": float(L.detach()), "rho": par[0].grad, "kappa": par[1].grad, "mu": par[2].grad}


def _moduli(inp):
    """kappa and mu as the program hands them over (32-bit values)."""
    rho, vp, vs = (inp.point[k].astype(np.float64) for k in ("rho", "vp", "vs"))
    mu = rho * vs * vs
    kappa = rho * vp * vp - 4.0 / 3.0 * mu
    return kappa.astype(np.float32).astype(np.float64), mu.astype(np.float32).astype(np.float64)


def _exact3d(case, seed):
    inp = _inputs3d(case, seed)
    m, dev = inp.mesh, _dev()
    T = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)  # noqa: E731
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dt = inp.dt
    e = np.arange(nx * ny * nz)
    ex, ey, ez = e % nx, e // nx % ny, e // (nx * ny)
    cs = np.array([[a, b, c] for c in (-1, 1) for b in (-1, 1) for a in (-1, 1)], float)
    idx = np.stack([((ez + (c[2] > 0)) * (ny + 1) + ey + (c[1] > 0)) * (nx + 1) + ex + (c[0] > 0) for c in cs], 1)
    C = T(m.nodes[idx])                                       # [ne, 8, 3]

    def shape(x, y, z):
        f = np.stack([(1 + c[0] * x) * (1 + c[1] * y) * (1 + c[2] * z) / 8 for c in cs], -1)
        d = [np.stack([c[0] * (1 + c[1] * y) * (1 + c[2] * z) / 8 for c in cs], -1),
             np.stack([c[1] * (1 + c[0] * x) * (1 + c[2] * z) / 8 for c in cs], -1),
             np.stack([c[2] * (1 + c[0] * x) * (1 + c[1] * y) / 8 for c in cs], -1)]
        return f, d

    gz, gy, gx = np.meshgrid(NODES, NODES, NODES, indexing="ij")
    _, d = shape(gx.ravel(), gy.ravel(), gz.ravel())
    dX = torch.stack([torch.einsum("qa,eaj->eqj", T(dk), C) for dk in d], -1)     # [ne, 125, j, k] = dx_j / dxi_k
    c0, c1, c2 = dX[..., 0], dX[..., 1], dX[..., 2]
    r0, r1, r2 = torch.cross(c1, c2, dim=-1), torch.cross(c2, c0, dim=-1), torch.cross(c0, c1, dim=-1)
    J = (c0 * r0).sum(-1)
    A = [r0, r1, r2]                                          # J d xi_k / d x_j
    del dX, c0, c1, c2
    NX, NY = 4 * nx + 1, 4 * ny + 1
    q = np.arange(125)
    qx, qy, qz = q % 5, q // 5 % 5, q // 25
    gi = ((4 * ez[:, None] + qz) * NY + 4 * ey[:, None] + qy) * NX + 4 * ex[:, None] + qx
    ib = T(gi)
    npts = NX * NY * (4 * nz + 1)
    w3 = (WEIGHTS[:, None, None] * WEIGHTS[None, :, None] * WEIGHTS[None, None, :]).ravel()
    W, D = T(w3), T(_gll_cache)
    rho, vp, vs = (T(a.astype(np.float64)) for a in (m.rho, m.vp, m.vs))
    mu, l2m = rho * vs ** 2, rho * vp ** 2
    mass = torch.zeros((npts, 3), dtype=torch.float64, device=dev)
    mass.index_add_(0, ib.reshape(-1), (rho * W * J).reshape(-1, 1).expand(-1, 3))
    faces = []
    for f in range(6):
        if not m.absorbing[f]:
            continue
        k, hi = divmod(f, 2)
        el = T(np.nonzero([ex, ey, ez][k] == ([nx, ny, nz][k] - 1 if hi else 0))[0])
        pts = np.nonzero([qx, qy, qz][k] == (4 if hi else 0))[0]
        wf = T(w3[pts] / 0.1)
        pts = T(pts)
        n = (1.0 if hi else -1.0) * A[k][el][:, pts]
        nn = n.norm(dim=-1, keepdim=True)
        rvp, rvs = ((rho * v)[el][:, pts][..., None] for v in (vp, vs))
        g = ib[el][:, pts].reshape(-1)
        wn = wf[None, :, None] * nn
        mass.index_add_(0, g, (dt / 2 * wn * (n.sum(-1, keepdim=True) * n / nn ** 2 * (rvp - rvs) + rvs)).reshape(-1, 3))
        faces.append((g, (n / nn).reshape(-1, 3), (wn * (rvp - rvs)).reshape(-1, 1), (wn * rvs).reshape(-1, 1)))
    minv = 1 / mass
    mu_, l2m_ = mu / J, l2m / J
    lam_ = l2m_ - 2 * mu_

    def locate(p):
        best = None
        col, row = min(nx - 1, max(0, int(p[0] // H))), min(ny - 1, max(0, int(p[1] // H)))
        for lay in range(nz):
            el = (lay * ny + row) * nx + col
            c = m.nodes[idx[el]]
            if not c[:, 2].min() - H <= p[2] <= c[:, 2].max() + H:
                continue
            s = np.zeros(3)
            for _ in range(12):
                f, dd = shape(*(np.float64(v) for v in s))
                s = s + np.linalg.solve(np.stack([k @ c for k in dd], 1), p - f @ c)
            t = np.abs(s).max()
            if best is None or t < best[0]:
                best = (t, el, np.clip(s, -1, 1))
        return best[1:]

    se, sx = locate(np.array([inp.src.x, inp.src.y, inp.src.z]))
    (hx, dx), (hy, dy), (hz, dz) = (_lag(v) for v in sx)
    k3 = lambda c, b, a: (c[:, None, None] * b[None, :, None] * a[None, None, :]).ravel()  # noqa: E731
    h = k3(hz, hy, hx)
    inv = torch.stack([(T(h)[:, None] * (A[k] / J[..., None])[se]).sum(0) for k in range(3)])   # [k, j]
    dxi = T(np.stack([k3(hz, hy, dx), k3(hz, dy, hx), k3(dz, hy, hx)], 1))
    cp = inp.src.comp
    M = T(np.array([[cp[0], cp[3], cp[4]], [cp[3], cp[1], cp[5]], [cp[4], cp[5], cp[2]]]))
    arr = (dxi @ inv) @ M
    t = np.arange(case["steps"]) * dt - 1.2 / inp.src.f0
    a2 = (math.pi * inp.src.f0 * t) ** 2
    stf = inp.src.factor * (1 - 2 * a2) * np.exp(-a2)
    R = [locate(p) for p in inp.rec]
    re = T(np.array([r[0] for r in R]))
    rh = T(np.array([k3(_lag(r[1][2])[0], _lag(r[1][1])[0], _lag(r[1][0])[0]) for r in R]))
    u, v, a = (torch.zeros((npts, 3), dtype=torch.float64, device=dev) for _ in range(3))
    out = []
    for k in range(case["steps"]):
        u, v = u + dt * v + dt * dt / 2 * a, v + dt / 2 * a
        U = u[ib].reshape(-1, 5, 5, 5, 3)
        dU = [torch.einsum("ezyxc,ix->ezyic", U, D).reshape(-1, 125, 3),
              torch.einsum("ezyxc,iy->ezixc", U, D).reshape(-1, 125, 3),
              torch.einsum("ezyxc,iz->eiyxc", U, D).reshape(-1, 125, 3)]
        # J du_c / dx_j = sum_k A[k][j] dU[k][c]
        gr = [[sum(A[kk][..., j] * dU[kk][..., c] for kk in range(3)) for j in range(3)] for c in range(3)]
        tr = gr[0][0] + gr[1][1] + gr[2][2]
        S = [[(lam_ * tr + 2 * mu_ * gr[c][c]) if c == j else mu_ * (gr[c][j] + gr[j][c]) for j in range(3)] for c in range(3)]
        r = torch.zeros_like(U)
        for kk, sb in enumerate(("ezyxc,xi->ezyic", "ezyxc,yi->ezixc", "ezyxc,zi->eiyxc")):
            F = torch.stack([W * sum(S[c][j] * A[kk][..., j] for j in range(3)) for c in range(3)], -1)
            r -= torch.einsum(sb, F.reshape(U.shape), D)
        f = torch.zeros_like(u).index_add_(0, ib.reshape(-1), r.reshape(-1, 3))
        for g, n, d1, d2 in faces:
            vv = v[g]
            f.index_add_(0, g, -(d1 * (vv * n).sum(-1, keepdim=True) * n + d2 * vv))
        f.index_add_(0, ib[se], float(stf[k]) * arr)
        a = f * minv
        v = v + dt / 2 * a
        out.append(torch.stack([torch.einsum("rq,rqc->rc", rh, {"displacement": u, "velocity": v}[ty][ib[re]])
                                for ty in inp.types]))
    return {"seismograms": torch.stack(out), "u": u}


def exact(case, seed):
    return _exact3d(case, seed) if case["kind"] == "elastic3d" else _exact2d(case, seed)
