"""The workloads whose speed is followed from change to change, as a user's program calls them.

    listed()            the cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what the program holds before the call: the simulation on the GPU, loaded
    run(state)          one pass through the public entry points, and its outputs
    work(case)          bytes and operations one pass cannot do without
    exact(case, seed)   the outputs of the first pass in 64-bit arithmetic, where they are computed

Kinds of case:

    steps      a simulation advanced by some gas steps, then its fields read (the library use: the benchmark's
               grids, its three pressure solvers, fixed and CFL time steps)
    frame      one frame of the campfire app without its host-side wood model: pieces and parameters up,
               geometry, the frame's gas steps with the reference's one V-cycle each, radiation, readback and
               the photo view (the app's three grids and time steps)
    batch      many scenes of uneven size advanced together, then every scene's fields read
    serve      jobs of several sizes handed to the continuous-batching server, and their results fetched
    render     one view of a scene as an image on the GPU
    radiation  the ray-cast radiation to wood faces and floor, read back
    monitor    the FP64 checks a long run makes now and then: pressure residual and mass / energy sums

Every scene is made here from the seed alone: separate wood pieces above the floor, hot and burning gas
plumes around them and a swirling velocity field of the speed a fire of that size has.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import campfire_b200 as cb
from campfire_b200.fluid import load_scene
from campfire_b200.render import VIEWS, Renderer, render_device

TAMB, YO_AMB, RHO_AMB = 300.0, 0.233, 101325.0 * 0.0289 / (8.314462 * 300.0)
ACC_PER_JOULE, ACC_PER_KG, ACC_PER_WATT = 1e6, 1e12, 1e3     # the readback's fixed-point scales
# the benchmark's batch sizes
CLASSES = ((96, 144), (128, 192), (192, 288), (256, 384))


def listed():
    return [
        # the smallest call: one step of a small scene with the reference's solver, and its fields (tests' size)
        {"name": "step 32x48", "kind": "steps", "nx": 32, "ny": 48, "width": 0.8, "pieces": 3, "mode": "fixed",
         "tol": 0.0, "w": 0, "cells": 6144, "cfl": 0.0, "dt": 0.002, "steps": 1},
        # FP32 cycles to a tolerance at a fixed 2 ms step (the smallest benchmark grid)
        {"name": "run 128x192 tol", "kind": "steps", "nx": 128, "ny": 192, "width": 0.8, "pieces": 3, "mode": "tol",
         "tol": 1e-4, "w": 0, "cells": 6144, "cfl": 0.0, "dt": 0.002, "steps": 10},
        # the headline: FP64 outer loop to 1e-6, CFL 0.5 capped at 2 ms
        {"name": "run 256x384 fp64", "kind": "steps", "nx": 256, "ny": 384, "width": 0.8, "pieces": 3,
         "mode": "fp64", "tol": 1e-6, "w": 0, "cells": 1536, "cfl": 0.5, "dt": 0.002, "steps": 20},
        # the fine grid to 1e-10 with the W tail
        {"name": "run 512x768 fp64", "kind": "steps", "nx": 512, "ny": 768, "width": 0.8, "pieces": 5,
         "mode": "fp64", "tol": 1e-10, "w": 1536, "cells": 1536, "cfl": 0.5, "dt": 0.002, "steps": 20},
        # the app's frames: coarse, balanced and fine grid, 16 pieces (its default fire has 16)
        {"name": "frame 160x224", "kind": "frame", "nx": 160, "ny": 224, "pieces": 16, "dt": 0.004, "steps": 4,
         "W": 480, "H": 704},
        {"name": "frame 224x320", "kind": "frame", "nx": 224, "ny": 320, "pieces": 16, "dt": 0.003, "steps": 5,
         "W": 734, "H": 1080},
        {"name": "frame 352x512", "kind": "frame", "nx": 352, "ny": 512, "pieces": 40, "dt": 0.002, "steps": 8,
         "W": 1468, "H": 2160},
        # 64 uneven scenes to 1e-10, one launch per kernel for all of them
        {"name": "batch 64", "kind": "batch", "scenes": 64, "steps": 20, "tol": 1e-10, "cells": 6144, "krylov": 2},
        # a burst of jobs at the server
        {"name": "serve 12 jobs", "kind": "serve", "jobs": 12, "steps": 40, "tol": 1e-10},
        # a full-window picture of a balanced scene
        {"name": "photo 734x1080", "kind": "render", "nx": 224, "ny": 320, "pieces": 16, "W": 734, "H": 1080,
         "view": "photo", "zoom": 1.0},
        # radiation alone (a coarser host loop asks for it more often than it steps)
        {"name": "radiation 352x512", "kind": "radiation", "nx": 352, "ny": 512, "width": 0.8, "pieces": 16,
         "nray": 64},
        # checks of the fine run
        {"name": "monitor 512x768", "kind": "monitor", "nx": 512, "ny": 768, "width": 0.8, "pieces": 5},
    ]


def _grid(rng, most):
    """A grid the multigrid hierarchy takes (a coarsest level of at most 256 cells), odd widths among them."""
    while True:
        a, b, k = rng.randint(5, 16), rng.randint(7, 24), rng.randint(2, 5)
        if a * b <= 256 and a < b <= 2 * a and 1500 <= (a * b) << (2 * k) <= most:
            return a << k, b << k


def draw(rng):
    kind = rng.choice(["steps"] * 5 + ["frame"] * 4 + ["batch", "serve", "render", "render", "radiation", "monitor"])
    if kind == "steps":
        nx, ny = _grid(rng, 512 * 768)
        mode = rng.choice(["fixed", "tol", "fp64", "fp64"])
        cfl = 0.5 if mode == "fp64" else rng.choice([0.0, 0.5])
        return {"kind": kind, "nx": nx, "ny": ny, "width": 0.8, "pieces": rng.randint(1, 8), "mode": mode,
                "tol": {"fixed": 0.0, "tol": 1e-4, "fp64": rng.choice([1e-6, 1e-8, 1e-10])}[mode],
                "w": 1536 if mode == "fp64" and rng.random() < 0.4 else 0, "cells": rng.choice([1536, 6144]), "cfl": cfl,
                "dt": 0.002 if cfl else 0.0025 * rng.uniform(0.2, 1.0), "steps": rng.randint(2, 16)}
    if kind == "frame":
        nx, ny = _grid(rng, 352 * 512)
        dt = rng.uniform(0.002, 0.004)
        h = int(round(math.exp(rng.uniform(math.log(400), math.log(2000)))))
        return {"kind": kind, "nx": nx, "ny": ny, "pieces": rng.randint(1, 40), "dt": dt, "steps": int(1 / 60 / dt),
                "W": max(1, h * nx // ny), "H": h}
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(2, 60), "steps": rng.randint(2, 16),
                "tol": rng.choice([1e-6, 1e-8, 1e-10]), "cells": 6144, "krylov": rng.choice([1, 2])}
    if kind == "serve":
        return {"kind": kind, "jobs": rng.randint(2, 12), "steps": rng.randint(10, 40), "tol": rng.choice([1e-6, 1e-8])}
    if kind == "render":
        nx, ny = _grid(rng, 352 * 512)
        h = int(round(math.exp(rng.uniform(math.log(300), math.log(2160)))))
        return {"kind": kind, "nx": nx, "ny": ny, "pieces": rng.randint(0, 40), "W": max(1, h * nx // ny), "H": h,
                "view": rng.choice(["photo", "photo", "temperature", "reaction", "oxygen", "fuel", "velocity", "soot"]),
                "zoom": rng.choice([1.0, 1.0, rng.uniform(1.5, 4.0)])}
    nx, ny = _grid(rng, 512 * 768)
    if kind == "radiation":
        return {"kind": kind, "nx": nx, "ny": ny, "width": 0.8, "pieces": rng.randint(1, 40),
                "nray": rng.choice([32, 64, 64, 128])}
    return {"kind": kind, "nx": nx, "ny": ny, "width": 0.8, "pieces": rng.randint(1, 8)}


# ------------------------------------------------------------------ scenes
def _pieces(rng, n, W, H, dx):
    """Up to n separate rotated squares above the floor in the lower half of the domain: 64 x 20 floats
    (position, angle, half side, velocity, spin, alive; per face temperature, fuel flux, char cover)."""
    a = np.zeros((64, 20), np.float32)
    size = min(0.05, 0.16 / math.sqrt(max(n, 1))) * W
    placed = []
    for _ in range(400 * max(n, 1)):
        if len(placed) == n:
            break
        h = size * rng.uniform(0.6, 1.0) * 0.5
        r = h * math.sqrt(2.0)
        x = rng.uniform(r + 0.1 * W, 0.9 * W - r)
        y = rng.uniform(r + 3 * dx, max(r + 4 * dx, 0.45 * H - r))
        if all(math.hypot(x - q[0], y - q[1]) >= r + q[2] + 4 * dx for q in placed):
            a[len(placed)] = [x, y, rng.uniform(-1.5, 1.5), h, 0, 0, 0, 1, *rng.uniform(500, 900, 4),
                              *rng.uniform(2e-3, 8e-3, 4), *rng.uniform(0, 1, 4)]
            placed.append((x, y, r))
    return a.ravel(), len(placed)


def _scene(nx, ny, width, npieces, seed, dt):
    """The scene as load_scene takes it."""
    rng = np.random.default_rng([int(seed), nx, ny])
    dx = width / nx
    H = dx * ny
    pieces, n = _pieces(rng, npieces, width, H, dx)
    x, y = (np.arange(nx) + 0.5) * dx, (np.arange(ny) + 0.5) * dx

    def blob(sx, sy):
        cx, cy = rng.uniform(0.25, 0.75) * width, rng.uniform(0.08, 0.6) * H
        return np.exp(-((y - cy) / (sy * H)) ** 2)[:, None] * np.exp(-((x - cx) / (sx * width)) ** 2)[None, :]

    hot = np.minimum(sum(rng.uniform(0.4, 1.0) * blob(rng.uniform(0.05, 0.12), rng.uniform(0.08, 0.25))
                         for _ in range(4)), 1.0)
    T = TAMB + 1500.0 * hot
    fuel = 0.25 * np.minimum(sum(blob(0.08, 0.08) for _ in range(3)), 1.0)
    Y = np.empty((ny, nx, 4))
    Y[..., 0] = fuel
    Y[..., 3] = 2e-3 * hot * blob(0.2, 0.3)
    Y[..., 1] = YO_AMB * (1.0 - fuel) * (1.0 - 0.8 * hot)
    Y[..., 2] = 1.0 - Y[..., 0] - Y[..., 1] - Y[..., 3]
    # swirls and an upward draught from a stream function (no divergence), 1.2 m/s at most, and some noise
    xv, yv = np.arange(nx + 1) * dx, np.arange(ny + 1) * dx
    psi = np.zeros((ny + 1, nx + 1))
    for _ in range(6):
        cx, cy, s = rng.uniform(0.2, 0.8) * width, rng.uniform(0.1, 0.8) * H, rng.uniform(0.06, 0.15) * width
        psi += rng.uniform(-1, 1) * s * np.exp(-((yv - cy) / s) ** 2)[:, None] * np.exp(-((xv - cx) / s) ** 2)[None, :]
    psi -= 0.15 * width * np.tanh((xv - 0.5 * width) / (0.15 * width))[None, :] * np.tanh(yv / (0.2 * H))[:, None]
    U, V = np.diff(psi, axis=0) / dx, -np.diff(psi, axis=1) / dx
    top = max(np.abs(U).max(), np.abs(V).max())
    U = U * (1.2 / top) + rng.uniform(-0.01, 0.01, U.shape)
    V = V * (1.2 / top) + rng.uniform(-0.01, 0.01, V.shape)
    params = {"Tamb": TAMB, "rhoAmb": float(np.float32(RHO_AMB)), "YOamb": YO_AMB, "reactB": 2e10, "reactTa": 15000.0,
              "dHc": 15.0e6, "Pr": 0.7, "exchAlpha": 0.05, "depth": 0.3}
    f = lambda a: np.ascontiguousarray(a, np.float32).ravel()   # noqa: E731
    return {"T": f(T), "Y": f(Y), "U": f(U), "V": f(V), "pieces": pieces, "npieces": n, "params": params, "dt": dt,
            "nx": nx, "ny": ny, "width": width}


def _wood_buffer(seed):
    """The renderer's wood buffer: Tp[4], d[4], char fraction, core temperature, irradiance, has virgin wood."""
    rng = np.random.default_rng([int(seed), 7])
    w = np.empty((64, 12), np.float32)
    w[:, 0:4] = rng.uniform(450, 800, (64, 4))
    w[:, 4:8] = rng.uniform(0.0005, 0.004, (64, 4))
    w[:, 8], w[:, 9], w[:, 10] = rng.uniform(0, 1, 64), rng.uniform(300, 600, 64), rng.uniform(0, 0.05, 64)
    w[:, 11] = rng.uniform(0, 1, 64) < 0.8
    return w.ravel()


def _batch_dims(case):
    return [CLASSES[k] for k in np.random.default_rng(11).integers(0, len(CLASSES), case["scenes"])]


def _rates(nx, ny, seed):
    """A heat release and divergence source field as the last step left it."""
    return np.random.default_rng([int(seed), 3]).uniform(0, 1, (ny, nx, 2)) * np.array([4.0, 2e6])


def _pressure(nx, ny, seed):
    rng = np.random.default_rng([int(seed), 5])
    x, y = np.linspace(0, 1, nx), np.linspace(0, 1, ny)
    p = sum(rng.uniform(-1, 1) * np.sin(rng.integers(1, 6) * np.pi * y)[:, None] *
            np.sin(rng.integers(1, 6) * np.pi * x)[None, :] for _ in range(5))
    return p + 0.01 * rng.uniform(-1, 1, (ny, nx))


# ------------------------------------------------------------------ what a program holds, and one pass
def _sim(case, seed, width, dt):
    sc = _scene(case["nx"], case["ny"], width, case["pieces"], seed, dt)
    sim = cb.FluidSim(0, {"nx": case["nx"], "ny": case["ny"], "dt": dt}, width=width).init()
    load_scene(sim, sc)
    return sim, sc


def prepare(case, seed):
    kind = case["kind"]
    if kind == "steps":
        sim, _ = _sim(case, seed, case["width"], case["dt"])
        if case["mode"] == "fixed":
            sim.set_solver(cb.SOLVE_FIXED, 1)
        elif case["mode"] == "tol":
            sim.set_solver(cb.SOLVE_TOL, 1, case["tol"], 50)
        else:
            sim.set_solver(cb.SOLVE_FP64, 1, case["tol"], 300)
            sim.set_coarse_solve("pipelined")
            sim.set_krylov(True)
        sim.set_coarse_cells(case["cells"])
        sim.set_coarse_w(case["w"])
        if case["cfl"] > 0:
            sim.set_cfl(case["cfl"], case["dt"])
        return {"kind": kind, "sim": sim, "steps": case["steps"]}
    if kind == "frame":
        sim, sc = _sim(case, seed, cb.SCENE_WIDTH, case["dt"])
        sim.set_solver(cb.SOLVE_FIXED, 1)
        st = torch.cuda.Stream()
        sim.set_stream(st.cuda_stream)
        ren = Renderer(sim)
        ren.writeWood(_wood_buffer(seed))
        return {"kind": kind, "sim": sim, "scene": sc, "steps": case["steps"], "stream": st, "ren": ren,
                "W": case["W"], "H": case["H"], "img": torch.empty(case["H"], case["W"], 4, device="cuda")}
    if kind == "batch":
        dims = _batch_dims(case)
        scenes = [_scene(nx, ny, 0.8, 2 + k % 5, seed * 100 + k, 0.002) for k, (nx, ny) in enumerate(dims)]
        b = cb.Batch(dims, 0.8, [0.002] * len(dims), device=0)
        for v, s in zip(b.scenes, scenes):
            load_scene(v, s)
        b.set_solver(cb.SOLVE_FP64, 1, case["tol"], 300)
        b.set_coarse_solve("pipelined")
        b.set_coarse_cells(case["cells"])
        b.set_krylov(case["krylov"])
        size = {"T": sum(x * y for x, y in dims), "Y": sum(4 * x * y for x, y in dims),
                "U": sum((x + 1) * y for x, y in dims), "V": sum(x * (y + 1) for x, y in dims)}
        return {"kind": kind, "batch": b, "steps": case["steps"],
                "out": {f: np.zeros(n, np.float32) for f, n in size.items()}}
    if kind == "serve":
        s = cb.Server(CLASSES, [3] * len(CLASSES), 100e9, device=0)
        s.set_solver(cb.SOLVE_FP64, 1, case["tol"], 300, coarse_direct=True, coarse_cells=6144, krylov=1)
        jobs = [(k % len(CLASSES), int(seed) * 100 + k, case["steps"] - (k % 5)) for k in range(case["jobs"])]
        return {"kind": kind, "server": s, "jobs": jobs}
    if kind == "render":
        sim, sc = _sim(case, seed, cb.SCENE_WIDTH, 0.003)
        sim.writeBuffer("SQ", _rates(case["nx"], case["ny"], seed))
        st = torch.cuda.Stream()
        sim.set_stream(st.cuda_stream)
        ren = Renderer(sim)
        ren.writeWood(_wood_buffer(seed))
        cam = None if case["zoom"] == 1.0 else {"x": 0.2, "y": 0.02, "zoom": case["zoom"]}
        ren.writeParams({"view": case["view"], "nPieces": sc["npieces"], "exposure": 1.0, "time": 0.0, "cam": cam})
        return {"kind": kind, "sim": sim, "stream": st, "ren": ren, "W": case["W"], "H": case["H"],
                "img": torch.empty(case["H"], case["W"], 4, device="cuda")}
    sim, _ = _sim(case, seed, case["width"], 0.002)
    if kind == "radiation":
        sim.set_nray(case["nray"])
        return {"kind": kind, "sim": sim, "frame": 0}
    sim.writeBuffer("SQ", _rates(case["nx"], case["ny"], seed))
    sim.run_stage("coef_rhs")
    sim.writeBuffer("p", _pressure(case["nx"], case["ny"], seed))
    return {"kind": kind, "sim": sim}


def _fields(sim):
    return {f: sim.readBuffer(f) for f in ("T", "Y", "U", "V")}


def _units(acc):
    """The accumulators in SI units, as the app converts them: heat to each wood face (J/m), char burnt (kg/m),
    heat release and radiative loss (J/m), peak temperature (K)."""
    faces = acc[:512].astype(np.float64).reshape(256, 2)
    return {"heat": (faces[:, 0] / ACC_PER_JOULE).astype(np.float32),
            "char": (faces[:, 1] / ACC_PER_KG).astype(np.float32),
            "total": (acc[512:514] / ACC_PER_WATT).astype(np.float32), "tmax": int(acc[514])}


def run(state):
    kind = state["kind"]
    if kind == "steps":
        state["sim"].encodeStep(n=state["steps"])
        return _fields(state["sim"])
    if kind == "frame":
        sim, sc, ren = state["sim"], state["scene"], state["ren"]
        sim.uploadPieces(sc["pieces"], sc["npieces"])
        sim.writeParams()
        sim.clearGeometry()
        sim.encodeGeometry()
        sim.encodeStep(n=state["steps"])
        sim.encodeRadiation()
        rb = sim.readback()
        sim.setFrame(sim.frame + 1)
        ren.writeParams({"view": 0, "exposure": 1.0, "time": sim.time})
        render_device(sim, ren.rp, state["W"], state["H"], state["img"].data_ptr(), ren.wood)
        return {**_units(rb["acc"]), "rad": rb["rad"], "faceW": rb["faceW"], "img": state["img"]}
    if kind == "batch":
        state["batch"].step(state["steps"])
        for f, out in state["out"].items():
            at = 0
            for v in state["batch"].scenes:
                a = v.readBuffer(f)
                out[at:at + a.size] = a
                at += a.size
        return state["out"]
    if kind == "serve":
        s = state["server"]
        tickets = [s.submit(c, 2, seed, n, keep_fields=True) for c, seed, n in state["jobs"]]
        out = {f: [] for f in ("T", "Y", "U", "V")}
        for t, (c, _, _) in zip(tickets, state["jobs"]):
            s.wait(t, 60.0)
            nx, ny = CLASSES[c]
            for f, n in (("T", nx * ny), ("Y", 4 * nx * ny), ("U", (nx + 1) * ny), ("V", nx * (ny + 1))):
                out[f].append(s.fetch(t, f, n))
            s.release(t)
        return out
    if kind == "render":
        render_device(state["sim"], state["ren"].rp, state["W"], state["H"], state["img"].data_ptr(),
                      state["ren"].wood)
        return state["img"]
    sim = state["sim"]
    if kind == "radiation":
        state["frame"] += 1
        sim.setFrame(state["frame"])
        sim.writeParams()
        sim.encodeRadiation()
        return sim.readback()["rad"]
    return {"residual": sim.pressure_residual(), "sums": sim.budgets()}


def work(case):
    """State (T, four species, two velocities) read and written once per step with the geometry beside it; the
    operations of a step by its formulas: about 1500 per cell outside the pressure solve, 90 per cell and V-cycle."""
    kind = case["kind"]
    if kind == "batch":
        cells = sum(a * b for a, b in CLASSES) / len(CLASSES) * case["scenes"]
    elif kind == "serve":
        cells = sum(a * b for a, b in CLASSES) / len(CLASSES) * case["jobs"]
    else:
        cells = case["nx"] * case["ny"]
    px = case.get("W", 0) * case.get("H", 0)
    if kind == "render":
        return {"bytes": 16.0 * px + 36.0 * cells, "flops": 900.0 * px if case["view"] == "photo" else 60.0 * px}
    if kind == "radiation":
        samples = (4 * case["pieces"] + 64) * case["nray"] * 0.5 * case["ny"]
        return {"bytes": 20.0 * cells, "flops": 60.0 * samples}
    if kind == "monitor":
        return {"bytes": 48.0 * cells, "flops": 60.0 * cells}
    fp64 = kind in ("batch", "serve") or case.get("mode") == "fp64"
    cycles = 10 if fp64 else 4 if case.get("mode") == "tol" else 1
    w = {"bytes": case["steps"] * cells * (72.0 + (16.0 if fp64 else 0.0)),
         "flops": case["steps"] * cells * (1500.0 + 90.0 * cycles)}
    if kind == "frame":
        samples = (4 * case["pieces"] + 64) * 64 * 0.5 * case["ny"]
        w = {"bytes": w["bytes"] + 16.0 * px + 36.0 * cells, "flops": w["flops"] + 900.0 * px + 60.0 * samples}
    return w


# ------------------------------------------------------------------ the same physics in 64-bit arithmetic
class _Exact:
    """The gas step's formulas on dense (row, column) tensors of doubles."""

    PHYS = {"cp": 1300.0, "sO2": 15.0 / 13.1, "sootFormA": 6.0e6, "sootFormTa": 25000.0, "sootOxA": 5.4e8,
            "sootOxTa": 19800.0, "kappaSootC": 1862.0, "kappaGas": 0.8, "charA": 6.6, "charTa": 5800.0,
            "sootDensity": 1800.0, "sigma": 5.670374e-8, "charO2": 2.667, "grav": 9.81}

    def __init__(self, sc, dt, cfl=0.0, w=0):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a: torch.as_tensor(np.asarray(a, np.float64), device=self.dev)   # noqa: E731
        self.nx, self.ny, self.dx = sc["nx"], sc["ny"], sc["width"] / sc["nx"]
        nx, ny = self.nx, self.ny
        self.T, self.Y = t(sc["T"]).view(ny, nx), t(sc["Y"]).view(ny, nx, 4)
        self.U, self.V = t(sc["U"]).view(ny, nx + 1), t(sc["V"]).view(ny + 1, nx)
        self.SQ = torch.zeros(ny, nx, 2, dtype=torch.float64, device=self.dev)
        self.p = torch.zeros(ny, nx, dtype=torch.float64, device=self.dev)
        self.P = {**self.PHYS, **sc["params"]}
        self.amb = t([0.0, self.P["YOamb"], 0.0, 0.0])
        self.dt = self.cap = dt
        self.cfl, self.w, self.inv = cfl, w, None
        self.pieces, self.np_ = t(sc["pieces"]).view(64, 20), sc["npieces"]
        self.heat, self.char = t(np.zeros(256)), t(np.zeros(256))
        self.total, self.tmax = t(np.zeros(2)), 0.0
        self.geometry()

    def _axis(self, n, off):
        return torch.arange(n, dtype=torch.float64, device=self.dev) + off

    def _points(self, h, w, oy, ox):
        y, x = torch.meshgrid(self._axis(h, oy), self._axis(w, ox), indexing="ij")
        return x, y

    # ---- geometry: distance to the nearest rotated square, open fractions of the faces
    def _nearest(self, px, py):
        best, who = torch.full_like(px, 1e9), torch.full_like(px, -1, dtype=torch.int64)
        for n in range(self.np_):
            q = self.pieces[n]
            c, s = torch.cos(q[2]), torch.sin(q[2])
            lx, ly = c * (px - q[0]) + s * (py - q[1]), -s * (px - q[0]) + c * (py - q[1])
            qx, qy = lx.abs() - q[3], ly.abs() - q[3]
            d = torch.hypot(qx.clamp(min=0), qy.clamp(min=0)) + torch.maximum(qx, qy).clamp(max=0)
            face = torch.where(lx.abs() > ly.abs(), torch.where(lx > 0, 0, 2), torch.where(ly > 0, 1, 3))
            near = d < best
            best, who = torch.where(near, d, best), torch.where(near, 4 * n + face, who)
        return best, who

    def geometry(self):
        nx, ny, dx = self.nx, self.ny, self.dx
        x, y = self._points(ny, nx, 0.5, 0.5)
        self.sdf, self.sid = self._nearest(x * dx, y * dx)
        wgt = (1 - (self.sdf - dx).abs() / dx).clamp(min=0) / dx
        m = (self.sid >= 0) & (self.sdf >= 0) & (self.sdf < 2 * dx)
        self.band = torch.zeros(256, dtype=torch.float64, device=self.dev)
        self.band.index_add_(0, self.sid[m], (wgt * dx * dx)[m])
        x, y = self._points(ny, nx + 1, 0.5, 0.0)
        self.fx = (0.5 + self._nearest(x * dx, y * dx)[0] / dx).clamp(0, 1)
        x, y = self._points(ny + 1, nx, 0.0, 0.5)
        self.fy = (0.5 + self._nearest(x * dx, y * dx)[0] / dx).clamp(0, 1)
        self.fy[0] = 0

    # ---- samplers: cells see the ambient outside, U a no-slip floor, V a clamped one
    def _at(self, f, kind, i, j, amb):
        h, w = f.shape[:2]
        v = f[j.clamp(0, h - 1), i.clamp(0, w - 1)]
        if kind == "U":
            v = torch.where(j < 0, -v, v)
        out = (i < 0) | (i >= w) | (j >= h)
        return torch.where(out.unsqueeze(-1) if f.dim() == 3 else out, amb, v)

    def _corners(self, f, kind, gx, gy, amb):
        ox, oy = {"C": (0.5, 0.5), "U": (0.0, 0.5), "V": (0.5, 0.0)}[kind]
        bx, by = torch.floor(gx - ox), torch.floor(gy - oy)
        i, j = bx.long(), by.long()
        q = [self._at(f, kind, i + a, j + b, amb) for b in (0, 1) for a in (0, 1)]
        return q, gx - ox - bx, gy - oy - by

    def _sample(self, f, kind, gx, gy, amb=None):
        (a, c, d, e), tx, ty = self._corners(f, kind, gx, gy, self._zero if amb is None else amb)
        if f.dim() == 3:
            tx, ty = tx.unsqueeze(-1), ty.unsqueeze(-1)
        return (a * (1 - tx) + c * tx) * (1 - ty) + (d * (1 - tx) + e * tx) * ty

    def _range(self, f, kind, gx, gy, amb=None):
        q, _, _ = self._corners(f, kind, gx, gy, self._zero if amb is None else amb)
        q = torch.stack(q)
        return q.amin(0), q.amax(0)

    @property
    def _zero(self):
        return torch.zeros((), dtype=torch.float64, device=self.dev)

    def _trace(self, gx, gy, dt):
        def vel(x, y):
            return self._sample(self.U, "U", x, y) / self.dx, self._sample(self.V, "V", x, y) / self.dx
        vx, vy = vel(gx, gy)
        vx, vy = vel(gx - 0.5 * dt * vx, gy - 0.5 * dt * vy)
        return gx - dt * vx, gy - dt * vy

    def _advect(self):
        nx, ny, dt = self.nx, self.ny, self.dt
        Ta = torch.tensor(self.P["Tamb"], dtype=torch.float64, device=self.dev)
        gx, gy = self._points(ny, nx, 0.5, 0.5)
        d, b = self._trace(gx, gy, dt), self._trace(gx, gy, -dt)
        Th, Yh = self._sample(self.T, "C", *d, Ta), self._sample(self.Y, "C", *d, self.amb)
        Tc = Th + 0.5 * (self.T - self._sample(Th, "C", *b, Ta))
        Yc = Yh + 0.5 * (self.Y - self._sample(Yh, "C", *b, self.amb))
        tl, th = self._range(self.T, "C", *d, Ta)
        yl, yh = self._range(self.Y, "C", *d, self.amb)
        s = self.P["sO2"]
        ok = (Tc >= tl) & (Tc <= th) & ((Yc >= yl) & (Yc <= yh)).all(-1)
        ok &= torch.minimum(Yc[..., 0], Yc[..., 1] / s) <= torch.minimum(Yh[..., 0], Yh[..., 1] / s) + 1e-5
        new = []
        for f, kind, pt in ((self.U, "U", self._points(ny, nx + 1, 0.5, 0.0)),
                            (self.V, "V", self._points(ny + 1, nx, 0.0, 0.5))):
            d, b = self._trace(*pt, dt), self._trace(*pt, -dt)
            fh = self._sample(f, kind, *d)
            lo, hi = self._range(f, kind, *d)
            new.append(torch.minimum(torch.maximum(fh + 0.5 * (f - self._sample(fh, kind, *b)), lo), hi))
        return torch.where(ok, Tc, Th), torch.where(ok.unsqueeze(-1), Yc, Yh), new[0], new[1]

    # ---- gas properties
    def _rho(self, T):
        return self.P["rhoAmb"] * self.P["Tamb"] / T

    @staticmethod
    def _mu(T):
        return 1.716e-5 * (T / 273.15) ** 1.5 * (273.15 + 110.4) / (T + 110.4)

    def _substeps(self):
        T = 2200.0
        alpha = (1.716e-5 * (T / 273.15) ** 1.5 * 383.55 / (T + 110.4) / 0.7 /
                 (101325 * 0.0289 / 8.314462 / T))
        n = math.ceil(self.dt / (self.dx ** 2 / (4.5 * alpha)))
        return max(1, min(5, n if n % 2 else n + 1))

    def _diffuse(self, T, Y):
        n = self._substeps()
        for _ in range(n):
            sT, sY = torch.zeros_like(T), torch.zeros_like(Y[..., :3])
            for ax, f in ((1, self.fx[:, 1:-1]), (0, self.fy[1:-1])):
                m = T.shape[ax]
                lo, hi = (slice(None),) * ax + (slice(0, m - 1),), (slice(None),) * ax + (slice(1, m),)
                a = f * self._mu(0.5 * (T[lo] + T[hi])) / self.P["Pr"]
                fT, fY = a * (T[hi] - T[lo]), a.unsqueeze(-1) * (Y[hi] - Y[lo])[..., :3]
                sT[lo] += fT
                sT[hi] -= fT
                sY[lo] += fY
                sY[hi] -= fY
            c = self.dt / n / (self._rho(T) * self.dx ** 2)
            T, Y = T + c * sT, torch.cat([Y[..., :3] + c.unsqueeze(-1) * sY, Y[..., 3:]], -1).clamp(min=0)
        return T, Y

    def _add(self, T, Y, madd, Ya, Ta, on):
        r = self._rho(T)
        Y2 = (r.unsqueeze(-1) * Y + madd.unsqueeze(-1) * Ya) / (r + madd).unsqueeze(-1)
        return torch.where(on, (r * T + madd * Ta) / (r + madd), T), torch.where(on.unsqueeze(-1), Y2, Y)

    def _sources(self, T, Y, Tadv):
        P, dx, dt = self.P, self.dx, self.dt
        cell = dx * dx
        T0, Y0 = T, Y
        pc = self.pieces[(self.sid.clamp(min=0) // 4)]
        face = (self.sid.clamp(min=0) % 4).unsqueeze(-1)
        Ts, mfl, cov = (pc[..., k:k + 4].gather(-1, face).squeeze(-1) for k in (8, 12, 16))
        solid = (self.sdf < 0) & (self.sid >= 0)
        wet = (self.sid >= 0) & (self.sdf < 2 * dx) & ~solid
        sid = self.sid.clamp(min=0)
        w = ((1 - (self.sdf - dx).abs() / dx).clamp(min=0) / dx * (2 * pc[..., 3]) / self.band[sid].clamp(min=1e-6))
        mass = torch.zeros_like(T)
        k = self._mu(0.5 * (T + Ts)) / P["Pr"] * P["cp"]
        rate = k * w / (self.sdf.clamp(min=0.5 * dx) * self._rho(T) * P["cp"])
        dT = torch.where(wet, (Ts - T) * (1 - torch.exp(-rate * dt)), self._zero)
        rho = self._rho(T)
        T = T + dT
        self.heat.index_add_(0, sid[wet], (-rho * P["cp"] * dT * cell)[wet])
        e = lambda k: torch.eye(4, dtype=torch.float64, device=self.dev)[k]   # noqa: E731
        mf = mfl * w
        on = wet & (mf > 0)
        T, Y = self._add(T, Y, mf * dt, e(0), Ts, on)
        mass = mass + torch.where(on, mf, self._zero)
        on = wet & (cov > 0) & (Y[..., 1] > 0)
        r = self._rho(T)
        kc = P["charA"] * torch.exp(-P["charTa"] / Ts.clamp(min=1.0)) * cov
        mO2 = torch.minimum(kc * r * Y[..., 1] * w * dt, 0.9 * r * Y[..., 1])
        mC = mO2 / P["charO2"]
        add = torch.stack([torch.zeros_like(mC), -mO2, mC + mO2, torch.zeros_like(mC)], -1)
        Yn = (r.unsqueeze(-1) * Y + add) / (r + mC).unsqueeze(-1)
        T, Y = torch.where(on, (r * T + mC * Ts) / (r + mC), T), torch.where(on.unsqueeze(-1), Yn, Y)
        mass = mass + torch.where(on, mC / dt, self._zero)
        self.char.index_add_(0, sid[on], (mC * cell)[on])
        rho0, burned = self._rho(T), torch.zeros_like(T)
        sO2 = P["sO2"]
        burn = torch.tensor([-1.0, -sO2, 1 + sO2, 0.0], dtype=torch.float64, device=self.dev)
        for _ in range(8):
            wr = P["reactB"] * rho0 * Y[..., 0] * Y[..., 1] * torch.exp(-P["reactTa"] / T)
            dF = torch.minimum(wr * dt / 8, torch.minimum(Y[..., 0], Y[..., 1] / sO2))
            Y = Y + dF.unsqueeze(-1) * burn
            T = T + dF * P["dHc"] / P["cp"]
            burned = burned + dF
        dS = torch.minimum(P["sootFormA"] * torch.exp(-P["sootFormTa"] / T) * Y[..., 0] * dt, Y[..., 0])
        Y = Y + dS.unsqueeze(-1) * (e(3) - e(0))
        dS = torch.minimum(P["sootOxA"] * Y[..., 3] * Y[..., 1] * torch.exp(-P["sootOxTa"] / T) * dt,
                           torch.minimum(Y[..., 3], Y[..., 1] / sO2))
        Y = Y + dS.unsqueeze(-1) * (burn + e(0) - e(3))
        T = T + dS * P["dHc"] / P["cp"]
        q = rho0 * (burned + dS) * P["dHc"] / dt
        r1 = self._rho(T)
        kap = P["kappaSootC"] * r1 * Y[..., 3] / P["sootDensity"] * T + P["kappaGas"] * Y[..., 2]
        qr = 4 * kap * P["sigma"] * (T ** 4 - P["Tamb"] ** 4)
        T = T - qr * dt / (r1 * P["cp"]) / (1 + 16 * kap * P["sigma"] * T ** 3 * dt / (r1 * P["cp"]))
        u, v = 0.5 * (self.U[:, 1:] + self.U[:, :-1]), 0.5 * (self.V[1:] + self.V[:-1])
        me = 2 * P["exchAlpha"] * torch.hypot(u, v) * P["rhoAmb"] / P["depth"]
        T, Y = self._add(T, Y, me * dt, self.amb, P["Tamb"], me > 0)
        mass = mass + me
        T, Y = T.clamp(min=0.5 * P["Tamb"]), Y.clamp(min=0)
        S = mass / self._rho(T) + torch.log(T / Tadv) / dt
        gas = ~solid
        self.total += torch.stack([(q * gas).sum(), (qr * gas).sum()]) * cell * dt
        self.tmax = max(self.tmax, float((T * gas).max()))
        self.SQ = torch.where(gas.unsqueeze(-1), torch.stack([S, q], -1), self._zero)
        return torch.where(gas, T, Ts), torch.where(gas.unsqueeze(-1), Y, Y0)

    def _forces(self, T, U2, V2):
        P, nx, ny, dx, dt = self.P, self.nx, self.ny, self.dx, self.dt
        u, v = torch.where(self.fx > 0, U2, self._zero), torch.where(self.fy > 0, V2, self._zero)
        mu = self._mu(T)
        Tv = 0.25 * (T[1:, 1:] + T[:-1, 1:] + T[1:, :-1] + T[:-1, :-1])      # inner corners
        muv = self._mu(Tv)

        def drag(spd, Tf):
            return torch.exp(-2 * P["exchAlpha"] * spd * (Tf / P["Tamb"]) / P["depth"] * dt)
        # U faces away from the sides
        Tf = 0.5 * (T[:, 1:] + T[:, :-1])
        c = U2[:, 1:-1]
        muf = self._mu(Tf)
        muN, muS = torch.cat([muv, muf[-1:]]), torch.cat([muf[:1], muv])
        uN, uS = torch.cat([u[1:, 1:-1], c[-1:]]), torch.cat([-c[:1], u[:-1, 1:-1]])
        vis = (mu[:, 1:] * (u[:, 2:] - c) + mu[:, :-1] * (u[:, :-2] - c) + muN * (uN - c) + muS * (uS - c)) / dx ** 2
        va = 0.25 * (V2[:-1, :-1] + V2[:-1, 1:] + V2[1:, :-1] + V2[1:, 1:])
        un = (c + dt * vis / self._rho(Tf)) * drag(torch.hypot(c, va), Tf)
        U = torch.cat([U2[:, 1:2].clamp(max=0), un, U2[:, -2:-1].clamp(min=0)], 1)
        # V faces away from floor and top
        Tf = 0.5 * (T[1:] + T[:-1])
        c = V2[1:-1]
        muf = self._mu(Tf)
        muE, muW = torch.cat([muv, muf[:, -1:]], 1), torch.cat([muf[:, :1], muv], 1)
        vE, vW = torch.cat([v[1:-1, 1:], c[:, -1:]], 1), torch.cat([c[:, :1], v[1:-1, :-1]], 1)
        vis = (mu[1:] * (v[2:] - c) + mu[:-1] * (v[:-2] - c) + muE * (vE - c) + muW * (vW - c)) / dx ** 2
        ua = 0.25 * (U2[:-1, :-1] + U2[:-1, 1:] + U2[1:, :-1] + U2[1:, 1:])
        vn = (c + dt * (vis / self._rho(Tf) + P["grav"] * (Tf / P["Tamb"] - 1))) * drag(torch.hypot(ua, c), Tf)
        V = torch.cat([torch.zeros_like(vn[:1]), vn, V2[-2:-1].clamp(min=0)])
        return torch.where(self.fx > 0, U, self._zero), torch.where(self.fy > 0, V, self._zero)

    # ---- pressure
    def _face_T(self, T):
        return (0.5 * (torch.cat([T[:, :1], T], 1) + torch.cat([T, T[:, -1:]], 1)),
                0.5 * (torch.cat([T[:1], T]) + torch.cat([T, T[-1:]])))

    def coefficients(self):
        P, rT = self.P, self.P["rhoAmb"] * self.P["Tamb"]
        Tx, Ty = self._face_T(self.T)
        ax, ay, h2 = self.fx * Tx / rT, self.fy * Ty / rT, self.dx ** 2
        self.lev = []
        while True:
            ny, nx = ax.shape[0], ay.shape[1]
            w, e, s, n = ax[:, :-1].clone(), ax[:, 1:].clone(), ay[:-1].clone(), ay[1:].clone()
            diag = w + e + s + n
            diag[:, 0] += w[:, 0]
            diag[:, -1] += e[:, -1]
            diag[0] -= s[0]
            diag[-1] += n[-1]
            w[:, 0], e[:, -1], s[0], n[-1] = 0, 0, 0, 0
            y, x = torch.meshgrid(torch.arange(ny, device=self.dev), torch.arange(nx, device=self.dev), indexing="ij")
            red = ((x + y) % 2 == 0)
            self.lev.append((w, e, s, n, diag, torch.where(diag > 0, 1 / diag.clamp(min=1e-300), self._zero), h2, red))
            if nx % 2 or ny % 2 or nx * ny <= 256:
                break
            ax, ay, h2 = 0.5 * (ax[::2, ::2] + ax[1::2, ::2]), 0.5 * (ay[::2, ::2] + ay[::2, 1::2]), 4 * h2
        div = (self.fx[:, 1:] * self.U[:, 1:] - self.fx[:, :-1] * self.U[:, :-1] +
               self.fy[1:] * self.V[1:] - self.fy[:-1] * self.V[:-1]) / self.dx
        opened = self.fx[:, 1:] + self.fx[:, :-1] + self.fy[1:] + self.fy[:-1] > 0
        return torch.where(opened, (div - self.SQ[..., 0]) / self.dt, self._zero)

    @staticmethod
    def _off(p, L):
        q = torch.nn.functional.pad(p, (1, 1, 1, 1))
        return L[0] * q[1:-1, :-2] + L[1] * q[1:-1, 2:] + L[2] * q[:-2, 1:-1] + L[3] * q[2:, 1:-1]

    def apply(self, p, L):
        return torch.where(L[4] > 0, (self._off(p, L) - L[4] * p) / L[6], self._zero)

    def _relax(self, p, rhs, L, red):
        new = (self._off(p, L) - rhs * L[6]) * L[5]
        return torch.where(L[7] if red else ~L[7], new, p)

    def _inverse(self):
        """The coarsest operator's inverse (the FP64 modes solve that level directly)."""
        L = self.lev[-1]
        n = L[7].numel()
        one = torch.eye(n, dtype=torch.float64, device=self.dev).view(n, *L[7].shape)
        q = torch.nn.functional.pad(one, (1, 1, 1, 1))
        A = L[0] * q[:, 1:-1, :-2] + L[1] * q[:, 1:-1, 2:] + L[2] * q[:, :-2, 1:-1] + L[3] * q[:, 2:, 1:-1] - L[4] * one
        A = A.reshape(n, n).T / L[6] - torch.diag((L[4].flatten() <= 0).double())
        return torch.linalg.inv(A) * (L[4].flatten() > 0)

    def _cycle(self, p, rhs, l=0):
        L = self.lev[l]
        if l == len(self.lev) - 1:
            if self.inv is not None:
                return (self.inv @ rhs.flatten()).view_as(rhs)
            p = torch.zeros_like(rhs)
            for _ in range(120):
                p = self._relax(self._relax(p, rhs, L, True), rhs, L, False)
            return p
        for _ in range(2):
            p = self._relax(self._relax(p, rhs, L, True), rhs, L, False)
        r = torch.where(L[4] > 0, rhs - self.apply(p, L), self._zero)
        r = 0.25 * (r[::2, ::2] + r[1::2, ::2] + r[::2, 1::2] + r[1::2, 1::2])
        c = self._cycle(torch.zeros_like(r), r, l + 1)
        if l == len(self.lev) - 3 and p.numel() <= self.w:   # the W tail
            c = self._cycle(c, r, l + 1)
        q = torch.nn.functional.pad(c[None, None], (1, 1, 1, 1), mode="replicate")[0, 0]
        x = 0.75 * q + 0.25 * torch.roll(q, 1, 1), 0.75 * q + 0.25 * torch.roll(q, -1, 1)
        fine = torch.empty_like(p)
        for a in (0, 1):
            lo, hi = 0.75 * x[a] + 0.25 * torch.roll(x[a], 1, 0), 0.75 * x[a] + 0.25 * torch.roll(x[a], -1, 0)
            fine[::2, a::2], fine[1::2, a::2] = lo[1:-1, 1:-1], hi[1:-1, 1:-1]
        p = p + torch.where(L[4] > 0, fine, self._zero)
        for _ in range(2):
            p = self._relax(self._relax(p, rhs, L, False), rhs, L, True)
        return p

    def solve(self, rhs, mode, tol):
        L, norm = self.lev[0], rhs.norm()
        if mode == "fixed":
            self.p = self._cycle(self.p, rhs)
        elif mode == "tol":
            for _ in range(50):
                self.p = self._cycle(self.p, rhs)
                r = torch.where(L[4] > 0, rhs - self.apply(self.p, L), self._zero)
                if r.norm() <= tol * norm:
                    break
        else:   # conjugate gradients with a V-cycle each; the direction by the change of the residual
            p = self.p
            r = torch.where(L[4] > 0, rhs - self.apply(p, L), self._zero)
            d, old, rz = None, None, None
            self.inv = self._inverse()
            for _ in range(300):
                if r.norm() <= tol * norm:
                    break
                z = self._cycle(torch.zeros_like(r), r)
                beta = 0.0 if d is None else float((z * (r - old)).sum() / rz)
                d = z if d is None else z + beta * d
                q, rz, old = self.apply(d, L), (r * z).sum(), r
                a = rz / (d * q).sum()
                p, r = p + a * d, r - a * q
            self.p = p

    def _project(self):
        rT, p, dt, dx = self.P["rhoAmb"] * self.P["Tamb"], self.p, self.dt, self.dx
        Tx, Ty = self._face_T(self.T)
        gx = torch.cat([p, -p[:, -1:]], 1) - torch.cat([-p[:, :1], p], 1)
        gy = torch.cat([p, -p[-1:]]) - torch.cat([p[:1], p])
        self.U = torch.where(self.fx > 0, self.U - dt * Tx / rT * gx / dx, self._zero)
        self.V = torch.where(self.fy > 0, self.V - dt * Ty / rT * gy / dx, self._zero)

    def step(self, mode, tol):
        T2, Y2, U2, V2 = self._advect()
        T, Y = self._sources(*self._diffuse(T2, Y2), T2)
        self.T, self.Y = T, Y
        self.U, self.V = self._forces(T, U2, V2)
        self.solve(self.coefficients(), mode, tol)
        self._project()
        if self.cfl > 0:
            m = max(float(self.U.abs().max()), float(self.V.abs().max()))
            self.dt = min(self.cap, self.cfl * self.dx / m) if m > 0 else self.cap

    # ---- radiation: rays from each wood face and floor probe, marched in steps of about a cell
    def radiation(self, nray, frame):
        P, nx, ny, dx = self.P, self.nx, self.ny, self.dx
        nf, nt, pi = 4 * self.np_, 4 * self.np_ + 64, math.pi
        tgt = torch.arange(nt, device=self.dev)[:, None].double()
        li = torch.arange(nray, device=self.dev)[None, :].double()
        pc = self.pieces[(tgt[:nf].long() // 4).squeeze(1)].view(nf, 20)
        f = (tgt[:nf].long() % 4).squeeze(1)
        n0 = torch.tensor([[1.0, 0], [0, 1], [-1, 0], [0, -1]], dtype=torch.float64, device=self.dev)[f]
        c, s = torch.cos(pc[:, 2]), torch.sin(pc[:, 2])
        nrx, nry = (c * n0[:, 0] - s * n0[:, 1])[:, None], (s * n0[:, 0] + c * n0[:, 1])[:, None]
        frac = lambda x: x - torch.floor(x)   # noqa: E731
        u = (frac(li * 0.618034 + frame * 0.1234) - 0.5) * 1.6 * pc[:, 3:4]
        ox, oy = pc[:, 0:1] + nrx * (pc[:, 3:4] + 1e-4) - nry * u, pc[:, 1:2] + nry * (pc[:, 3:4] + 1e-4) + nrx * u
        fl = (torch.arange(64, device=self.dev).double()[:, None] + 0.5) / 64 * nx * dx
        one = torch.ones(64, nray, dtype=torch.float64, device=self.dev)
        ox, oy = torch.cat([ox, fl * one]), torch.cat([oy, 1e-4 * one])
        base = torch.cat([torch.atan2(nry, nrx), torch.full((64, 1), pi / 2, dtype=torch.float64, device=self.dev)])
        a = ((li + frac(frame * 0.7548777 + tgt * 0.5698403)) / nray - 0.5) * pi
        dxr, dyr = torch.cos(base + a), torch.sin(base + a)
        J, Jv = torch.zeros_like(ox), torch.zeros_like(ox)
        wall = torch.full_like(ox, P["Tamb"])
        live = torch.ones_like(ox, dtype=torch.bool)
        rho = self._rho(self.T)
        fv = rho * self.Y[..., 3] / P["sootDensity"]
        kap = P["kappaSootC"] * fv * self.T + P["kappaGas"] * self.Y[..., 2]
        g1 = kap * P["sigma"] * (self.T ** 4 - P["Tamb"] ** 4) / pi
        l = 580e-9
        x = 1.438777e-2 / (l * self.T)
        pl = torch.where(x > 80, self._zero, 1.191042e-16 / l ** 5 / torch.expm1(x.clamp(max=80)) * 1e-9)
        g2 = 6.3 * fv / l * pl
        for bounce in (0, 1):
            hit, hT = torch.full_like(ox, 1e9), torch.zeros_like(ox)
            for n in range(self.np_):
                q = self.pieces[n]
                c, s = torch.cos(q[2]), torch.sin(q[2])
                lx, ly = c * (ox - q[0]) + s * (oy - q[1]), -s * (ox - q[0]) + c * (oy - q[1])
                kx, ky = c * dxr + s * dyr, -s * dxr + c * dyr
                ix, iy = (1 / torch.where(k.abs() < 1e-9, torch.full_like(k, 1e-9), k) for k in (kx, ky))
                t1x, t2x, t1y, t2y = (-q[3] - lx) * ix, (q[3] - lx) * ix, (-q[3] - ly) * iy, (q[3] - ly) * iy
                mx, my = torch.minimum(t1x, t2x), torch.minimum(t1y, t2y)
                tn, tf = torch.maximum(mx, my), torch.minimum(torch.maximum(t1x, t2x), torch.maximum(t1y, t2y))
                face = torch.where(mx > my, torch.where(kx < 0, 0, 2), torch.where(ky < 0, 1, 3))
                near = (tf >= 0) & (tn <= tf) & (tn >= 1e-5) & (tn < hit)
                hit, hT = torch.where(near, tn, hit), torch.where(near, q[8:12][face], hT)
            far = torch.full_like(ox, 1e9)
            floor = torch.where(dyr < -1e-6, -oy / dyr, far)
            W, H = nx * dx, ny * dx
            tx = torch.where(dxr > 1e-6, (W - ox) / dxr, torch.where(dxr < -1e-6, -ox / dxr, far))
            ty = torch.where(dyr > 1e-6, (H - oy) / dyr, far)
            out = torch.minimum(torch.minimum(tx, ty), torch.minimum(hit, floor))
            ns = torch.ceil(out / dx)
            for m in range(int(ns[live].max()) if bool(live.any()) else 0):
                t = (m + 0.5) * out / ns
                i, j = ((ox + dxr * t) / dx).trunc().long(), ((oy + dyr * t) / dx).trunc().long()
                ok = live & (m < ns) & (i >= 0) & (j >= 0) & (i < nx) & (j < ny)
                k = (j.clamp(0, ny - 1), i.clamp(0, nx - 1))
                J += torch.where(ok, g1[k] * out / ns, self._zero)
                Jv += torch.where(ok, g2[k] * out / ns, self._zero)
            struck = live & (hit < floor) & (hit < 1e8)
            wall = torch.where(struck, hT, wall)
            live = live & ~struck & (floor < 1e8)
            ox, oy = ox + dxr * floor, oy + dyr * floor + 1e-5
            dyr = -dyr
        wgt = pi / nray * torch.cos(a)
        rad = torch.zeros(320, 4, dtype=torch.float64, device=self.dev)
        rad[:nt, 0] = (wgt * (0.5 * P["sigma"] * wall ** 4 + 2 * J)).sum(1)
        rad[:nt, 1] = (wgt * 2 * Jv).sum(1)
        return rad.flatten()

    def sums(self):
        gas = ~((self.sdf < 0) & (self.sid >= 0))
        rho = self._rho(self.T)
        m = rho * self.dx ** 2 * gas
        return torch.stack([m.sum(), (m * self.P["cp"] * self.T).sum(), *((m * self.Y[..., k]).sum() for k in range(4)),
                            (self.SQ[..., 1] * gas).sum() * self.dx ** 2, (self.T * gas).max()])


def _inferno(t):
    t = t.clamp(0, 1).unsqueeze(-1)
    c = torch.tensor([[0.0002, 0.0016, -0.0194], [0.1065, 0.5640, 3.9327], [11.6024, -3.9728, -15.9423],
                      [-41.7040, 17.4364, 44.3541], [77.1629, -33.4023, -81.8073], [-71.3194, 32.6261, 73.2095],
                      [25.1311, -12.2426, -23.0703]], dtype=torch.float64, device=t.device)
    v = c[6]
    for k in range(5, -1, -1):
        v = c[k] + t * v
    return v.clamp(0, 1)


def _exact_view(x, case, zoom, cam):
    """The scalar views (reaction, oxygen, fuel, velocity, soot) with the pieces' outlines."""
    W, H, view, ground = case["W"], case["H"], VIEWS[case["view"]], 0.03
    py, px = torch.meshgrid(x._axis(H, 0.5), x._axis(W, 0.5), indexing="ij")
    wx = px / W * (x.nx * x.dx) / zoom + cam[0]
    wy = (1 - py / H) * (x.ny * x.dx + ground) / zoom + cam[1]
    gx, gy = wx / x.dx, wy / x.dx
    Y = x._sample(x.Y, "C", gx, gy, x.amb)
    vec = lambda *v: torch.tensor(v, dtype=torch.float64, device=x.dev)   # noqa: E731
    if view == 2:
        q = torch.nn.functional.pad(x.SQ[..., 1], (1, 1, 1, 1))
        i, j = torch.floor(gx - 0.5), torch.floor(gy - 0.5)
        at = lambda a, b: q[(j.long() + 1 + b).clamp(0, x.ny + 1), (i.long() + 1 + a).clamp(0, x.nx + 1)]   # noqa: E731
        tx, ty = gx - 0.5 - i, gy - 0.5 - j
        col = _inferno((((at(0, 0) * (1 - tx) + at(1, 0) * tx) * (1 - ty) +
                         (at(0, 1) * (1 - tx) + at(1, 1) * tx) * ty) / 2.0e7) ** 0.5)
    elif view == 3:
        t = (Y[..., 1] / x.P["YOamb"]).unsqueeze(-1)
        col = vec(0.02, 0.02, 0.08) * (1 - t) + vec(0.35, 0.85, 1.0) * t
    elif view == 4:
        col = _inferno((Y[..., 0] / 0.4) ** 0.5)
    elif view == 5:
        i, j = gx.trunc().long().clamp(0, x.nx - 1), gy.trunc().long().clamp(0, x.ny - 1)
        u, v = 0.5 * (x.U[j, i] + x.U[j, i + 1]), 0.5 * (x.V[j, i] + x.V[j + 1, i])
        col = _inferno(torch.hypot(u, v) / 3.0)
    else:
        Ta = vec(x.P["Tamb"])[0]
        col = _inferno((x._rho(x._sample(x.T, "C", gx, gy, Ta)) * Y[..., 3] / x.P["sootDensity"] / 1e-6) ** 0.5)
    col = torch.where((wy < 0).unsqueeze(-1), vec(0.08, 0.08, 0.08), col)
    for n in range(x.np_):
        q = x.pieces[n]
        c, s = torch.cos(q[2]), torch.sin(q[2])
        lx, ly = c * (wx - q[0]) + s * (wy - q[1]), -s * (wx - q[0]) + c * (wy - q[1])
        e = q[3] - torch.maximum(lx.abs(), ly.abs())
        t = (e / 0.0012).clamp(0, 1)
        mix = ((1 - t * t * (3 - 2 * t)) * 0.6).unsqueeze(-1)
        body = vec(0.35, 0.3, 0.25) * (1 - mix) + 0.85 * mix
        col = torch.where((e >= 0).unsqueeze(-1), body, col)
    return torch.cat([col, torch.ones_like(col[..., :1])], -1)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        return None   # dozens of scenes solved to convergence: minutes in 64 bits
    width = cb.SCENE_WIDTH if kind in ("frame", "render") else case["width"]
    x = _Exact(_scene(case["nx"], case["ny"], width, case["pieces"], seed, case.get("dt", 0.002)),
               case.get("dt", 0.002), case.get("cfl", 0.0), case.get("w", 0))
    if kind == "steps":
        for _ in range(case["steps"]):
            x.step(case["mode"], case["tol"])
        return {"T": x.T.flatten(), "Y": x.Y.flatten(), "U": x.U.flatten(), "V": x.V.flatten()}
    if kind == "frame":
        for _ in range(case["steps"]):
            x.step("fixed", 0.0)
        # faceW and tmax are whole numbers; the picture's wood and ground are shaded with a hash of the sine of
        # large numbers, whose 64-bit value is another noise
        return {"heat": x.heat, "char": x.char, "total": x.total, "tmax": None, "rad": x.radiation(64, 0),
                "faceW": None, "img": None}
    if kind == "render":
        if case["view"] in ("photo", "temperature"):
            return None   # the hash noise above; the wood's inner profile
        x.SQ = torch.as_tensor(np.asarray(_rates(case["nx"], case["ny"], seed), np.float64), device=x.dev)
        zoom = case["zoom"]
        return _exact_view(x, case, zoom, (0.0, -0.03) if zoom == 1.0 else (0.2, 0.02))
    if kind == "radiation":
        return x.radiation(case["nray"], 1)
    x.SQ = torch.as_tensor(np.asarray(_rates(case["nx"], case["ny"], seed), np.float64), device=x.dev)
    rhs = x.coefficients()
    p = torch.as_tensor(_pressure(case["nx"], case["ny"], seed), device=x.dev)
    r = torch.where(x.lev[0][4] > 0, rhs - x.apply(p, x.lev[0]), x._zero)
    return {"residual": float(r.norm() / rhs.norm()), "sums": x.sums()}
