"""Performance cases: what a user of the framework has it do, through its public entry points.

Kinds of pass (a case's `kind`):

  live   one frame of an interactive fire: a simulation step, then the volume render of the new
         state into a device image (FluidSimulation.step, render_device).
  bake   `steps` simulation steps, then the state read back for export (FluidSimulation.step,
         field: velocity and scalars).
  batch  `steps` steps of many independent simulations through one SimulationBatch, then every
         simulation's scalars read back.
  serve  `steps` rounds of one request per session to a FireServer, drained, then every
         session's scalars read back.
  mesh   one frame's moving mesh: its collider occupancy (mesh.voxelize) and the emission
         records of its surface samples (mesh.splat).

Scenes and grids are those of the repository's scenes, benchmark and tests. A simulation is grown
`grow` steps in prepare, to where its brick count no longer changes much (its natural size or its
voxel budget), so a pass costs the same however often it is repeated; after that it plays a loop
of CLIP prepared frames. Every simulation's scene derives from the seed.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

_PACKAGE = str(Path.cwd() / "threejs-fire-pro_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

from firepro import abi, mesh, render, scenes  # noqa: E402
from firepro.engine import FIXED_DT, FireServer, FluidSimulation, SimulationBatch, reserved_tiles  # noqa: E402

CLIP = 48  # prepared frames a simulation plays in a loop
VOXEL = 0.025

# Camera (eye, target) per scene, near enough that the fire fills a good part of the view.
CAMERAS = {
    "plume": ((0.0, 0.8, 2.2), (0.0, 0.6, 0.0)),
    "large": ((0.0, 1.2, 4.0), (0.0, 1.0, 0.0)),
    "force": ((0.0, 1.0, 3.0), (0.0, 0.5, 0.0)),
    "jet": ((-0.5, 1.2, 3.2), (-0.2, 0.6, 0.0)),
    "member": ((0.0, 0.9, 2.6), (0.0, 0.6, 0.0)),
}
# Computing 8^3 bricks the scenes hold after a growth of so many steps (measured, seed 1); bricks
# of side B hold about 1.35 (B / 8)^3 fewer. Used by `work` only.
GROWTH = {
    "plume": ((0, 216), (60, 216), (120, 244), (180, 368), (240, 479), (400, 800)),
    "large": ((0, 216), (30, 752), (60, 765), (120, 2373), (180, 4300), (400, 3800)),
    "force": ((0, 71), (30, 147), (60, 331), (120, 1066), (180, 1827), (400, 1900)),
    "jet": ((0, 16), (30, 95), (60, 268), (120, 804), (180, 1518), (400, 1400)),
    "member": ((0, 100), (60, 150), (120, 300), (400, 600)),
}


def _case(name, kind, scene, **kw):
    case = {
        "name": name, "kind": kind, "scene": scene,
        # grid: field cells a brick side, velocity and smoke divisors, storage, limiter, voxels
        "brick": 8, "vdiv": 1, "sdiv": 1, "mixed": False, "maccormack": True, "budget": 1600000,
        # flow: steps grown in prepare, steps a pass, V-cycles (0: the reference's single one;
        # else flexible CG around a red-black V-cycle), simulations of a batch or a server
        "grow": 200, "steps": 1, "vcycles": 0, "sims": 1,
        # image: pixels, half-resolution slices, ray steps, shadow samples, filter, light texel
        "width": 0, "height": 0, "half": 1, "rays": 256, "shadow": 32, "filter": 2, "light": 4,
        # mesh: icosphere subdivisions and radius
        "subdiv": 0, "radius": 0.0,
    }
    case.update(kw)
    return case


def listed():
    return [
        # A small ember effect, one of many in a scene: 90 bricks, where a step is launches and
        # latency. Its state is exported at a tenth of a second.
        _case("member_bake", "bake", "member", budget=90 * 512, grow=30, steps=8),
        # The benchmark's and tests' large scene at a voxel budget it has reached, exported four
        # times a simulated second: the throughput of the default solve.
        _case("large_bake", "bake", "large", steps=16),
        # Every force and collider kind in FP_PRECISION_MIXED on a small budget of an odd number
        # of bricks.
        _case("force_mixed_bake", "bake", "force", mixed=True, budget=1021 * 512, grow=160, steps=16),
        # The accurate solve of the benchmark (flexible CG, red-black, topology each step), for
        # renders that must hold volume; exported often.
        _case("accurate_bake", "bake", "large", budget=1200000, vcycles=5, steps=8),
        # Many independent effects stepped by one launch: the benchmark's batched form.
        _case("batch_bake", "batch", "member", sims=24, budget=0, grow=60, steps=12),
        # A serving host's tick: every session's next request, mixed precision.
        _case("serve_ticks", "serve", "member", sims=10, mixed=True, budget=0, grow=60, steps=6),
        # The smallest interactive frame: the plume in a small preview.
        _case("plume_preview", "live", "plume", budget=2 ** 19, grow=400, width=320, height=180, rays=128, shadow=16),
        # The reference's default grid (16^3 bricks, velocity divisor 2, smoke divisor 2, 8M
        # voxels) with its default render settings.
        _case("default_live", "live", "large", brick=16, vdiv=2, sdiv=2, budget=8000000, grow=240, width=960, height=540),
        # The benchmark's stress form: a 25 m/s jet with its long back-traces, half resolution.
        _case("jet_live", "live", "jet", budget=2 ** 22, grow=300, width=960, height=540, rays=128, shadow=16),
        # Colliders and forces at an odd size, full resolution, quadratic filter, finer lighting.
        _case("force_odd_live", "live", "force", budget=700 * 512, grow=160, width=641, height=361, half=0, rays=160,
              shadow=24, filter=1, light=2),
        # The largest frame: the large scene at its natural size in full HD.
        _case("large_hd_live", "live", "large", budget=8000000, grow=240, width=1920, height=1080),
        # A moving mesh emitter and collider, rebuilt each frame.
        _case("mesh_frame", "mesh", "mesh", subdiv=3, radius=0.31),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case of the listed ones' ranges."""
    kind = rng.choice(("live", "live", "live", "bake", "bake", "bake", "batch", "serve", "mesh"))
    if kind == "mesh":
        return _unnamed(_case("", kind, "mesh", subdiv=rng.randint(2, 4), radius=round(_log(rng, 0.08, 0.5), 4)))
    if kind in ("batch", "serve"):
        return _unnamed(_case("", kind, "member", sims=rng.randint(2, 24 if kind == "batch" else 10), budget=0,
                              mixed=rng.random() < 0.5, grow=rng.randint(5, 60),
                              steps=rng.randint(1, 12 if kind == "batch" else 6)))
    scene = rng.choice(("plume", "large", "force", "jet", "member"))
    brick, vdiv, sdiv = rng.choice(((8, 1, 1), (8, 1, 1), (8, 1, 2), (8, 2, 1), (16, 1, 1), (16, 2, 2), (16, 2, 2),
                                    (16, 2, 4), (32, 4, 4)))
    cells = brick ** 3
    budget = int(max(_log(rng, 4e4, 2e6), 12 * cells))
    case = _case("", kind, scene, brick=brick, vdiv=vdiv, sdiv=sdiv, mixed=rng.random() < 0.3,
                 maccormack=rng.random() < 0.85, budget=budget, grow=rng.randint(10, 240))
    if kind == "bake":
        case["vcycles"] = rng.choice((0, 0, 0, 2, 4, 5))
        case["steps"] = rng.randint(1, 8 if case["vcycles"] or brick == 32 else 16)
    else:
        case["width"] = int(_log(rng, 160, 1280))
        case["height"] = int(case["width"] * rng.uniform(0.5, 0.8))
        case["half"] = rng.randint(0, 1)
        case["rays"] = rng.randint(64, 256)
        case["shadow"] = rng.randint(8, 32)
        case["filter"] = rng.choice((0, 1, 2, 2))
        case["light"] = rng.choice((2, 4, 4))
    return _unnamed(case)


def _unnamed(case):
    del case["name"]
    return case


def _scene(case, seed, index=0):
    kind = case["scene"]
    if kind == "plume":
        sc = scenes.SinglePlume(seed)
    elif kind == "large":
        sc = scenes.LargeScene(seed)
    elif kind == "force":
        sc = scenes.ForceScene(seed)
    elif kind == "jet":
        sc = scenes.StressScene(seed)
    else:
        sc = scenes.MemberScene(seed, index, 16, 512)
        sc.bricks = scenes.MemberScene(1, index, 16, 512).bricks  # budgets alike for every seed
    sc.voxel_size = VOXEL
    sc.brick_size, sc.velocity_divisor = case["brick"], case["vdiv"]
    return sc


def _frame(case, sc, step):
    """The scene's frame. The force scene is the same for every seed but for its noise: its
    emitters' rates and the forces vary here."""
    fd = sc.frame(step)
    if case["scene"] == "force":
        for k in range(fd.frame.source_count):
            src = fd.frame.sources[k]
            gain = 0.8 + 0.4 * scenes.value_noise_1d(0.37 * k + 0.5, sc.seed) ** 2
            src.heat_rate, src.smoke_rate = src.heat_rate * gain, src.smoke_rate * gain
        for k in range(fd.frame.force_count):
            fd.frame.forces[k].strength *= 1.0 + 0.2 * scenes.value_noise_1d(0.61 * k + 0.5, sc.seed + 1)
    return fd


def _grid(case, sc, budget):
    grid = sc.grid(budget=float(budget), maccormack=case["maccormack"],
                   precision=abi.FP_PRECISION_MIXED if case["mixed"] else abi.FP_PRECISION_FP32)
    grid.smoke_divisor = case["sdiv"]
    return grid


def _simulation(case, seed):
    sc = _scene(case, seed)
    sim = FluidSimulation(_grid(case, sc, case["budget"]))
    sim.set_runtime(0.05, float(case["budget"]), True)
    for s in range(case["grow"]):
        sim.step(_frame(case, sc, s).frame)
    if case["vcycles"]:
        sim.set_schedule(abi.schedule(abi.FP_SMOOTHER_REDBLACK, 0, 2, 2, 8, abi.FP_KRYLOV_FCG, 1))
        sim.set_solver(case["vcycles"], 0.0)
    sim.synchronize()
    return sim, [_frame(case, sc, case["grow"] + k) for k in range(CLIP)]


def _mesh_inputs(case, seed):
    """A dented icosphere (a collider of the same box for every seed), its placement, and its
    emitter's placed samples, weights, area and rates."""
    rng = np.random.RandomState(seed & 0x7FFFFFFF)
    pos, idx = mesh.icosphere(case["subdiv"], case["radius"])
    samples, weights, area = mesh.surface_samples(pos, idx, VOXEL)
    dent = 1.0 - 0.15 * rng.uniform(0.0, 1.0, len(pos))
    for axis in range(3):
        dent[[pos[:, axis].argmin(), pos[:, axis].argmax()]] = 1.0
    pos = (pos * dent[:, None]).astype(np.float32)
    ax, ay = 0.3, 0.7
    cx, sx, cy, sy = math.cos(ax), math.sin(ax), math.cos(ay), math.sin(ay)
    world = np.eye(4)
    world[:3, :3] = (np.array([[cy, 0, sy], [0, 1, 0], [-sy, 0, cy]]) @ np.array([[1, 0, 0], [0, cx, -sx], [0, sx, cx]]) @
                     np.diag((1.2, 0.8, 1.1)))
    world[:3, 3] = (-0.21, 0.83, 0.11)
    r = rng.uniform(0.5, 1.5, 8)
    rates = dict(flame=0.6 * r[0], heat=2.0 * r[1], smoke=1.2 * r[2], fuel=0.5 * r[3],
                 velocity=(r[4] - 1.0, 1.5 * r[5], r[6] - 1.0), response=4.0 * r[7])
    return pos, idx, world, mesh.place(samples, world), weights, area, rates


def prepare(case, seed):
    kind = case["kind"]
    if kind == "mesh":
        pos, idx, world, samples, weights, area, rates = _mesh_inputs(case, seed)
        return {"kind": kind, "pos": pos, "idx": idx, "world": world,
                "emitter": mesh.MeshEmitter(samples, weights, area, **rates)}
    if kind in ("batch", "serve"):
        members = [_scene(case, seed, k) for k in range(case["sims"])]
        frames = [[m.frame(case["grow"] + k) for m in members] for k in range(CLIP)]
        if kind == "batch":
            host = SimulationBatch(case["brick"])
            ids = []
            for m in members:
                grid = _grid(case, m, m.budget)
                i = host.add(grid)
                host.set_runtime(i, 0.05, m.budget, True)
                host.reserve_tiles(i, reserved_tiles(grid))
                ids.append(i)
            for s in range(case["grow"]):
                held = [m.frame(s) for m in members]
                host.step([(i, fd.frame, FIXED_DT) for i, fd in zip(ids, held)])
            host.synchronize()
        else:
            host = FireServer(64 << 30, max_sessions=64, brick_size=case["brick"])
            ids = [host.open(_grid(case, m, m.budget)) for m in members]
            for s in range(case["grow"]):
                held = [m.frame(s) for m in members]
                for i, fd in zip(ids, held):
                    host.submit(i, fd.frame)
            host.drain()
            while host.poll():
                pass
        return {"kind": kind, "host": host, "ids": ids, "frames": frames, "steps": case["steps"], "next": 0}
    sim, frames = _simulation(case, seed)
    state = {"kind": kind, "sim": sim, "frames": frames, "steps": case["steps"], "next": 0}
    if kind == "live":
        eye, target = CAMERAS[case["scene"]]
        cams = []
        for k in range(CLIP):
            cam = render.look_at(eye, target, case["width"], case["height"], time=(case["grow"] + k) / 60.0)
            cam.half_resolution = case["half"]
            cams.append(cam)
        state["cameras"] = cams
        state["settings"] = render.default_settings(case["filter"], case["rays"], case["light"], case["shadow"])
        state["image"] = torch.zeros((case["height"], case["width"], 4), dtype=torch.float32, device="cuda")
        state["stream"] = torch.cuda.ExternalStream(sim.stream())
    return state


def run(state):
    kind = state["kind"]
    if kind == "mesh":
        collider, words = mesh.voxelize(state["pos"], state["idx"], state["world"], VOXEL)
        records = mesh.splat([state["emitter"]], VOXEL)
        rows = np.frombuffer((abi.fp_mesh_source * len(records))(*records), np.float32).reshape(len(records), -1)
        return {"lo": np.array(collider.lo[:], np.int32), "dims": np.array(collider.dims[:], np.int32),
                "words": words.view(np.int32), "cells": rows[:, :4].view(np.int32), "rates": rows[:, 4:]}
    if kind == "live":
        sim, k = state["sim"], state["next"]
        state["next"] = (k + 1) % CLIP
        sim.step(state["frames"][k].frame)
        sim.render_device(state["cameras"][k], state["settings"], state["image"].data_ptr())
        torch.cuda.current_stream().wait_stream(state["stream"])
        return state["image"]
    for _ in range(state["steps"]):
        k = state["next"]
        state["next"] = (k + 1) % CLIP
        frames = state["frames"][k]
        if kind == "bake":
            state["sim"].step(frames.frame)
        elif kind == "batch":
            state["host"].step([(i, fd.frame, FIXED_DT) for i, fd in zip(state["ids"], frames)])
        else:
            for i, fd in zip(state["ids"], frames):
                state["host"].submit(i, fd.frame)
    if kind == "bake":
        sim = state["sim"]
        return {"velocity": sim.field(abi.FP_FIELD_VELOCITY), "scalars": sim.field(abi.FP_FIELD_SCALARS)}
    host = state["host"]
    if kind == "serve":
        host.drain()
        while host.poll():
            pass
    return [host.field(i, abi.FP_FIELD_SCALARS) for i in state["ids"]]


def _bricks(case):
    """About how many bricks compute (for `work`)."""
    table, g = GROWTH[case["scene"]], case["grow"]
    at = [float(v) for v in np.interp([g], [t for t, _ in table], [v for _, v in table])][0]
    scale = (case["brick"] / 8.0) ** 3
    if case["kind"] in ("batch", "serve"):
        return case["sims"] * 110.0  # budgets log-uniform in 16..512 bricks
    return max(1.0, min(case["budget"] / case["brick"] ** 3, at * (1.35 if scale > 1 else 1.0) / scale))


def work(case):
    if case["kind"] == "mesh":
        triangles, r = 20 * 4 ** case["subdiv"], case["radius"] / VOXEL
        cells = (2 * r + 3) ** 3
        samples = min(8192.0, max(256.0, 4 * math.pi * r * r * 8))
        return {"bytes": triangles * 24 + cells / 8 + samples * 32 + 4 * math.pi * r * r * 3 * 48,
                "flops": triangles * 200 + samples * 8 * 20}
    voxels = _bricks(case) * case["brick"] ** 3
    # A step: every field a kernel needs read once and written once (68 predict, 36 correct, 64
    # evolve, 28 curl, 56 forces, 24 divergence, 61 multigrid, 28 project; FP32 at one lattice):
    # 96 bytes a field voxel, the rest a velocity cell.
    per = (72.0 if case["mixed"] else 96.0) + (269.0 + 70.0 * max(0, case["vcycles"] - 1)) / case["vdiv"] ** 3
    step = {"bytes": voxels * per, "flops": voxels * (300.0 + 400.0 / case["vdiv"] ** 3)}
    if case["kind"] != "live":
        fields = 4 if case["kind"] in ("batch", "serve") else 4 + 3 / case["vdiv"] ** 3
        return {"bytes": case["steps"] * step["bytes"] + voxels * 4 * fields, "flops": case["steps"] * step["flops"]}
    # A render: the scalars read, the render field and the lighting lattice written and read, the
    # image written; a shaded sample of 4^3 (cubic) cells on a quarter of the rays' steps.
    pixels = case["width"] * case["height"]
    rays = pixels * (0.25 if case["half"] else 1.0)
    taps = 8.0 if case["filter"] == 0 else 64.0
    texels = voxels / case["light"] ** 3
    return {"bytes": step["bytes"] + voxels * 16 * 3 + texels * 32 + pixels * 16 + (rays * 128 if case["half"] else 0),
            "flops": step["flops"] + voxels * 60 + texels * (case["shadow"] + 36) * 80 +
            rays * case["rays"] * 0.25 * (taps * 8 + 150)}


def exact(case, seed):
    """The mesh emission records in 64 bits (MeshSourceRasterizer: every sample splats its share of
    the surface over the eight cells around it, coverage capped at one scales the rates). The
    occupancy is bits, and a grown simulation's fields and images have no value to be had without
    the whole solver (hundreds of steps of a branching flow): minutes in numpy."""
    if case["kind"] != "mesh":
        return None
    _, _, _, samples, weights, area, rates = _mesh_inputs(case, seed)
    q = samples / VOXEL - 0.5
    base = np.floor(q)
    frac = q - base
    share = weights * area / (VOXEL * VOXEL)
    cover = {}
    for k in range(8):
        d = np.array([k & 1, (k >> 1) & 1, k >> 2])
        w = np.prod(np.where(d == 1, frac, 1.0 - frac), axis=1) * share
        for cell, v in zip(map(tuple, (base + d).astype(np.int64)), w):
            if v > 0.0:
                cover[cell] = cover.get(cell, 0.0) + v
    rows = []
    v = np.array(rates["velocity"])
    for cell in sorted(cover):
        c = min(1.0, cover[cell])
        rows.append(np.concatenate([[rates["flame"] * c, rates["heat"] * c, rates["smoke"] * c, rates["fuel"] * c],
                                    v * (rates["response"] * c), [rates["response"] * c]]))
    return {"lo": None, "dims": None, "words": None, "cells": None, "rates": np.array(rows)}
