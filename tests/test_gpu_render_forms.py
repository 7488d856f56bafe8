"""The render's forms by what the device has room for and by the image's size, against the oracle.

The tolerance is test_gpu_render's: relative L2 2e-3 between the FP32 image and the oracle's FP64
one of the same state.
"""
import ctypes as C
import json
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from firepro import abi, render, scenes
from firepro.engine import FluidSimulation
import parity

pytestmark = pytest.mark.gpu

RENDER_TOL = 2e-3


class DiagonalScene(scenes.Scene):
    """A small fire in every tile along a diagonal: the tiles touch, so one box spans them all,
    `count` tiles (four bricks each) a side."""

    name = "diagonal"

    def __init__(self, count, seed=1):
        self.count = count
        self.settings = scenes.settings(buoyancy=1.0, vorticity=0.0, seed=seed)
        self.comb = scenes.combustion()

    def frame(self, step):
        tile = 4 * 8 * self.voxel_size
        srcs = [scenes.source(1 + k, "sphere", ((k + 0.4) * tile,) * 3, (0.12, 0.12, 0.12), flame=0.8, heat=3.0,
                              smoke=8.0, velocity=(0.0, 1.0, 0.0), response=30.0) for k in range(self.count)]
        return scenes.make_frame(self.settings, self.comb, True, srcs)


def images(scene, steps, cameras, settings, budget):
    """Each camera's image of the last step's state, the simulation's and the oracle's."""
    out = []

    def after(gpu, orc):
        out.extend((gpu.render(cam, settings), orc.render(cam, settings)) for cam in cameras)

    parity.lockstep(scene, steps, lambda g: FluidSimulation(g), budget=budget, after=after)
    return out


def check(gpu, orc):
    assert np.isfinite(gpu).all()
    assert orc[..., 3].max() > 0.05, "something should be visible"
    assert parity.rel_l2(gpu, orc.astype(np.float64)) <= RENDER_TOL


def test_box_too_large_for_tables():
    """A box of more than 2^24 bricks (66 tiles a side: 258^3 at the least) renders through the tile
    hash, at both resolutions."""
    cams = []
    for half in (0, 1):
        cam = render.look_at((2.6, 1.3, -1.2), (1.1, 1.1, 1.1), 97, 65, time=0.5)
        cam.half_resolution = half
        cams.append(cam)
    st = render.default_settings(ray_steps=1024, shadow_samples=8)
    for gpu, orc in images(DiagonalScene(66), 3, cams, st, 2 ** 22):
        check(gpu, orc)


# Rays: 15,931 (16 lanes a ray), 16,037 and 35,649 (8), 36,045 and 99,855 (4), 100,233 and 402,003 (2):
# odd and either side of each line, so that every form has tiles partly outside.
SIZES = [(179, 89), (203, 79), (233, 153), (267, 135), (317, 315), (333, 301), (709, 567)]


@pytest.mark.parametrize("width,height", SIZES)
def test_lanes_a_ray(width, height):
    """Each number of lanes a ray: at full resolution, and in the half-resolution slices (of an odd
    image), with a scene's depth through the flames, for which all slices are written and read, and
    without."""
    cams, depths = [], []
    for half, depth in ((0, False), (0, True), (1, False), (1, True)):
        w, h = (2 * width - 1, 2 * height - 1) if half else (width, height)
        cam = render.look_at((1.4, 1.0, 2.0), (0.0, 0.45, 0.0), w, h, time=0.5)
        cam.half_resolution = half
        if depth:  # clip z of a plane 2.15 to 2.55 m from the eye, left to right; a band with nothing
            near, far = 0.05, 50.0
            d = 2.35 + 0.4 * ((np.arange(w) + 0.5) / w - 0.5) + np.zeros((h, 1))
            z = np.ascontiguousarray((far * (d - near) / (d * (far - near))).astype(np.float32))
            z[:, : w // 8] = 1.0
            depths.append(z)  # the camera points into it
            cam.scene_depth = z.ctypes.data_as(C.POINTER(C.c_float))
        cams.append(cam)
    st = render.default_settings(ray_steps=40, shadow_samples=4)
    for gpu, orc in images(scenes.ForceScene(), 12, cams, st, 2 ** 20):
        check(gpu, orc)


@pytest.mark.parametrize("width,height", [(112, 96), (160, 160), (224, 208), (304, 272), (480, 400), (720, 560)])
def test_opacity_below_zero(width, height):
    """A negative flame opacity raises the transmittance along a ray: whatever number of lanes shares
    it, the steps compose as one after the other."""
    cam = render.look_at((1.4, 1.0, 2.0), (0.0, 0.45, 0.0), width, height, time=0.5)
    st = render.default_settings(ray_steps=64, shadow_samples=8)
    st.flame_opacity = -1.5
    (gpu, orc), = images(scenes.ForceScene(), 10, [cam], st, 2 ** 20)
    assert np.isfinite(gpu).all() and orc[..., 3].min() < -0.05, "some ray should gain"
    assert parity.rel_l2(gpu, orc.astype(np.float64)) <= RENDER_TOL


class SparseScene(scenes.Scene):
    """`side`^3 puffs of smoke, each within a brick of its own, three bricks apart: every brick has its
    seven apron bricks, more than the render keeps room for (two a slot)."""

    name = "sparse"

    def __init__(self, side=4, seed=1):
        self.side = side
        self.settings = scenes.settings(buoyancy=0.0, smoke_weight=0.0, vorticity=0.0, seed=seed)
        self.comb = scenes.combustion()

    def frame(self, step):
        brick, n = 8 * self.voxel_size, range(self.side)
        at = [((3 * x + 0.5) * brick, (3 * y + 0.5) * brick, (3 * z + 0.5) * brick) for z in n for y in n for x in n]
        srcs = [scenes.source(1 + k, "sphere", p, (0.03, 0.03, 0.03), smoke=400.0 + k) for k, p in enumerate(at)]
        return scenes.make_frame(self.settings, self.comb, False, srcs)


@pytest.mark.parametrize("smoke_divisor", [1, 2])
def test_more_aprons_than_room(smoke_divisor):
    """With places for a third of the aprons a frame is still the oracle's, and repeats bit for bit."""
    sc = SparseScene()
    budget = sc.side ** 3 * 512
    cam = render.look_at((3.2, 1.9, 3.6), (1.0, 1.0, 1.0), 200, 150, time=0.5)
    st = render.default_settings(ray_steps=256, shadow_samples=16)
    grid = sc.grid(budget=budget)
    grid.smoke_divisor = smoke_divisor
    out = {}

    def after(gpu, orc):
        assert gpu.stats().active_bricks == gpu.stats().pool_slots == sc.side ** 3
        out["gpu"] = [gpu.render(cam, st) for _ in range(12)]
        out["orc"] = orc.render(cam, st)

    parity.lockstep(sc, 4, lambda g: FluidSimulation(g), budget=budget, grid=grid, after=after)
    check(out["gpu"][0], out["orc"])
    for img in out["gpu"][1:]:
        assert np.array_equal(img, out["gpu"][0])


# Runs with and without memory to spare, which the checked build refuses when the environment says so.
WITHOUT = r"""
import json, os, sys
sys.path[:0] = [{root!r}, {root!r} + "/threejs-fire-pro_b200", {root!r} + "/tests"]
import numpy as np
from firepro import abi, render, scenes
from firepro.engine import FluidSimulation
import parity

sc = scenes.ForceScene()
grid = sc.grid(budget=2 ** 20, precision=abi.FP_PRECISION_MIXED)
grid.smoke_divisor = {divisor}
out = {{}}

def after(gpu, orc):
    errors = []
    before = gpu.lib.fp_last_error(gpu.h).decode()
    for half in (0, 1):
        cam = render.look_at((1.4, 1.0, 2.0), (0.0, 0.45, 0.0), 97, 65, time=0.5)
        cam.half_resolution = half
        st = render.default_settings(ray_steps=128, shadow_samples=16)
        img, ref = gpu.render(cam, st), orc.render(cam, st)
        assert ref[..., 3].max() > 0.05
        errors.append(parity.rel_l2(img, ref.astype(np.float64)))
    halves = gpu.field(abi.FP_FIELD_SCALARS)
    blob = bytes(gpu.snapshot())
    out.update(errors=errors, before=before, message=gpu.lib.fp_last_error(gpu.h).decode(), checked=gpu.read_bounds().checked,
               bad=gpu.read_bounds().count, field=float(np.abs(halves).max()),
               same=blob.find(halves.astype(np.float16).tobytes()) >= 0)

os.environ["FIREPRO_SPARE"] = "{spare}"
parity.lockstep(sc, 8, lambda g: FluidSimulation(g), budget=2 ** 20, grid=grid, after=after)
print("WITHOUT " + json.dumps(out))
"""


@pytest.mark.parametrize("divisor", [1, 2])
@pytest.mark.parametrize("spare", [0, 1])
def test_no_memory_to_spare(spare, divisor):
    """Without room for the boxes' tables, the aprons, the occupancy's maxima and the widening buffer
    (and with all of it, in the same build): the images are the oracle's, FP16 pools read back as the
    snapshot's halves, and a call that did without memory leaves no error behind."""
    if not abi.DEBUG_LIB_PATH.exists():
        pytest.fail("the bounds-checked build is missing: build.py --debug (or __graft_entry__.build())")
    root = str(Path(__file__).resolve().parent.parent)
    env = dict(os.environ, FIREPRO_LIBRARY=str(abi.DEBUG_LIB_PATH))
    r = subprocess.run([sys.executable, "-c", WITHOUT.format(root=root, spare=spare, divisor=divisor)], env=env,
                       capture_output=True, text=True, timeout=1200)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-3000:]
    out = json.loads([x for x in r.stdout.splitlines() if x.startswith("WITHOUT ")][-1][len("WITHOUT "):])
    assert out["checked"] == 1 and out["bad"] == 0
    assert max(out["errors"]) <= RENDER_TOL, out
    assert out["field"] > 0 and out["same"], out
    assert out["message"] == out["before"], out
