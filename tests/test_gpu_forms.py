"""The kernels' forms chosen by size, at the sizes where one takes over from another.

Tolerances are those of the suites whose oracle comparison each test repeats: fields within
test_gpu_parity's bound every step, images within relative L2 2e-3 (test_gpu_render), stored
halves widened exactly.
"""
import numpy as np
import pytest

from firepro import abi, render, scenes
from firepro.engine import FluidSimulation
import parity
from test_gpu_parity import check, run

pytestmark = pytest.mark.gpu

RENDER_TOL = 2e-3


@pytest.mark.parametrize("levels,pre,post,bottom", [(0, 3, 2, 5), (0, 1, 1, 1), (2, 2, 3, 3)])
def test_redblack_sweep_counts(levels, pre, post, bottom):
    """Two sweeps a launch, one left over (odd counts), and the finest level whose launches would
    not end in the buffer they started from (an odd number of them: half-sweeps in place), over
    two V-cycles; the coarsest levels' launch (all levels) and without it."""
    sched = abi.schedule(abi.FP_SMOOTHER_REDBLACK, levels=levels, pre=pre, post=post, bottom=bottom)
    check(run(scenes.SinglePlume(), 8, budget=2 ** 19, vcycles=2, schedule=sched))


@pytest.mark.parametrize("width,height", [(176, 176), (224, 144), (288, 224), (416, 304)])
def test_render_lanes(width, height):
    """16, 8, 4 and 2 lanes a ray, by the image's pixels (31250, 62500 and 125000 the lines)."""
    cam = render.look_at((1.4, 1.0, 2.0), (0.0, 0.45, 0.0), width, height, time=0.5)
    st = render.default_settings(ray_steps=32)
    out = {}

    def after(gpu, orc):
        out["gpu"], out["orc"] = gpu.render(cam, st), orc.render(cam, st)

    parity.lockstep(scenes.ForceScene(), 8, lambda g: FluidSimulation(g), budget=2 ** 20, after=after)
    err = parity.rel_l2(out["gpu"], out["orc"].astype(np.float64))
    assert out["orc"][..., 3].max() > 0.05
    assert err <= RENDER_TOL


@pytest.mark.parametrize("slots", [512, 1024, 1100])
def test_mixed_scalars_read_widened(slots):
    """The FP16 pools read back through the widening buffer (2^21 values: 1024 slots of 8^3 cells)
    are the halves that the snapshot holds."""
    scene = scenes.ForceScene()
    sim = FluidSimulation(scene.grid(budget=slots * 512, precision=abi.FP_PRECISION_MIXED))
    sim.set_runtime(0.05, slots * 512, True)
    for s in range(30):
        sim.step(scene.frame(s).frame)
    scalars = sim.field(abi.FP_FIELD_SCALARS)
    assert scalars.shape[0] == slots and np.abs(scalars).max() > 0
    halves = scalars.astype(np.float16)
    assert np.array_equal(halves.astype(np.float32), scalars)
    assert bytes(sim.snapshot()).find(halves.tobytes()) >= 0
    sim.dispose()
