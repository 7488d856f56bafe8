"""The step's forms chosen by a launch's size: the same results either side of a line, and a step that
crosses one replays the graph it has.

The lines (csrc/fp_engine.hpp): MANY_BRICKS computing bricks a launch, from which the multigrid's finest
restriction and brick levels' prolongation run apart from the sweeps, and OVERLAP_BLOCKS blocks of 8^3
cells an SM, up to which launches overlap.
"""
import numpy as np
import pytest

from firepro import abi, scenes
from firepro.engine import FIXED_DT, FluidSimulation, SimulationBatch
import parity
from test_gpu_batch import assert_same, snapshot
from test_gpu_parity import check

pytestmark = pytest.mark.gpu

MANY_BRICKS, OVERLAP_BRICKS = 1000, 6 * 148
BUDGET = 330 * 512  # of each member: reached by the burst's step


def members(count):
    return [scenes.LargeScene(seed=3 + k) for k in range(count)]


def add(batch, scene, precision, vcycles, schedule):
    i = batch.add(scene.grid(budget=BUDGET, precision=precision))
    batch.set_runtime(i, 0.05, BUDGET, True)
    if vcycles > 1:
        batch.set_solver(i, vcycles, 0.0)
    if schedule is not None:
        batch.set_schedule(i, schedule)
    return i


JACOBI_FCG = abi.schedule(krylov=abi.FP_KRYLOV_FCG, topology=1)
RB = abi.schedule(abi.FP_SMOOTHER_REDBLACK)


@pytest.mark.parametrize("precision", [abi.FP_PRECISION_FP32, abi.FP_PRECISION_MIXED])
@pytest.mark.parametrize("vcycles,schedule", [(1, None), (2, None), (2, JACOBI_FCG), (2, RB)])
def test_batch_across_the_lines_matches_alone(precision, vcycles, schedule):
    """Four members whose sum is past both lines while each alone is below them, bit for bit; the first
    steps of each in a launch of its own, so that the batch crosses the lines at once."""
    mem, grown, together = members(4), 34, 6
    batch = SimulationBatch(8)
    ids = [add(batch, sc, precision, vcycles, schedule) for sc in mem]
    for sc, i in zip(mem, ids):
        for s in range(grown):
            batch.step([(i, sc.frame(s).frame, FIXED_DT)])
    for s in range(grown, grown + together):
        frames = [sc.frame(s) for sc in mem]
        batch.step([(i, fd.frame, FIXED_DT) for i, fd in zip(ids, frames)])
    bricks = [batch.stats(i).active_bricks for i in ids]
    assert max(bricks) < OVERLAP_BRICKS < MANY_BRICKS < sum(bricks)
    for sc, i in zip(mem, ids):
        sim = FluidSimulation(sc.grid(budget=BUDGET, precision=precision))
        sim.set_runtime(0.05, BUDGET, True)
        if vcycles > 1:
            sim.set_solver(vcycles, 0.0)
        if schedule is not None:
            sim.set_schedule(schedule)
        for s in range(grown + together):
            sim.step(sc.frame(s).frame)
        assert_same(snapshot(lambda f: batch.field(i, f), lambda t: batch.table(i, t)),
                    snapshot(sim.field, sim.table), f"member {i}")
        sim.dispose()
    batch.dispose()


def test_crossing_step_replays_the_graph_it_has():
    """The first step past a line launches what the steps before it did; the next one its own form
    (which has other launches: prolongation apart)."""
    sched = abi.schedule(topology=1)  # every step with the same optional launches
    mem = members(4)
    batch = SimulationBatch(8)
    ids = [add(batch, sc, abi.FP_PRECISION_FP32, 1, sched) for sc in mem]
    step = dict.fromkeys(ids, 0)

    def launch(which):
        """The launches of one step of these members."""
        frames = {i: mem[ids.index(i)].frame(step[i]) for i in which}
        before = batch.stats(which[0]).kernel_launches
        batch.step([(i, frames[i].frame, FIXED_DT) for i in which])
        for i in which:
            step[i] += 1
        return batch.stats(which[0]).kernel_launches - before

    for pair in (ids[:2], ids[2:]):
        for _ in range(40):
            below = launch(pair)
    bricks = [batch.stats(i).active_bricks for i in ids]
    assert max(sum(bricks[:2]), sum(bricks[2:])) < OVERLAP_BRICKS < MANY_BRICKS < sum(bricks)
    assert launch(ids) == below
    past = launch(ids)
    assert past != below and launch(ids) == past
    assert launch(ids[:2]) == below
    batch.dispose()


@pytest.mark.parametrize("divisor,brick", [(2, 16), (2, 8), (4, 16)])
def test_redblack_on_a_divided_lattice(divisor, brick):
    """Red-black legs where the velocity lattice is coarser: 8, 4 and 2 cells a brick are other levels."""
    sc = scenes.ForceScene()
    sc.brick_size, sc.velocity_divisor = brick, divisor
    sched = abi.schedule(abi.FP_SMOOTHER_REDBLACK, pre=3, post=2, bottom=4)
    check(parity.lockstep(sc, 8, lambda g: FluidSimulation(g), budget=2 ** 20, vcycles=2, schedule=sched), min_active=4)


def test_widened_past_the_buffer():
    """FP16 pools of more values than the widening buffer holds (2^21), with data in every piece: the
    stored halves, exactly."""
    scene = scenes.LargeScene()
    slots = 1600
    sim = FluidSimulation(scene.grid(budget=slots * 512, precision=abi.FP_PRECISION_MIXED))
    sim.set_runtime(0.05, slots * 512, True)
    for s in range(130):
        sim.step(scene.frame(s).frame)
    scalars = sim.field(abi.FP_FIELD_SCALARS)
    piece = 2 ** 21 // (4 * 512)
    assert scalars.shape[0] == slots > piece
    assert np.abs(scalars[:piece]).max() > 0 and np.abs(scalars[piece:]).max() > 0
    halves = scalars.astype(np.float16)
    assert np.array_equal(halves.astype(np.float32), scalars)
    assert bytes(sim.snapshot()).find(halves.tobytes()) >= 0
    sim.dispose()
