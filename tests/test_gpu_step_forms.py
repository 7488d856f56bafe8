"""The step's forms chosen by a launch's size: a step that crosses a line replays the graph it has.

The lines (csrc/fp_engine.hpp): MANY_BRICKS computing bricks a launch, from which the multigrid's finest
restriction and brick levels' prolongation run apart from the sweeps, and OVERLAP_BLOCKS blocks of 8^3
cells an SM, up to which launches overlap.
"""
import pytest

from firepro import abi, scenes
from firepro.engine import FIXED_DT, SimulationBatch

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
