"""Simulations that join a batch or a server while a step is in flight start as they do on an idle
device: what is written into their pools at creation is ordered with the launches around it."""
import numpy as np
import pytest

from firepro import abi, scenes
from firepro.engine import FIXED_DT, FireServer, FluidSimulation, SimulationBatch
from test_gpu_batch import assert_same, snapshot

pytestmark = pytest.mark.gpu

BUDGET = 64 * 512


def newcomers(count):
    return [scenes.SinglePlume(seed=20 + k) for k in range(count)]


def alone(scene, steps):
    sim = FluidSimulation(scene.grid(budget=BUDGET))
    sim.set_runtime(0.05, BUDGET, True)
    for s in range(steps):
        sim.step(scene.frame(s).frame)
    snap = snapshot(sim.field, sim.table)
    sim.dispose()
    return snap


def test_batch_members_added_behind_a_step():
    """Several members are added right behind a large one's step, which is still running, and step with
    it: tables and fields are those of the member alone, bit for bit."""
    large, count, steps = scenes.LargeScene(seed=5), 6, 5
    batch = SimulationBatch(8)
    big = batch.add(large.grid(budget=2 ** 21))
    batch.set_runtime(big, 0.05, 2 ** 21, True)
    at = 0
    for at in range(60):
        batch.step([(big, large.frame(at).frame, FIXED_DT)])
    mem, ids = newcomers(count), []
    for sc in mem:
        for _ in range(4):
            at += 1
            batch.step([(big, large.frame(at).frame, FIXED_DT)])
        i = batch.add(sc.grid(budget=BUDGET))
        batch.set_runtime(i, 0.05, BUDGET, True)
        ids.append(i)
    for s in range(steps):
        at += 1
        frames = [sc.frame(s) for sc in mem] + [large.frame(at)]
        batch.step([(i, fd.frame, FIXED_DT) for i, fd in zip(ids + [big], frames)])
    for sc, i in zip(mem, ids):
        assert_same(snapshot(lambda f: batch.field(i, f), lambda t: batch.table(i, t)), alone(sc, steps), f"member {i}")
    batch.dispose()


def test_sessions_opened_while_others_step():
    """Sessions opened while another's requests run hold the fields of their scene alone."""
    large, count, steps = scenes.LargeScene(seed=5), 6, 5
    server = FireServer(16 << 30, max_sessions=16, brick_size=8)
    big = server.open(large.grid(budget=2 ** 21))
    for s in range(40):
        server.submit(big, large.frame(s).frame)
    mem, ids = newcomers(count), []
    for sc in mem:
        i = server.open(sc.grid(budget=BUDGET))
        ids.append(i)
        for s in range(steps):
            server.submit(i, sc.frame(s).frame)
    server.drain()
    for sc, i in zip(mem, ids):
        got = server.field(i, abi.FP_FIELD_SCALARS)
        assert np.abs(got).max() > 0
        assert np.array_equal(got, alone(sc, steps)[("f", abi.FP_FIELD_SCALARS)])
    server.dispose()


def test_restored_behind_a_step():
    """A snapshot restored into a batch member right behind another's step steps on as the original."""
    large, sc = scenes.LargeScene(seed=5), scenes.SinglePlume(seed=21)
    source = FluidSimulation(sc.grid(budget=BUDGET))
    source.set_runtime(0.05, BUDGET, True)
    for s in range(6):
        source.step(sc.frame(s).frame)
    blob = bytes(source.snapshot())
    source.dispose()
    batch = SimulationBatch(8)
    big, i = batch.add(large.grid(budget=2 ** 21)), batch.add(sc.grid(budget=BUDGET))
    batch.set_runtime(big, 0.05, 2 ** 21, True)
    for s in range(60):
        batch.step([(big, large.frame(s).frame, FIXED_DT)])
    batch.restore(i, blob)
    for s in range(6, 9):
        fd, fl = sc.frame(s), large.frame(54 + s)
        batch.step([(i, fd.frame, FIXED_DT), (big, fl.frame, FIXED_DT)])
    assert_same(snapshot(lambda f: batch.field(i, f), lambda t: batch.table(i, t)), alone(sc, 9), "restored member")
    batch.dispose()
