"""Served scenes that take the one-scene path through the barrier-free sweeps
(csrc/flow.cu): the sweep path and an island past a CTA's shared memory, alone,
in the mix, spilled and restored, and given back."""
from __future__ import annotations

import time

import numpy as np
import pytest

from bepuphysics1_gb300 import native as N
from bepuphysics1_gb300 import scenes
from bepuphysics1_gb300.serve import Server
from bepuphysics1_gb300.solver import GpuSpace, default_settings

from parity import DT

pytestmark = pytest.mark.gpu
SWEEPS = (0, 1024, 4096, 64, 0)  # no island groups
STEPS = 40
# Both sides run the same graph, so they take the same time: four times the
# scene's own is far from that and from the dozens of times that a launch on a
# fraction of the SMs takes.
SLACK, SLACK_US = 4.0, 4000.0


def _pile(seed=3):
    return scenes.make_pile(nx=16, ny=16, nz=16, spacing=1.05, size_min=1.0, size_max=1.0, jitter=0.05, seed=seed)[:2]


def _island(seed=8):
    return scenes.make_pile(nx=9, ny=8, nz=9, spacing=1.05, size_min=1.0, size_max=1.0, jitter=0.05, seed=seed)[:2]


SCENES = {"sweeps": (_pile, SWEEPS), "large_island": (_island, None)}


def _step_us(ctx, sp, steps):
    ctx.synchronize()
    t = time.perf_counter()
    for _ in range(steps):
        sp.step(DT)
    ctx.synchronize()
    return (time.perf_counter() - t) * 1e6


def _state(sp, b, m):
    return sp.download_bodies(b.copy()), sp.download_constraints(m.copy())[0]


def _assert_same(got, want):
    for f in ("position", "orientation", "linear_velocity", "angular_velocity"):
        np.testing.assert_array_equal(got[0][f], want[0][f])
    np.testing.assert_array_equal(got[1]["contacts"]["penetration_impulse"], want[1]["contacts"]["penetration_impulse"])
    np.testing.assert_array_equal(got[1]["sliding_impulse"], want[1]["sliding_impulse"])


@pytest.mark.parametrize("kind", sorted(SCENES))
@pytest.mark.parametrize("spilled", [False, True])
def test_a_served_scene_steps_like_its_own(gpu_context, kind, spilled):
    gpu_context.set_settings(default_settings())
    make, policy = SCENES[kind]
    b, m = make()
    alone = GpuSpace(gpu_context, b, m, group_policy=policy)
    served = GpuSpace(gpu_context, b, m, group_policy=policy)
    other = GpuSpace(gpu_context, b, m, group_policy=policy)
    alone.step(DT)  # the step graph
    own_us = _step_us(gpu_context, alone, STEPS)
    # a budget for one of the two served scenes: adding the second spills the first
    srv = Server(gpu_context, dt=float(DT), budget_bytes=_bytes(gpu_context, served) * 3 // 2 if spilled else None)
    srv.add(served)
    srv.add(other)
    assert srv.stats()["spills"] == (1 if spilled else 0)
    srv.submit(served.id, 1, 0)
    srv.drain()
    srv.submit(served.id, STEPS, 1)
    srv.drain()
    done = srv.poll()
    assert done["status"].tolist() == [N.OK, N.OK]
    served_us = float(done["done_us"][1] - done["start_us"][1])
    srv.release(served)
    srv.release(other)
    srv.close()
    _assert_same(_state(served, b, m), _state(alone, b, m))
    # the step graph that the worker built goes on with the scene
    back_us = _step_us(gpu_context, served, STEPS)
    for sp in (alone, served, other):
        sp.close()
    assert served_us < SLACK * own_us + SLACK_US, (served_us, own_us)
    assert back_us < SLACK * own_us + SLACK_US, (back_us, own_us)


def _bytes(ctx, sp):
    srv = Server(ctx, dt=float(DT))
    srv.add(sp)
    n = int(srv.stats()["resident_bytes"])
    srv.release(sp)
    srv.close()
    return n


def test_sweep_scenes_and_towers_in_one_wave(gpu_context):
    """Several scenes' sweeps beside one another and beside a wave's batched groups."""
    gpu_context.set_settings(default_settings())
    parts = [(_pile(s), SWEEPS) for s in (3, 4, 5)] + [(_island(), None)]
    parts += [(scenes.make_tower(60 + 20 * i, seed=i)[:2], None) for i in range(8)]
    spaces = [GpuSpace(gpu_context, b, m, group_policy=pol) for (b, m), pol in parts]
    srv = Server(gpu_context, dt=float(DT), waves_in_flight=4)
    for sp in spaces:
        srv.add(sp)
    for tag in range(3):
        for sp in spaces:
            while srv.submit(sp.id, 5, tag) == N.QUEUE_FULL:
                pass
    srv.drain()
    done = srv.poll()
    assert len(done) == 3 * len(spaces) and np.all(done["status"] == N.OK)
    for sp in spaces:
        srv.release(sp)
    srv.close()
    for sp, ((b, m), pol) in zip(spaces, parts):
        alone = GpuSpace(gpu_context, b, m, group_policy=pol)
        for _ in range(15):
            alone.step(DT)
        _assert_same(_state(sp, b, m), _state(alone, b, m))
        alone.close()
        sp.close()


def test_scenes_without_sweeps_hold_no_tables(gpu_context):
    """The sweeps' tables, 26 bytes a manifold and 40 a body, come with the first
    constraints that need them and stay."""
    gpu_context.set_settings(default_settings())
    b, m = scenes.make_tower(150, seed=6)[:2]  # one island group by default
    GpuSpace(gpu_context, b, m).close()  # blocks that an earlier test's spills left pending are reclaimed here

    def bytes_of(make):
        before = gpu_context.memory_usage()[1]
        sp = make()
        return sp, gpu_context.memory_usage()[1] - before

    grouped, none = bytes_of(lambda: GpuSpace(gpu_context, b, m))
    swept, tables = bytes_of(lambda: GpuSpace(gpu_context, b, m, group_policy=SWEEPS))
    extra = tables - none
    assert 24 * len(m) + 40 * len(b) <= extra < 24 * len(m) + 40 * len(b) + 8192
    before = gpu_context.memory_usage()[1]
    grouped.set_group_policy(*SWEEPS)
    for _ in range(2):
        grouped.upload_constraints(m)
        assert gpu_context.memory_usage()[1] - before == extra
    for sp in (grouped, swept):
        for _ in range(3):
            sp.step(DT)
    _assert_same(_state(grouped, b, m), _state(swept, b, m))
    grouped.close()
    swept.close()
    assert gpu_context.memory_usage()[1] == before - none - tables
