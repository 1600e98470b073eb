"""What follows a device-side wait that ran out: the call says so, the scene is
as it was, and its next calls are right.  The waits themselves never run out
here: bepugpu_probe_expired_wait sets their status words."""
from __future__ import annotations

import numpy as np
import pytest

from bepuphysics1_gb300 import native as N
from bepuphysics1_gb300 import scenes
from bepuphysics1_gb300.serve import Server
from bepuphysics1_gb300.solver import GpuSpace, batch_step, body_states, default_settings, islands_of

from parity import DT

pytestmark = pytest.mark.gpu
FLAGS = N.STEP_ALL | N.STEP_COLLIDE
COLOURING, SLOTS, BROAD_PHASE, PERSISTENT, SWEEPS, TABLES = 1, 2, 4, 8, 16, 32


def _expire(sp, where):
    sp.ctx.check(sp.ctx.lib.bepugpu_probe_expired_wait(sp.ctx.handle, sp.id, where))


def _timeout(call, *args):
    with pytest.raises(N.BepuError) as e:
        call(*args)
    assert e.value.status == N.TIMEOUT
    return str(e.value)


def _heap(ctx, seed):
    """Overlapping layers of boxes after a few frames: pairs for several blocks
    of a sort, kept on the device."""
    b, sh, fr = scenes.dropped_pile(nx=12, ny=8, nz=12, drop_spacing=0.7, seed=seed)
    sp = GpuSpace(ctx, b, None, capacity=(len(b), 16 * len(b), 0), shapes=sh)
    sp.set_materials(np.stack([fr, fr, np.zeros_like(fr)], 1))
    for _ in range(10):
        sp.update_pairs(float(DT))
        sp.step(DT, FLAGS)
    return sp


def _state(sp):
    m, _ = sp.download_constraints()
    return [sp.download_bodies(), m, *sp.colouring()[:2], sp.broad_phase(float(DT))]


def _same(a, b):
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


def _frames(sp, n):
    for _ in range(n):
        sp.update_pairs(float(DT))
        sp.step(DT, FLAGS)


@pytest.mark.parametrize("where", [COLOURING, SLOTS, BROAD_PHASE])
def test_pair_update_that_gave_up(gpu_context, where):
    gpu_context.set_settings(default_settings())
    sp, twin = _heap(gpu_context, 21), _heap(gpu_context, 21)
    before = _state(sp)
    for _ in range(2):
        _expire(sp, where)
        assert ("broad phase" if where == BROAD_PHASE else "update_pairs") in _timeout(sp.update_pairs, float(DT))
        _same(_state(sp), before)
    # the scene steps on with the list it has, and the next update is whole
    sp.step(DT, FLAGS)
    twin.step(DT, FLAGS)
    _same(_state(sp), _state(twin))
    _frames(sp, 5)
    _frames(twin, 5)
    _same(_state(sp), _state(twin))
    sp.close()
    twin.close()


def test_broad_phase_that_gave_up(gpu_context):
    gpu_context.set_settings(default_settings())
    sp = _heap(gpu_context, 22)
    want = sp.broad_phase(float(DT))
    assert len(want) > 0
    for _ in range(2):
        _expire(sp, BROAD_PHASE)
        _timeout(sp.broad_phase, float(DT))
        np.testing.assert_array_equal(sp.broad_phase(float(DT)), want)
    sp.close()


def test_sorts_after_a_persistent_step_that_gave_up(gpu_context):
    gpu_context.set_settings(default_settings())
    sp, twin = _heap(gpu_context, 23), _heap(gpu_context, 23)
    sp.ctx.check(sp.ctx.lib.bepugpu_set_solve_mode(sp.ctx.handle, sp.id, N.MODE_PERSISTENT))
    _expire(sp, PERSISTENT)
    _same(_state(sp), _state(twin))
    assert sp.update_pairs(float(DT)) == twin.update_pairs(float(DT))
    _same(_state(sp), _state(twin))
    _timeout(sp.ctx.synchronize)
    _frames(sp, 3)
    _frames(twin, 3)
    sp.ctx.synchronize()
    _same(_state(sp), _state(twin))
    sp.close()
    twin.close()


GROUPS_OFF = (0, 1024, 4096, 64, 0)


def _flowing(ctx, seed):
    b, m, _ = scenes.make_pile(nx=4, ny=3, nz=4, seed=seed)
    sp = GpuSpace(ctx, b, m, group_policy=GROUPS_OFF)
    sp.step(DT)
    ctx.synchronize()
    return sp, b, m


# the calls that hand a scene's results out
READS = {
    "step_state": lambda sp, b, m: sp.step_state(body_states(b), None, DT),
    "step_host": lambda sp, b, m: sp.step_host(b, m, DT),
    "download_state": lambda sp, b, m: sp.download_state(body_states(b)),
    "download_bodies": lambda sp, b, m: sp.download_bodies(),
    "download_constraints": lambda sp, b, m: sp.download_constraints(),
    "get_islands": lambda sp, b, m: (sp.set_islands(islands_of(b, m)), sp.get_islands()),
    "batch_step": lambda sp, b, m: batch_step(sp.ctx, [sp], DT),
}


@pytest.mark.parametrize("call", sorted(READS))
def test_a_scenes_own_call_reports_its_sweeps(gpu_context, call):
    gpu_context.set_settings(default_settings())
    (a, ab, am), (o, ob, om) = _flowing(gpu_context, 3), _flowing(gpu_context, 4)
    for sp, b, m in ((a, ab, am), (o, ob, om)):
        sp.download_bodies(b)
    _expire(a, SWEEPS)
    READS[call](o, ob, om)  # another scene's call neither reports nor clears it
    assert f"scene {a.id}" in _timeout(READS[call], a, ab, am)
    READS[call](a, ab, am)
    gpu_context.synchronize()
    a.close()
    o.close()


def test_synchronize_reports_every_scene(gpu_context):
    gpu_context.set_settings(default_settings())
    (a, _, _), (o, _, _) = _flowing(gpu_context, 3), _flowing(gpu_context, 4)
    _expire(o, SWEEPS)
    _expire(a, SWEEPS)
    assert f"scene {a.id}:" in _timeout(gpu_context.synchronize)
    gpu_context.synchronize()
    a.download_bodies()
    o.close()  # a closed scene's word goes to the next one, clear
    p, _, _ = _flowing(gpu_context, 5)
    p.download_bodies()
    a.close()
    p.close()


def test_batch_advances_every_scene_before_it_reports(gpu_context):
    gpu_context.set_settings(default_settings())
    (a, _, _), (o, _, _), (t, _, _) = (_flowing(gpu_context, s) for s in (3, 4, 4))
    _expire(a, SWEEPS)
    _timeout(batch_step, gpu_context, [a, o], DT, 3)
    for _ in range(3):
        t.step(DT)
    np.testing.assert_array_equal(o.download_bodies(), t.download_bodies())
    for sp in (a, o, t):
        sp.close()


def test_a_served_requests_completion_reports_its_sweeps(gpu_context):
    gpu_context.set_settings(default_settings())
    (a, _, _), (o, _, _) = _flowing(gpu_context, 3), _flowing(gpu_context, 4)
    _expire(a, SWEEPS)
    srv = Server(gpu_context, dt=float(DT))
    srv.add(a)
    srv.add(o)
    status = {}
    for tag, sp in enumerate((o, a, a, o)):
        srv.submit(sp.id, 2, tag)
        srv.drain()
    for c in srv.poll():
        status[int(c["tag"])] = int(c["status"])
    assert status == {0: N.OK, 1: N.TIMEOUT, 2: N.OK, 3: N.OK}
    assert f"scene {a.id}" in srv.last_error()
    srv.release(a)
    srv.release(o)
    srv.close()
    gpu_context.synchronize()
    a.close()
    o.close()


def test_upload_that_gave_up(gpu_context):
    gpu_context.set_settings(default_settings())
    (a, _, m), (o, _, _) = _flowing(gpu_context, 3), _flowing(gpu_context, 3)
    _expire(a, TABLES)
    assert "upload_constraints" in _timeout(a.upload_constraints, m)
    with pytest.raises(N.InvalidOperationException):
        a.step(DT)
    a.upload_constraints(m)
    o.upload_constraints(m)
    for sp in (a, o):
        sp.step(DT)
    np.testing.assert_array_equal(a.download_bodies(), o.download_bodies())
    a.close()
    o.close()


def test_unknown_waits_are_refused(gpu_context):
    b, m, _ = scenes.make_pile(nx=2, ny=2, nz=2)
    sp = GpuSpace(gpu_context, b, m)
    probe = sp.ctx.lib.bepugpu_probe_expired_wait
    assert probe(sp.ctx.handle, sp.id, 1 << 31) == N.INVALID_ARGUMENT
    assert probe(sp.ctx.handle, sp.id, SWEEPS) == N.INVALID_OPERATION  # island groups alone
    sp.close()
