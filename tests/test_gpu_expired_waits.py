"""What follows a device-side wait that ran out: the call says so, the scene is
as it was, and its next calls are right.  The waits themselves never run out
here: bepugpu_probe_expired_wait sets their status words."""
from __future__ import annotations

import numpy as np
import pytest

from bepuphysics1_gb300 import native as N
from bepuphysics1_gb300 import scenes
from bepuphysics1_gb300.solver import GpuSpace, default_settings

from parity import DT

pytestmark = pytest.mark.gpu
FLAGS = N.STEP_ALL | N.STEP_COLLIDE
COLOURING, SLOTS, BROAD_PHASE, PERSISTENT = 1, 2, 4, 8


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


def test_unknown_waits_are_refused(gpu_context):
    b, m, _ = scenes.make_pile(nx=2, ny=2, nz=2)
    sp = GpuSpace(gpu_context, b, m)
    assert sp.ctx.lib.bepugpu_probe_expired_wait(sp.ctx.handle, sp.id, 1 << 31) == N.INVALID_ARGUMENT
    sp.close()
