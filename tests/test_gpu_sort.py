"""The broad phase's and pair bookkeeping's sorts, hash table and colouring at
the sizes where they can go wrong: few keys, keys on either side of a block's
tile, more pairs than the first buffer holds, and colours past one 64-bit mask."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from bepuphysics1_gb300 import native as N
from bepuphysics1_gb300 import scenes
from bepuphysics1_gb300.solver import GpuSpace, colour_list, default_settings
from oracle import broad_phase as obp

from parity import DT
from test_gpu_collide import _jumble

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 31, 33, 255, 1024, 2112])
def test_sizes(gpu_context, n):
    if n < 256:
        b, _, sh = _jumble(seed=n, n=n, sphere_every=4)
    else:  # overlapping layers: thousands of entries and pairs
        b, sh, _ = scenes.dropped_pile(nx=8, ny=8, nz=n // 64, drop_spacing=0.7, seed=n)
    sp = GpuSpace(gpu_context, b, None, shapes=sh)
    np.testing.assert_array_equal(sp.broad_phase(DT), obp.overlapping_pairs(b, sh, DT))
    sp.close()


def _cluster(n, seed):
    """n boxes and spheres all but on top of one another: every pair overlaps."""
    b, _, sh = _jumble(seed=seed, n=n, sphere_every=3)
    b = b.copy()
    b["position"][:] = np.random.default_rng(seed).uniform(-0.01, 0.01, (len(b), 3)).astype(np.float32)
    return b, sh


@pytest.mark.parametrize("n", [65, 150])
def test_every_pair(gpu_context, n):
    b, sh = _cluster(n, n)
    gpu_context.set_settings(default_settings())
    sp = GpuSpace(gpu_context, b, None, capacity=(len(b), len(b) * len(b), 0), shapes=sh)
    want = obp.overlapping_pairs(b, sh, DT)
    assert len(want) > 8 * len(b)  # past the first pair buffer
    np.testing.assert_array_equal(sp.broad_phase(DT), want)
    sp.set_materials(np.full((len(b), 3), 0.5, np.float32))
    for _ in range(2):  # all new, then all kept
        assert sp.update_pairs(DT) == len(want)
        m, _ = sp.download_constraints()
        got = np.sort(np.stack([m["body_a"], m["body_b"]], 1), axis=1)
        np.testing.assert_array_equal(got, want)
        colour, order, k = sp.colouring()
        c2, o2, k2 = colour_list(b, m)
        assert k == k2 and k > 60
        np.testing.assert_array_equal(colour, c2)
        np.testing.assert_array_equal(order, o2)
    sp.close()


def test_pairs_that_come_and_go(gpu_context):
    """Half the bodies moved away and back: kept, dropped and new records."""
    gpu_context.set_settings(default_settings())
    b, _, sh = _jumble(seed=9, n=600, sphere_every=5)
    sp = GpuSpace(gpu_context, b, None, capacity=(len(b), 16 * len(b), 0), shapes=sh)
    sp.set_materials(np.full((len(b), 3), 0.5, np.float32))
    away = b.copy()
    moving = np.flatnonzero(b["is_dynamic"] != 0)[::2]
    away["position"][moving, 1] += 500 + 10 * np.arange(len(moving), dtype=np.float32)
    for state in (b, away, b, b):
        sp.update_bodies(state)
        assert sp.update_pairs(DT) == len(obp.overlapping_pairs(state, sh, DT))
        m, _ = sp.download_constraints()
        got = np.sort(np.stack([m["body_a"], m["body_b"]], 1), axis=1)
        got = got[np.lexsort((got[:, 1], got[:, 0]))]
        np.testing.assert_array_equal(got, obp.overlapping_pairs(state, sh, DT))
        np.testing.assert_array_equal(sp.colouring()[0], colour_list(state, m)[0])
    sp.close()


def test_colouring_is_kept_until_asked_for(gpu_context):
    """The colouring of the last pair update, or of the upload after it: read
    late, twice, past a refused count, and after the scene's buffers went."""
    gpu_context.set_settings(default_settings())
    b, _, sh = _jumble(seed=12, n=300, sphere_every=4)
    sp = GpuSpace(gpu_context, b, None, capacity=(len(b), 16 * len(b), 0), shapes=sh)
    sp.set_materials(np.full((len(b), 3), 0.5, np.float32))
    away = b.copy()
    away["position"][np.flatnonzero(b["is_dynamic"] != 0)[::3], 1] += 500
    sp.update_pairs(DT)
    sp.update_bodies(away)
    n = sp.update_pairs(DT)  # fewer records, the colours of the update before never read
    m, _ = sp.download_constraints()
    want = colour_list(away, m)
    out = np.zeros(n + 1, np.int32)
    k = ctypes.c_uint32()

    def status(count):
        return sp.ctx.lib.bepugpu_get_colouring(sp.ctx.handle, sp.id, N.ptr(out), None, count, ctypes.byref(k))

    for again in range(2):
        assert status(n + 1) == status(0) == N.INVALID_ARGUMENT
        for got, w in zip(sp.colouring(), want):
            np.testing.assert_array_equal(got, w)
    sp.update_pairs(DT)
    sp.upload_bodies(away)  # materials and their buffers are given up
    for got, w in zip(sp.colouring(), want):
        np.testing.assert_array_equal(got, w)
    sp.set_materials(np.full((len(b), 3), 0.5, np.float32))
    sp.update_pairs(DT)
    sp.upload_constraints(m[: n // 2])
    for got, w in zip(sp.colouring(), colour_list(away, m[: n // 2])):
        np.testing.assert_array_equal(got, w)
    sp.close()


@pytest.mark.parametrize("n", [34, 560])
def test_slots_of_one_and_two_digits_of_colours(gpu_context, n):
    """A cluster's colours number its bodies: one digit up to 512, two beyond."""
    gpu_context.set_settings(default_settings())
    b, sh = _cluster(200, n)
    b, sh = np.resize(b[1:], n), np.resize(sh[1:], n)  # without the ground
    sp = GpuSpace(gpu_context, b, None, capacity=(n, n * n // 2, 0), shapes=sh)
    sp.set_materials(np.full((n, 3), 0.5, np.float32))
    for _ in range(2):
        assert sp.update_pairs(DT) == n * (n - 1) // 2
    m, _ = sp.download_constraints()
    colour, order, k = sp.colouring()
    c2, o2, k2 = colour_list(b, m)
    assert k == k2 and (k > 512) == (n > 512)
    np.testing.assert_array_equal(colour, c2)
    np.testing.assert_array_equal(order, o2)
    sp.close()
