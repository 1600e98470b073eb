"""The narrow phase's contact bookkeeping on its own: uploaded contacts of which
any subset, in any list order, goes away, so that kept contacts' lanes move down
from every place to every place, and turned stacked faces that cross each
other's clip lines at every corner."""
import numpy as np
import pytest

from bepuphysics1_gb300 import native as N
from bepuphysics1_gb300.solver import default_settings

from parity import DT, Pair
from test_gpu_collide import _all_pairs, _jumble, _random_quats

pytestmark = pytest.mark.gpu


def _assert_records(p):
    gm, _ = p.gpu.download_constraints()
    om, _ = p.oracle.get_constraints()
    for f in ("contact_count", "contact_order", "sliding_axis", "sliding_impulse", "twist_impulse"):
        np.testing.assert_array_equal(gm[f], om[f], err_msg=f)
    for f in gm["contacts"].dtype.names:
        np.testing.assert_array_equal(gm["contacts"][f], om["contacts"][f], err_msg=f)
    return gm


def _scrambled(m, spheres, rng):
    """The records with some contacts dropped, some ids unknown, another list
    order and every field filled; sphere pairs keep at most one contact."""
    m = m.copy()
    for r, one in zip(m, spheres):
        n = int(rng.integers(0, int(r["contact_count"]) + 1))
        keep = rng.permutation(int(r["contact_count"]))[:min(n, 1) if one else n]
        c = r["contacts"][keep].copy()
        lost = rng.random(len(keep)) < 0.4
        if not one:
            c["id"][lost] += 1000003
        for f in ("local_offset_a", "local_offset_b", "base_penetration_depth", "penetration_impulse"):
            c[f] = rng.uniform(0, 1, c[f].shape)
        if r["flags"] & N.MANIFOLD_NONCONVEX:
            c["friction_impulse"] = rng.uniform(-1, 1, len(keep))
            c["friction_direction"] = rng.uniform(-1, 1, (len(keep), 3))
        r["contacts"] = np.zeros(4, r["contacts"].dtype)
        r["contacts"][:len(keep)] = c
        r["contact_count"] = len(keep)
        code = 0xE4
        for q, at in enumerate(rng.permutation(len(keep))):
            code = code & ~(3 << (2 * q)) | int(at) << (2 * q)
        r["contact_order"] = code ^ 0xE4
    return m


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_any_contacts_go(gpu_context, seed):
    rng = np.random.default_rng(seed)
    b, m, sh = _jumble(seed=seed, n=220, spread=0.3, sphere_every=6)
    sphere = sh["type"] == N.SHAPE_SPHERE
    spheres = sphere[m["body_a"]] | sphere[m["body_b"]]
    m["flags"][rng.random(len(m)) < 0.5] |= N.MANIFOLD_NONCONVEX
    p = Pair(gpu_context, b, m, settings=default_settings(), shapes=sh)
    p.step(N.STEP_COLLIDE)
    full = _assert_records(p)
    p.close()
    assert (full["contact_count"] == 4).any()
    for _ in range(3):
        p = Pair(gpu_context, b, _scrambled(full, spheres, rng), settings=default_settings(), shapes=sh)
        p.step(N.STEP_COLLIDE)
        _assert_records(p)
        p.close()


@pytest.mark.parametrize("tilt", [0.0, 0.05])
def test_turned_faces(gpu_context, tilt):
    """Boxes on boxes, turned about the vertical by every angle to 90 degrees."""
    rng = np.random.default_rng(11)
    b, _, sh = _jumble(seed=4, n=200, sphere_every=1000)
    sh["type"][:] = N.SHAPE_BOX
    n = (len(b) - 1) // 2 * 2
    b, sh = b[:n + 1].copy(), sh[:n + 1].copy()
    low, high = np.arange(1, n, 2), np.arange(2, n + 1, 2)
    sh["size"][1:] = rng.uniform(0.3, 0.6, (n, 3)).astype(np.float32)
    b["position"][low] = np.stack([4 * np.arange(len(low)), np.full(len(low), 50), np.zeros(len(low))], 1)
    b["position"][high] = b["position"][low]
    b["position"][high, 1] += sh["size"][low, 1] + sh["size"][high, 1] - np.float32(0.02)
    b["position"][high, 0] += rng.uniform(-0.4, 0.4, len(high)).astype(np.float32)
    b["orientation"][low] = [0, 0, 0, 1]
    half = np.linspace(0, np.pi / 4, len(high))
    b["orientation"][high] = np.stack([0 * half, np.sin(half), 0 * half, np.cos(half)], 1)
    if tilt:
        b["orientation"][low] = _random_quats(len(low), rng, tilt)
    m = _all_pairs(b, sh)
    p = Pair(gpu_context, b, m, settings=default_settings(), shapes=sh)
    for _ in range(6):
        p.step()
        gm = _assert_records(p)
    assert (gm["contact_count"] == 4).any()
    p.close()
