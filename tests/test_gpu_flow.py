"""The barrier-free sweeps (csrc/flow.cu) against the oracle where their turns
can go wrong: bodies on either side of the 16 manifolds a tag's set holds, steps
of more sweeps than a masked tag counts, chunks of every remainder, a step
without solve sweeps, and manifolds that stop and start between steps."""
from __future__ import annotations

import numpy as np
import pytest

from bepuphysics1_gb300 import native as N
from bepuphysics1_gb300 import scenes
from bepuphysics1_gb300.solver import default_settings
from parity import Pair

pytestmark = pytest.mark.gpu
SWEEPS = (0, 1024, 4096, 64, 0)  # no island groups
NO_REFRESH = N.STEP_ALL & ~N.STEP_REFRESH_CONTACTS


def _pile(nx, ny, nz, seed=3):
    return scenes.make_pile(nx=nx, ny=ny, nz=nz, spacing=1.05, size_min=1.0, size_max=1.0, jitter=0.05,
                            friction_min=0.6, friction_max=0.6, seed=seed)[:2]


def _run(ctx, b, m, s, steps=3, flags=N.STEP_ALL):
    p = Pair(ctx, b, m, settings=s, group_policy=SWEEPS)
    for _ in range(steps):
        p.step(flags=flags)
        errs, exact = p.compare()
        assert exact, errs
    p.close()


@pytest.mark.parametrize("degree", [1, 15, 16, 17, 40])
def test_a_body_with_many_manifolds(gpu_context, degree):
    b, m = _pile(5, 3, 5)
    hub = len(b) // 2
    free = np.flatnonzero((m["body_a"] != hub) & (m["body_b"] != hub))
    keep = np.setdiff1d(np.arange(len(m)), np.flatnonzero((m["body_a"] == hub) | (m["body_b"] == hub)))
    m["body_a"][free[:degree]] = hub  # contacts far from the hub: long lever arms, kept without the refresh
    _run(gpu_context, b, m[keep], default_settings(), flags=NO_REFRESH)


@pytest.mark.parametrize("iterations", [0, 1, 4093, 4094, 4096])
def test_sweep_counts(gpu_context, iterations):
    s = default_settings()
    s["iteration_limit"] = iterations
    b, m = _pile(3, 2, 2)
    _run(gpu_context, b, m, s, steps=2)


@pytest.mark.parametrize("columns", [1, 31, 32, 33, 65])
def test_chunk_remainders(gpu_context, columns):
    """Separate two-box columns: a colour holds one manifold per column."""
    b, m, _ = scenes.make_pile(nx=columns, ny=2, nz=1, spacing=2.0, jitter=0.02, ground_size=(300.0, 1.0, 10.0), seed=4)
    _run(gpu_context, b, m, default_settings())


def test_manifolds_without_work(gpu_context):
    b, m = _pile(4, 3, 4)
    m["contact_count"][::5] = 0
    m["flags"][::7] = N.MANIFOLD_ACTIVE
    s = default_settings()
    s["minimum_impulse"] = 0.05
    _run(gpu_context, b, m, s, steps=5)


def _together(*parts):
    """Scenes side by side: bodies and manifolds concatenated."""
    bodies, manifolds, at, x = [], [], 0, 0.0
    for b, m in parts:
        b, m = b.copy(), m.copy()
        b["position"][:, 0] += x
        m["contacts"]["position"][..., 0] += x
        x += 300.0
        for end in ("body_a", "body_b"):
            m[end] += np.where(m[end] >= 0, at, 0).astype(np.int32)
        at += len(b)
        bodies.append(b)
        manifolds.append(m)
    return np.concatenate(bodies), np.concatenate(manifolds)


@pytest.mark.parametrize("policy", [None, (1, 400, 4096, 64, 0)], ids=["groups", "groups_and_sweeps"])
@pytest.mark.parametrize("flags", [N.STEP_ALL, N.STEP_FORCES | N.STEP_SOLVE, N.STEP_POSITIONS])
def test_large_islands_beside_small_ones(gpu_context, policy, flags):
    """Islands past a CTA's shared memory (stepped by grid-wide launches), small
    islands in group CTAs and, with 400 bodies a group, sweep islands at once."""
    b, m = _together(_pile(7, 7, 7), scenes.make_tower(150, seed=2)[:2], _pile(8, 6, 9, seed=8))
    b["linear_velocity"][1:40, 1] = -0.5
    s = default_settings()
    p = Pair(gpu_context, b, m, settings=s, group_policy=policy)
    for _ in range(4):
        p.step(flags=flags)
        errs, exact = p.compare()
        assert exact, errs
        assert errs["position"] == 0 and errs["orientation"] == 0
    p.close()
