"""A solver visit's bookkeeping on the device: the children's zero-impulse
counts share one word with their activity, so every minimum iteration count up
to the largest allowed (whose count is the word's mark of a stopped child), the
maximum iteration count and every number of contacts run against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from bepuphysics1_gb300 import scenes
from bepuphysics1_gb300.solver import default_settings
from parity import Pair

pytestmark = pytest.mark.gpu


def _mixed():
    """Towers of boxes (four contacts) and spheres (one, NONCONVEX), some box
    manifolds cut to every smaller number of contacts."""
    b, m, _ = scenes.make_tower(180, seed=11)
    m = m.copy()
    boxes = np.flatnonzero(m["contact_count"] == 4)
    for k, i in enumerate(boxes[::2]):
        m["contact_count"][i] = k % 4
    return b, m


@pytest.mark.parametrize("policy", [None, (0, 1024, 4096, 64, 0)], ids=["groups", "sweeps"])
@pytest.mark.parametrize("minimum,maximum,iterations", [(0, 0x7FFFFFFF, 12), (1, 3, 12), (2, 0x7FFFFFFF, 40),
                                                        (14, 0x7FFFFFFF, 40)])
def test_iteration_counts(gpu_context, policy, minimum, maximum, iterations):
    s = default_settings()
    s["minimum_iteration_count"], s["maximum_iteration_count"], s["iteration_limit"] = minimum, maximum, iterations
    s["minimum_impulse"] = 0.02  # many children fall below it, some again after rising
    b, m = _mixed()
    p = Pair(gpu_context, b, m, settings=s, group_policy=policy)
    for _ in range(3):
        p.step()
        errs, exact = p.compare()
        assert exact, errs
    p.close()


@pytest.mark.parametrize("policy", [None, (0, 1024, 4096, 64, 0)], ids=["groups", "sweeps"])
@pytest.mark.parametrize("spheres", [0.0, 0.4])
def test_refresh_drops_contacts(gpu_context, policy, spheres):
    """Bodies turned and pushed so that the refresh drops first, middle and last
    contacts of a manifold: a group kernel compacts its staged copy and the
    manifold, and the prestep reads the copy."""
    b, m, _ = scenes.make_tower(260, seed=7, sphere_fraction=spheres)
    b = b.copy()
    rng = np.random.default_rng(4)
    dyn = b["is_dynamic"] != 0
    b["position"][dyn] += rng.uniform(-0.07, 0.07, (int(dyn.sum()), 3)).astype(np.float32)
    q = b["orientation"]
    q[dyn] += rng.normal(0, 0.06, (int(dyn.sum()), 4)).astype(np.float32)
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    gpu_context.set_settings(default_settings())
    p = Pair(gpu_context, b, m, group_policy=policy)
    before = m["contact_count"]
    for step in range(3):
        p.step()
        errs, exact = p.compare()
        assert exact, errs
        if step == 0:
            after = p.gpu.download_constraints()[0]["contact_count"]
            lost = before - after
            assert ((lost > 0) & (after > 0)).sum() > 5 or spheres  # some manifolds keep a part
            assert (lost > 0).sum() > 5
    p.close()
