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
