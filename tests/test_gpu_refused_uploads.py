"""A refused constraint upload leaves the scene as it was: its list, its
colouring and its steps, on the sweep path and in island groups."""
from __future__ import annotations

import numpy as np
import pytest

from bepuphysics1_gb300 import native as N
from bepuphysics1_gb300 import scenes
from bepuphysics1_gb300.solver import GpuSpace, default_settings

from parity import DT

pytestmark = pytest.mark.gpu
FLAGS = N.STEP_ALL | N.STEP_COLLIDE


def _refused(m, kind):
    """Another list (half the pairs, the others turned round in order) with one record refused."""
    m = m[::-2].copy()
    if kind == "order":
        m["contact_count"][3] = 2
        m["contact_order"][3] = 0xE4  # both contacts the first
    elif kind == "two_bodies":
        m["body_b"][3] = -1
    else:
        m["body_b"][3] = 1 << 20
    return m


@pytest.mark.parametrize("policy", [(0, 1024, 4096, 64, 0), None], ids=["sweeps", "groups"])
@pytest.mark.parametrize("kind", ["order", "two_bodies", "out_of_range"])
def test_the_scene_goes_on_as_it_was(gpu_context, policy, kind):
    gpu_context.set_settings(default_settings())
    b, m, _, sh = scenes.make_tower(60, seed=11, narrow_phase=1)
    sp, twin = (GpuSpace(gpu_context, b, m, shapes=sh, group_policy=policy) for _ in range(2))
    for s in (sp, twin):
        for _ in range(3):
            s.step(DT, FLAGS)
    with pytest.raises(N.ArgumentException):
        sp.upload_constraints(_refused(m, kind))
    sp.manifold_count = len(m)
    for got, want in zip(sp.colouring(), twin.colouring()):
        np.testing.assert_array_equal(got, want)
    for _ in range(3):
        sp.step(DT, FLAGS)
        twin.step(DT, FLAGS)
    np.testing.assert_array_equal(sp.download_bodies(), twin.download_bodies())
    np.testing.assert_array_equal(sp.download_constraints()[0], twin.download_constraints()[0])
    sp.close()
    twin.close()
