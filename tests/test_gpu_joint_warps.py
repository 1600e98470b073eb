"""Joint groups with several warps (the CTA size that keeps every group
resident): a colour's joints split into one part per warp, of every length,
beside contact-only groups launched on a stream of their own."""
from __future__ import annotations

import pytest

from bepuphysics1_gb300 import scenes
from bepuphysics1_gb300.solver import default_settings
from parity import Pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("added", [False, True])
@pytest.mark.parametrize("chains,links,threads", [(1, 3, 0), (5, 16, 0), (5, 16, 64), (40, 9, 0), (40, 9, 256)])
def test_chains_beside_loose_bodies(gpu_context, added, chains, links, threads):
    b, m, j = scenes.make_chain(chains=chains, links=links, loose_bodies=4 * chains, seed=chains + links)
    if added:
        j = scenes.with_added_joint_types(b, j)
    p = Pair(gpu_context, b, m, j, settings=default_settings(), group_policy=(1, 1024, 4096, 64, threads))
    p.step(steps=4)
    errs, exact = p.compare()
    assert exact, errs
    p.close()


def test_steps_without_waiting(gpu_context):
    """Steps queued one behind another: the joint branch of a step ends before
    the next step's launches."""
    b, m, j = scenes.make_chain(chains=24, links=16, loose_bodies=200, seed=5)
    p = Pair(gpu_context, b, m, j, settings=default_settings())
    p.step(steps=40)
    errs, exact = p.compare()
    assert exact, errs
    p.close()
