"""Record updates at the sizes of their blocks: the new state and the inertia of
the new orientation equal a fresh upload's, and a refused record leaves the
scene as it was and is named by the lowest index."""
import numpy as np
import pytest

from bepuphysics1_gb300 import native as N
from bepuphysics1_gb300 import scenes
from bepuphysics1_gb300.solver import GpuSpace, default_settings

from parity import DT
from test_gpu_collide import _random_quats

pytestmark = pytest.mark.gpu


def _scene(n, seed):
    b, m, _ = scenes.make_tower(600, seed=seed)
    b = b[:n].copy()
    return b, m[(m["body_a"] < n) & (m["body_b"] < n)].copy()


@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 256, 300])
def test_update_equals_upload(gpu_context, n):
    gpu_context.set_settings(default_settings())
    b, m = _scene(n, n)
    rng = np.random.default_rng(n)
    new = b.copy()
    new["orientation"] = _random_quats(n, rng, np.pi)
    for f in ("position", "linear_velocity", "angular_velocity"):
        new[f] += rng.normal(0, 0.1, new[f].shape).astype(np.float32)
    updated, fresh = GpuSpace(gpu_context, b, m), GpuSpace(gpu_context, new, m)
    updated.update_bodies(new)
    assert updated.download_bodies().tobytes() == new.tobytes()
    for sp in (updated, fresh):  # the solver reads the inertia that the update left
        sp.step(DT, N.STEP_SOLVE)
        sp.step(DT, N.STEP_ALL)
    assert updated.download_bodies().tobytes() == fresh.download_bodies().tobytes()
    updated.close()
    fresh.close()


@pytest.mark.parametrize("bad", [[0], [128, 129], [299], [5, 0, 299]])
def test_lowest_refused_record_is_named(gpu_context, bad):
    gpu_context.set_settings(default_settings())
    b, m = _scene(300, 4)
    sp = GpuSpace(gpu_context, b, m)
    wrong = b.copy()
    wrong["position"] += 1
    wrong["linear_damping"][bad] += np.float32(0.25)
    with pytest.raises(N.BepuError, match=f"body {min(bad)} "):
        sp.update_bodies(wrong)
    with pytest.raises(N.BepuError, match=f"body {min(bad)} "):
        sp.step_host(wrong, m.copy(), DT)
    assert sp.download_bodies().tobytes() == b.tobytes()
    which = [min(i, len(m) - 1) for i in bad]
    other = m.copy()
    other["contact_count"][which] = 7
    with pytest.raises(N.BepuError, match=f"manifold {min(which)} "):
        sp.update_manifolds(other)
    sp.close()
