"""The work a program has the solver do, as timed passes.

Every case is one of the workloads of this repository's benchmark and tests
(box piles, articulated chains, towers in batches, the dropped heap), driven
through `bepuphysics1_gb300.solver` as a C# engine or a batch of simulations
drives it: records go up once, a pass writes the state it starts from, steps,
and reads the results back into page-locked arrays.  A pass starts from the
same body state each time, so it does the same work however often it runs.

    frame    one engine frame: every body's state up, one step, every body's
             state and every manifold's impulses back (`step_state`)
    rollout  a snapshot restored (`update_bodies`, `update_manifolds`), `steps`
             steps on the device, the state read back (`download_state`)
    settle   frames of a heap whose pairs follow the broad phase:
             `update_pairs` and a step with the narrow phase
    broad    the overlapping pairs of the bodies as they lie (`broad_phase`)
    batch    many uneven scenes restored and advanced by one `batch_step`
"""
from __future__ import annotations

import math

import numpy as np
import torch

from bepuphysics1_gb300 import native as N
from bepuphysics1_gb300 import scenes
from bepuphysics1_gb300.solver import (Context, GpuSpace, batch_step, body_states, default_settings, islands_of,
                                       scene_ids, set_batch_threads)

DT = np.float32(1.0 / 60.0)


def listed():
    return [
        # The smallest scene an engine steps: eight boxes on the ground, a frame's latency.
        dict(name="frame_8", kind="frame", scene="packed", nx=2, ny=2, nz=2, iterations=10),
        # The 1,000-box pile (unit boxes at 1.05 m): one island, an ordinary game frame.
        dict(name="frame_1k", kind="frame", scene="packed", nx=10, ny=10, nz=10, iterations=10),
        # A larger packed frame with ragged extents: one island of 5,750 boxes.
        dict(name="frame_6k", kind="frame", scene="packed", nx=25, ny=10, nz=23, iterations=10),
        # The 65,536-box pile of separate columns, the benchmark's headline scene, rolled out.
        dict(name="rollout_64k", kind="rollout", scene="columns", nx=64, ny=16, nz=64, iterations=10, steps=10),
        # The same count packed at 1.05 m: one island of 65,536 boxes, 188,667 manifolds.
        dict(name="rollout_packed_64k", kind="rollout", scene="packed", nx=64, ny=16, nz=64, iterations=10, steps=4),
        # A level at rest: 4,096 columns of unit cubes as simulation islands, half of them asleep.
        dict(name="rollout_islands", kind="rollout", scene="cubes", nx=64, ny=16, nz=64, iterations=10, steps=10,
             asleep=0.5),
        # Ragdoll-like chains with limits: 8,192 chains of 16 capsules, 196,608 joints, 20,000 loose bodies.
        dict(name="chains_8k", kind="rollout", scene="chains", chains=8192, links=16, loose=20000, iterations=15,
             steps=8, added=False),
        # Machines of mixed joint and motor types: chains whose joints are ten further types in turn.
        dict(name="chains_added", kind="rollout", scene="chains", chains=384, links=16, loose=1000, iterations=15,
             steps=16, added=True),
        # The 65,536-box pile with its contacts regenerated by the narrow phase every step.
        dict(name="collide_64k", kind="rollout", scene="collide", nx=64, ny=16, nz=64, iterations=10, steps=8),
        # The dropped heap while it settles: pairs, records and colouring follow the broad phase.
        dict(name="settle_64k", kind="settle", nx=64, ny=16, nz=64, iterations=10, steps=4, fallen=140),
        # The broad phase alone, as a program asks for the pairs of 65,536 boxes.
        dict(name="broad_64k", kind="broad", nx=64, ny=16, nz=64),
        # Many simulations side by side: 256 towers of 8 to 2,048 boxes and spheres, 128 steps a call,
        # at the setting the autotuner finds for this mix.
        dict(name="batch_256", kind="batch", scenes=256, low=8, high=2048, iterations=8, steps=128, tuned=True),
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _grid(rng, low, high):
    """Grid extents of about `low` to `high` boxes, mostly odd and uneven."""
    n = _log(rng, low, high)
    ny = rng.randint(2, max(2, min(16, int(n ** (1 / 3)) + 2)))
    nx = max(1, min(64, int(round(math.sqrt(n / ny) * rng.uniform(0.8, 1.25)))))
    return dict(nx=nx, ny=ny, nz=max(1, min(64, n // (nx * ny))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "columns", "packed", "cubes", "chains", "chains", "collide", "settle",
                       "broad", "batch"])
    iterations = rng.choice([4, 8, 10, 15])
    if kind == "frame":
        return dict(kind="frame", scene="packed", iterations=iterations, **_grid(rng, 8, 8192))
    if kind in ("columns", "collide"):
        return dict(kind="rollout", scene=kind, iterations=min(iterations, 10), steps=rng.randint(2, 8),
                    **_grid(rng, 64, 65536))
    if kind == "packed":
        return dict(kind="rollout", scene="packed", iterations=min(iterations, 10), steps=rng.randint(1, 4),
                    **_grid(rng, 512, 65536))
    if kind == "cubes":
        return dict(kind="rollout", scene="cubes", iterations=min(iterations, 10), steps=rng.randint(2, 10),
                    asleep=round(rng.random(), 3), **_grid(rng, 512, 65536))
    if kind == "chains":
        added = rng.random() < 0.5
        return dict(kind="rollout", scene="chains", chains=_log(rng, 3, 384 if added else 8192),
                    links=rng.randint(3, 16), loose=_log(rng, 10, 1000 if added else 20000), iterations=iterations,
                    steps=rng.randint(2, 8), added=added)
    if kind == "settle":
        return dict(kind="settle", iterations=min(iterations, 10), steps=rng.randint(1, 4),
                    fallen=rng.randint(20, 140), **_grid(rng, 512, 65536))
    if kind == "broad":
        return dict(kind="broad", **_grid(rng, 64, 65536))
    return dict(kind="batch", scenes=_log(rng, 8, 256), low=8, high=rng.choice([64, 512, 2048]), iterations=8,
                steps=rng.randint(8, 64), tuned=rng.random() < 0.5)


# ------------------------------------------------------------------- inputs --
def _records(case, seed):
    """(bodies, manifolds, joints, shapes) of a one-scene case from the seeded scene source."""
    scene = case.get("scene")
    if scene == "chains":
        b, m, j = scenes.make_chain(chains=case["chains"], links=case["links"], loose_bodies=case["loose"],
                                    seed=seed + 3)
        return b, m, scenes.with_added_joint_types(b, j) if case["added"] else j, None
    grid = dict(nx=case["nx"], ny=case["ny"], nz=case["nz"], seed=seed + 11)
    if scene == "packed":
        b, m, j = scenes.make_pile(spacing=1.05, size_min=1.0, size_max=1.0, jitter=0.05, friction_min=0.6,
                                   friction_max=0.6, **grid)
        b["velocity_time_below_limit"][b["is_dynamic"] == 0] = 1.0  # the ground has been at rest for some steps
        return b, m, j, None
    if scene == "cubes":
        b, m, j = scenes.make_pile(spacing=2.0, size_min=1.0, size_max=1.0, jitter=0.02, friction_min=0.6,
                                   friction_max=0.6, ground_size=(140.0, 1.0, 140.0), **grid)
        b["activity"] &= ~np.uint32(N.BODY_ALWAYS_ACTIVE)
        return b, m, j, None
    if scene == "columns":
        return (*scenes.pile_64k(**grid), None)
    return scenes.pile_64k_collide(**grid)


def _scattered(case, seed):
    """(bodies, shapes): the boxes of the pile's columns knocked about, moving, on the ground."""
    b, _, _, shapes = scenes.pile_64k_collide(nx=case["nx"], ny=case["ny"], nz=case["nz"], seed=seed + 11)
    rng = np.random.default_rng(seed)
    moving = b["is_dynamic"] != 0
    b["position"][moving] += rng.uniform(-0.6, 0.6, (int(moving.sum()), 3)).astype(np.float32)
    b["linear_velocity"][moving] = rng.normal(0, 2, (int(moving.sum()), 3)).astype(np.float32)
    return b, shapes


def _pinned(records):
    """The records in a page-locked array of their own."""
    raw = torch.empty(max(records.nbytes, 1), dtype=torch.uint8, pin_memory=True).numpy()[:records.nbytes]
    out = raw.view(records.dtype)
    out[:] = records
    return out


def _state_arrays(bodies, manifolds):
    return _pinned(np.zeros(bodies, N.BODY_STATE_DTYPE)), _pinned(np.zeros(manifolds, N.MANIFOLD_STATE_DTYPE))


def _capacity(case):
    """Room for a scene's manifolds, whatever its seed (their number varies with the boxes' jitter)."""
    if case["scene"] == "chains":
        return 2 * case["loose"] + case["chains"] * case["links"]
    return (4 if case["scene"] == "packed" else 2) * case["nx"] * case["ny"] * case["nz"]


def _outputs(bodies, manifolds=None):
    """Every field of the state arrays (views: they follow the arrays' contents)."""
    out = {"body": {k: bodies[k] for k in bodies.dtype.names}}
    if manifolds is not None:
        out["manifold"] = {k: manifolds[k] for k in manifolds.dtype.names if k != "reserved"}
    return out


def _context(case):
    settings = default_settings()
    settings["iteration_limit"] = case.get("iterations", 10)
    return Context(0, settings)


def prepare(case, seed):
    ctx = _context(case)
    s = {"kind": case["kind"], "ctx": ctx, "steps": case.get("steps", 1)}
    if case["kind"] == "batch":
        sizes = scenes.batch_body_counts(case["scenes"], case["low"], case["high"], 4)
        recs = [scenes.make_tower(int(k), seed=(seed + 4) * 100003 + i)[:2] for i, k in enumerate(sizes)]
        how = dict(group_policy=(1, 1024, 4096, 128, 0), smem_budget=100 * 1024) if case["tuned"] else {}
        set_batch_threads(ctx, 128 if case["tuned"] else 0)
        s["spaces"] = [GpuSpace(ctx, b, m, **how) for b, m in recs]
        s["ids"] = scene_ids(s["spaces"])
        for _ in range(3):  # the snapshot is of running simulations
            for space in s["spaces"]:
                space.step(DT, N.STEP_ALL)
        start = _pinned(np.concatenate([sp.download_bodies(b.copy()) for sp, (b, _) in zip(s["spaces"], recs)]))
        out, _ = _state_arrays(len(start), 0)
        at = np.concatenate([[0], np.cumsum([len(b) for b, _ in recs])])
        s["start"] = [start[at[i]:at[i + 1]] for i in range(len(recs))]
        s["end"] = [out[at[i]:at[i + 1]] for i in range(len(recs))]
        s["out"] = _outputs(out)
        return s
    if case["kind"] == "settle":
        grid = dict(nx=case["nx"], ny=case["ny"], nz=case["nz"], seed=seed + 11)
        b, shapes, friction = scenes.dropped_pile(**grid)
        space = GpuSpace(ctx, b, None, capacity=(len(b), 8 * len(b) + 64, 0), shapes=shapes)
        space.set_materials(np.stack([friction, friction, np.zeros_like(friction)], 1))
        for _ in range(case["fallen"]):
            space.update_pairs(DT)
            space.step(DT, N.STEP_ALL)
        s["space"], s["start"] = space, _pinned(space.download_bodies(b.copy()))
        s["bodies"], _ = _state_arrays(len(b), 0)
        s["out"] = _outputs(s["bodies"])
        return s
    if case["kind"] == "broad":
        b, shapes = _scattered(case, seed)
        s["space"] = GpuSpace(ctx, b, None, shapes=shapes)
        s["pairs"] = np.zeros((8 * len(b), 2), np.int32)
        return s
    b, m, j, shapes = _records(case, seed)
    space = s["space"] = GpuSpace(ctx, b, m, j, shapes=shapes)
    s["bodies"], manifolds = _state_arrays(len(b), _capacity(case))
    s["manifolds"] = manifolds[:len(m)]
    s["out"] = _outputs(s["bodies"], manifolds)
    if case["kind"] == "frame":
        s["start"] = body_states(b)
        return s
    if case["scene"] == "cubes":
        isl = islands_of(b, m)
        count = int(isl.max(initial=-1)) + 1
        flags = np.full(count, N.ISLAND_ACTIVE | N.ISLAND_ALLOW_DEACTIVATION, np.uint32)
        sleeping = np.random.default_rng(seed).random(count) < case["asleep"]
        flags[sleeping] = N.ISLAND_ALLOW_DEACTIVATION
        space.set_islands(isl, flags)
    for _ in range(3):  # the snapshot is of a running simulation: warm impulses, contacts with ids
        space.step(DT, N.STEP_ALL)
    s["start"] = _pinned(space.download_bodies(b.copy()))
    s["records"] = _pinned(space.download_constraints()[0])
    return s


def run(s):
    kind = s["kind"]
    if kind == "frame":
        np.copyto(s["bodies"], s["start"])  # the engine writes its bodies' state
        s["space"].step_state(s["bodies"], s["manifolds"], DT)
    elif kind == "rollout":
        space = s["space"]
        space.update_bodies(s["start"])
        space.update_manifolds(s["records"])
        for _ in range(s["steps"]):
            space.step(DT, N.STEP_ALL)
        space.download_state(s["bodies"], s["manifolds"])
    elif kind == "settle":
        space = s["space"]
        space.update_bodies(s["start"])
        for _ in range(s["steps"]):
            count = space.update_pairs(DT)
            space.step(DT, N.STEP_ALL)
        space.download_state(s["bodies"], None)
        return {**s["out"], "pairs": count}
    elif kind == "broad":
        pairs = s["space"].broad_phase(DT)
        s["pairs"][:len(pairs)] = pairs  # into the program's own list
        return s["pairs"], len(pairs)
    else:
        for space, start in zip(s["spaces"], s["start"]):
            space.update_bodies(start)
        batch_step(s["ctx"], s["ids"], DT, s["steps"])
        for space, end in zip(s["spaces"], s["end"]):
            space.download_state(end, None)
    return s["out"]


# --------------------------------------------------------------------- work --
_BODY, _MANIFOLD, _JOINT = N.BODY_DTYPE.itemsize, N.MANIFOLD_DTYPE.itemsize, N.JOINT_DTYPE.itemsize
_BODY_OUT, _MANIFOLD_OUT = N.BODY_STATE_DTYPE.itemsize, N.MANIFOLD_STATE_DTYPE.itemsize


def _step_flops(contacts, manifolds, joints, bodies, iterations):
    """Arithmetic of one step: a contact's penetration child about 90 operations a visit, a manifold's
    friction children 250, a joint 300; the prestep about 150 a contact and 500 a manifold or joint."""
    visits = iterations + 1
    return (visits * (90 * contacts + 250 * manifolds + 300 * joints) + 150 * contacts +
            500 * (manifolds + joints) + 250 * bodies)


def work(case):
    k, it = case.get("steps", 1), case.get("iterations", 10)
    if case["kind"] == "batch":
        b = int(scenes.batch_body_counts(case["scenes"], case["low"], case["high"], 4).sum())
        return {"bytes": b * (_BODY + _BODY_OUT + _MANIFOLD), "flops": k * _step_flops(4 * b, b, 0, b, it)}
    if case["kind"] == "broad":
        n = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": n * (64 + 16 + 8), "flops": 100 * n}
    if case["kind"] == "settle":
        n = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": n * (_BODY + _BODY_OUT + 16), "flops": k * (_step_flops(8 * n, 2 * n, 0, n, it) + 4000 * n)}
    b, m, j, _ = _records(case, 0)
    contacts = 4 * len(m) if case["scene"] == "collide" else scenes.contact_count(m)
    awake = 1.0 - case.get("asleep", 0.0)
    flops = k * awake * _step_flops(contacts, len(m), len(j), len(b), it)
    if case["kind"] == "frame":
        return {"bytes": len(b) * (2 * _BODY_OUT + 64) + len(m) * (_MANIFOLD + _MANIFOLD_OUT), "flops": flops}
    if case["scene"] == "collide":
        flops += k * 3000 * len(m)
    return {"bytes": len(b) * (_BODY + _BODY_OUT) + len(m) * (_MANIFOLD + _MANIFOLD_OUT) + len(j) * _JOINT,
            "flops": flops}


# -------------------------------------------------------------------- exact --
def exact(case, seed):
    """A frame in 64 bits.  The other kinds run for seconds to minutes that way (10 to 128 steps of up to
    200,000 constraints, joints, clipping), and small differences grow from step to step in a pile."""
    if case["kind"] != "frame" or case["nx"] * case["ny"] * case["nz"] > 8192:
        return None
    b, m, _, _ = _records(case, seed)
    out = _frame64(b, m, case["iterations"])
    spare = _capacity(case) - len(m)
    out["manifold"] = {k: None if x is None else np.concatenate([x, np.zeros((spare,) + x.shape[1:])])
                       for k, x in out["manifold"].items()}
    return out


def _dot(a, b):
    return np.einsum("...i,...i->...", a, b)


def _rotation(q):
    """Row-vector rotation matrices (world = local @ R)."""
    x, y, z, w = q.T
    r = np.empty((len(q), 3, 3))
    r[:, 0] = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y + z * w), 2 * (x * z - y * w)], 1)
    r[:, 1] = np.stack([2 * (x * y - z * w), 1 - 2 * (x * x + z * z), 2 * (y * z + x * w)], 1)
    r[:, 2] = np.stack([2 * (x * z + y * w), 2 * (y * z - x * w), 1 - 2 * (x * x + y * y)], 1)
    return r


def _colours(a, b, dynamic):
    """Each manifold the smallest colour free at its dynamic bodies, in list order."""
    used = [0] * len(dynamic)
    out = np.empty(len(a), np.int64)
    for i, (x, y) in enumerate(zip(a.tolist(), b.tolist())):
        taken = (used[x] if dynamic[x] else 0) | (used[y] if dynamic[y] else 0)
        bit = ~taken & (taken + 1)
        out[i] = bit.bit_length() - 1
        if dynamic[x]:
            used[x] |= bit
        if dynamic[y]:
            used[y] |= bit
    return out


def _frame64(body, man, iterations):
    """Candidacy, contact refresh, forces, prestep, warm start, the colour sweeps and the position update
    of a pile of convex manifolds, in float64."""
    f8 = np.float64
    dt = f8(DT)
    dyn = body["is_dynamic"] != 0
    pos, q = body["position"].astype(f8), body["orientation"].astype(f8)
    v, w = body["linear_velocity"].astype(f8), body["angular_velocity"].astype(f8)
    inv_mass = np.where(dyn, body["inverse_mass"], 0).astype(f8)
    # candidacy
    speed = _dot(v, v) + _dot(w, w)
    below, activity = body["velocity_time_below_limit"].astype(f8), body["activity"]
    limit2 = f8(np.float32(.26)) ** 2
    candidate = dyn & (activity & N.BODY_DEACTIVATION_CANDIDATE != 0)
    always = activity & N.BODY_ALWAYS_ACTIVE != 0
    slowing = speed <= body["previous_velocity"]
    t = np.where(speed < limit2, below + dt, 0.0)
    t = np.where(always | (candidate & (t <= 1.0)), 0.0, t)
    still = ~dyn & (speed == 0) & ~always
    kin = np.where(still, np.where(below == 0, 1.0, np.where(below < 0, 0.0, below)), -1.0)
    active = dyn | (below <= 0)
    time_below = np.where(active, np.where(dyn, t, kin), below)
    slowing = np.where(active, slowing, activity & N.BODY_SLOWING != 0)
    # refresh
    a, b = man["body_a"], man["body_b"]
    c, rows = man["contacts"], np.arange(len(man))
    live = np.arange(4)[None, :] < man["contact_count"][:, None]
    rot = _rotation(q)
    wa = np.einsum("mki,mij->mkj", c["local_offset_a"].astype(f8), rot[a]) + pos[a][:, None]
    wb = np.einsum("mki,mij->mkj", c["local_offset_b"].astype(f8), rot[b]) + pos[b][:, None]
    n = c["normal"].astype(f8)
    ab = wb - wa
    along = _dot(ab, n)
    drift = ab - n * along[..., None]
    depth = c["base_penetration_depth"].astype(f8) - along
    keep = live & (_dot(drift, drift) <= f8(np.float32(.01))) & (depth >= -f8(np.float32(.1)))
    order = np.argsort(~keep, axis=1, kind="stable")
    pick = lambda x: np.take_along_axis(x, order.reshape(order.shape + (1,) * (x.ndim - 2)), axis=1)  # noqa: E731
    point, n, depth = pick((wa + wb) * .5), pick(n), pick(depth)
    acc = np.where(np.sort(~keep, axis=1), 0.0, pick(c["penetration_impulse"].astype(f8)))
    keep = np.sort(~keep, axis=1) == 0
    count = keep.sum(1)
    some = count > 0
    # forces
    v[dyn] += np.array([0, np.float32(-9.81), 0], f8) * dt
    lin, ang = body["linear_damping"].astype(f8), body["angular_damping"].astype(f8)
    energy = _dot(v, v) + _dot(w, w)
    boosted = (dyn & (activity & N.BODY_NO_STABILIZATION == 0) & (slowing | (time_below > 1.0)) & (energy < limit2))
    boost = np.where(boosted, 1 - np.sqrt(energy) / (2 * f8(np.float32(.26))), 0.0)
    lin, ang = lin + boost * (1 - lin), ang + boost * (1 - ang)
    v[dyn] *= (np.clip(1 - lin, 0, 1) ** dt)[dyn, None]
    w[dyn] *= (np.clip(1 - ang, 0, 1) ** dt)[dyn, None]
    local = np.where(dyn[:, None], body["local_inverse_inertia"], 0).astype(f8).reshape(-1, 3, 3)
    inertia = np.einsum("bki,bkl,blj->bij", rot, local, rot)
    turn = lambda k, x: np.einsum("mi,mij->mj", x, inertia[k])  # noqa: E731
    # prestep
    rate = 1 / dt
    lin_a = -n
    pen_a = np.cross(point - pos[a][:, None], lin_a)
    pen_b = np.cross(lin_a, point - pos[b][:, None])
    mass = (np.einsum("mki,mij,mkj->mk", pen_a, inertia[a], pen_a) +
            np.einsum("mki,mij,mkj->mk", pen_b, inertia[b], pen_b) + (inv_mass[a] + inv_mass[b])[:, None])
    soft = f8(np.float32(.001)) * mass * rate
    with np.errstate(divide="ignore", invalid="ignore"):
        to_impulse = -1 / (soft + mass)
    bias = np.where(depth >= 0, np.minimum(np.maximum(0, depth - f8(np.float32(.01))) * f8(np.float32(.2)) * rate, 2.0),
                    depth * rate)
    kinetic, static = man["kinetic_friction"].astype(f8), man["static_friction"].astype(f8)
    centre = (point * keep[..., None]).sum(1) / np.maximum(count, 1)[:, None]
    ra, rb = centre - pos[a], centre - pos[b]
    rel = v[a] + np.cross(w[a], ra) - v[b] - np.cross(w[b], rb)
    n0 = n[:, 0]
    rel = rel - n0 * _dot(rel, n0)[:, None]
    length2 = _dot(rel, rel)
    moving = length2 > 1e-7
    length = np.sqrt(np.where(moving, length2, 1.0))
    axis1 = man["sliding_axis"].astype(f8)
    fresh = np.cross(n0, np.array([1.0, 0, 0]))
    flat = _dot(fresh, fresh) <= 1e-7
    fresh[flat] = np.cross(n0[flat], np.array([0, 1.0, 0]))
    fresh /= np.maximum(np.linalg.norm(fresh, axis=1), 1e-30)[:, None]
    unset = ~moving & ~axis1.any(1)
    axis1 = np.where(moving[:, None], rel / length[:, None], np.where(unset[:, None], fresh, axis1))
    axis1 = np.where(some[:, None], axis1, man["sliding_axis"])
    friction = np.where(moving & (length > f8(np.float32(.2))), kinetic, static)
    axes = np.stack([axis1, np.cross(axis1, n0)], 1)
    slide_a, slide_b = np.cross(ra[:, None], axes), np.cross(axes, rb[:, None])
    k = -(np.einsum("mki,mij,mlj->mkl", slide_a, inertia[a], slide_a) +
          np.einsum("mki,mij,mlj->mkl", slide_b, inertia[b], slide_b) +
          (inv_mass[a] + inv_mass[b])[:, None, None] * np.eye(2))
    k[~some] = np.eye(2)
    k = np.linalg.inv(k)
    with np.errstate(divide="ignore", invalid="ignore"):
        twist_mass = -1 / (_dot(turn(a, n0), n0) + _dot(turn(b, n0), n0) + inv_mass[a] + inv_mass[b])
    spin = _dot(w[a] - w[b], n0)
    twist_friction = np.where((np.abs(spin) > f8(np.float32(.2))) | (np.abs(rel).sum(1) > f8(np.float32(.2))), kinetic,
                              static)
    lever = np.where(keep, np.linalg.norm(point - centre[:, None], axis=2), 0.0)
    slide = np.where(some[:, None], man["sliding_impulse"], 0).astype(f8)
    twist = np.where(some, man["twist_impulse"], 0).astype(f8)

    def apply(i, impulse, turn_a, turn_b):
        x, y = a[i], b[i]
        v[x] += impulse * inv_mass[x, None]
        w[x] += turn(x, turn_a)
        v[y] -= impulse * inv_mass[y, None]
        w[y] += turn(y, turn_b)

    colour = _colours(a, b, dyn)
    groups = [rows[colour == k] for k in range(int(colour.max(initial=-1)) + 1)]
    for g in groups:  # warm start
        for k4 in range(4):
            i = g[keep[g, k4]]
            p = acc[i, k4, None]
            apply(i, p * lin_a[i, k4], p * pen_a[i, k4], p * pen_b[i, k4])
        i = g[some[g]]
        on = lambda x: np.einsum("mk,mki->mi", slide[i], x[i])  # noqa: E731
        apply(i, on(axes), on(slide_a), on(slide_b))
        w[a[i]] += turn(a[i], twist[i, None] * n0[i])
        w[b[i]] -= turn(b[i], twist[i, None] * n0[i])
    # sweeps; a child with two impulses below the minimum in a row stops for the step
    least = f8(np.float32(.001))
    on_child = np.concatenate([keep, some[:, None], some[:, None]], 1)
    zeros = np.zeros((len(man), 6), np.int64)

    def account(i, child, size):
        small = size < least
        zeros[i, child] = np.where(small, zeros[i, child] + 1, 0)
        on_child[i, child] = zeros[i, child] <= 1

    for _ in range(iterations):
        for g in groups:
            for k4 in range(4):
                i = g[on_child[g, k4]]
                x, y = a[i], b[i]
                rv = (_dot(v[x] - v[y], lin_a[i, k4]) + _dot(w[x], pen_a[i, k4]) + _dot(w[y], pen_b[i, k4]))
                before = acc[i, k4]
                acc[i, k4] = np.maximum(0, before + (rv - bias[i, k4] + soft[i, k4] * before) * to_impulse[i, k4])
                p = (acc[i, k4] - before)[:, None]
                apply(i, p * lin_a[i, k4], p * pen_a[i, k4], p * pen_b[i, k4])
                account(i, k4, np.abs(p[:, 0]))
            i = g[on_child[g, 4]]
            x, y = a[i], b[i]
            dv = v[x] + np.cross(w[x], ra[i]) - v[y] - np.cross(w[y], rb[i])
            before = slide[i]
            now = before + np.einsum("mk,mkl->ml", np.einsum("mi,mki->mk", dv, axes[i]), k[i])
            most = (acc[i] * keep[i]).sum(1) * friction[i]
            size = np.linalg.norm(now, axis=1)
            now = np.where((size > most)[:, None], now * (most / np.maximum(size, 1e-300))[:, None], now)
            slide[i] = now
            p = now - before
            on = lambda z: np.einsum("mk,mki->mi", p, z[i])  # noqa: E731
            apply(i, on(axes), on(slide_a), on(slide_b))
            account(i, 4, np.abs(p).sum(1))
            i = g[on_child[g, 5]]
            x, y = a[i], b[i]
            most = (lever[i] * acc[i]).sum(1) * twist_friction[i]
            before = twist[i]
            twist[i] = np.clip(before + _dot(w[x] - w[y], n0[i]) * twist_mass[i], -most, most)
            p = (twist[i] - before)[:, None] * n0[i]
            w[x] += turn(x, p)
            w[y] -= turn(y, p)
            account(i, 5, np.abs(twist[i] - before))
    # positions (a kinematic body moves while its time flag is <= 0; here all of them stand still)
    half = w * (dt * .5)
    x, y, z, s = q.T
    hx, hy, hz = half.T
    q = q + np.stack([hx * s + hy * z - hz * y, hy * s + hz * x - hx * z, hz * s + hx * y - hy * x,
                      -hx * x - hy * y - hz * z], 1)
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    pos = pos + v * dt
    return {"body": {"position": pos, "orientation": q, "linear_velocity": v, "angular_velocity": w,
                     "activity": None, "previous_velocity": np.where(active, speed, body["previous_velocity"]),
                     "velocity_time_below_limit": time_below},
            "manifold": {"contact_count": None, "contact_id": None, "penetration_impulse": np.where(keep, acc, 0),
                         "sliding_impulse": slide, "twist_impulse": twist, "sliding_axis": axis1,
                         "friction_impulse": None}}
