"""The work that a program has the library do, as cases that can be timed.

Three kinds of call make up a program that steps rigid bodies on the GPU, and each appears from its
smallest to its largest size:

- the world step: a game's one small world, a heap in one island, thousands of small worlds as a
  learning loop steps them, ragdolls held by joints, every shape on a terrain mesh with continuous
  collision;
- queries against the bodies of a world between steps: rays, shape casts, overlap tests;
- the gradient of a rollout (a forward pass with checkpoints, and the backward pass).

Scenes are laid out at rest from the seed alone: stacks and rows of bodies that touch within the
penetration slop, some still tumbling, as a settled scene has them.  Every pass starts from the same
state rows, so a pass costs the same however many came before; sleeping is off for the same reason.
A state takes a few steps when it is prepared, so that a pass meets a filled contact cache, as in any
program but for its first frame.

A step's results have no value in plain 64-bit numpy short of a second engine, so ``exact`` gives the
ray fractions in the scenes of boxes and spheres, where a ray meets closed forms.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from crashcat_gb300 import _lib, scenes
from crashcat_gb300.world import GpuWorld, standard_settings


def listed():
    return [
        # a game's frame: one small world, state in and out every frame
        {"name": "frame_32", "kind": "step", "scene": "stacks", "worlds": 1, "low": 32, "high": 32,
         "hz": 60, "velocity": 10, "position": 2},
        # a learning environment of a few dozen worlds, four physics steps for each action
        {"name": "env_48_worlds", "kind": "substeps", "scene": "stacks", "worlds": 48, "low": 8, "high": 512,
         "hz": 120, "velocity": 8, "position": 2, "steps": 4},
        # the batched workload of the benchmark: 4,096 uneven worlds, state in and out every step
        {"name": "step_4096_worlds", "kind": "step", "scene": "stacks", "worlds": 4096, "low": 8, "high": 512,
         "hz": 120, "velocity": 8, "position": 2},
        # the cube heap: a thousand boxes in contact in one world
        {"name": "heap_1000", "kind": "step", "scene": "heap", "side": 10, "hz": 60, "velocity": 10, "position": 2},
        # a heap large enough for its one island to take the whole GPU
        {"name": "heap_4096", "kind": "step", "scene": "heap", "side": 16, "hz": 60, "velocity": 10, "position": 2},
        # ragdolls: hinges and swing-twist joints with limits
        {"name": "ragdolls_500", "kind": "step", "scene": "ragdolls", "ragdolls": 500, "hz": 60, "velocity": 12,
         "position": 4},
        # every convex shape on a terrain mesh, a fifth of them fast with continuous collision
        {"name": "terrain_6000", "kind": "step", "scene": "terrain", "bodies": 6000, "cells": 160, "hz": 60,
         "velocity": 8, "position": 2},
        # a frame's lines of sight: a few hundred rays in one small world, host buffers
        {"name": "rays_256", "kind": "rays", "scene": "stacks", "worlds": 1, "low": 200, "high": 200, "rays": 256,
         "device": False},
        # a sensor sweep: a million rays onto a terrain with bodies, buffers on the GPU
        {"name": "rays_1m", "kind": "rays", "scene": "terrain", "bodies": 6000, "cells": 160, "rays": 1 << 20,
         "device": True},
        # character and camera sweeps in bulk
        {"name": "casts_16k", "kind": "casts", "scene": "terrain", "bodies": 6000, "cells": 160, "casts": 1 << 14},
        # area queries: every body that a shape overlaps, and points inside bodies
        {"name": "overlaps_2k", "kind": "overlaps", "scene": "stacks", "worlds": 16, "low": 100, "high": 400,
         "shapes": 2048, "points": 8192},
        # the gradient of a rollout: sliding boxes, a checkpoint every ten steps
        {"name": "grad_128_worlds", "kind": "grad", "worlds": 128, "boxes": 64, "steps": 20},
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["stacks", "stacks", "env", "heap", "ragdolls", "terrain", "rays", "rays_mesh", "casts",
                       "overlaps", "grad"])
    hz, velocity, position = rng.choice([60, 120]), rng.randint(6, 12), rng.randint(1, 4)
    step = {"kind": "step", "hz": hz, "velocity": velocity, "position": position}
    if kind == "stacks":
        low = spread(8, 64)
        return {**step, "scene": "stacks", "worlds": spread(1, 3000), "low": low, "high": low * rng.randint(1, 8)}
    if kind == "env":
        low = spread(8, 64)
        return {**step, "kind": "substeps", "scene": "stacks", "worlds": spread(2, 256), "low": low,
                "high": low * rng.randint(1, 8), "steps": rng.randint(2, 4)}
    if kind == "heap":
        return {**step, "scene": "heap", "side": rng.randint(3, 15)}
    if kind == "ragdolls":
        return {**step, "scene": "ragdolls", "ragdolls": spread(4, 480)}
    bodies = spread(60, 5500)
    cells = max(16, int(2.0 * math.sqrt(bodies)) + rng.randint(0, 5))
    if kind == "terrain":
        return {**step, "scene": "terrain", "bodies": bodies, "cells": cells}
    if kind == "rays":
        low = spread(20, 200)
        return {"kind": "rays", "scene": "stacks", "worlds": spread(1, 64), "low": low, "high": low * 2,
                "rays": spread(100, 400000), "device": rng.random() < 0.5}
    if kind == "rays_mesh":
        return {"kind": "rays", "scene": "terrain", "bodies": bodies, "cells": cells, "rays": spread(100, 1000000),
                "device": rng.random() < 0.5}
    if kind == "casts":
        return {"kind": "casts", "scene": "terrain", "bodies": bodies, "cells": cells, "casts": spread(50, 16000)}
    if kind == "overlaps":
        low = spread(20, 200)
        return {"kind": "overlaps", "scene": "stacks", "worlds": spread(1, 24), "low": low, "high": low * 2,
                "shapes": spread(32, 2000), "points": spread(32, 8000)}
    return {"kind": "grad", "worlds": spread(2, 120), "boxes": rng.randint(8, 64), "steps": rng.randint(5, 20)}


# ---------------------------------------------------------------------------
# scenes at rest
# ---------------------------------------------------------------------------
def _quat_mul(a, b):
    ax, ay, az, aw = np.moveaxis(a, -1, 0)
    bx, by, bz, bw = np.moveaxis(b, -1, 0)
    return np.stack([ax * bw + aw * bx + ay * bz - az * by, ay * bw + aw * by + az * bx - ax * bz,
                     az * bw + aw * bz + ax * by - ay * bx, aw * bw - ax * bx - ay * by - az * bz], -1)


def _small_turns(rng, n, angle):
    """Unit quaternions of rotations by up to about ``angle`` about random axes."""
    v = rng.uniform(-0.5 * angle, 0.5 * angle, (n, 3))
    q = np.concatenate([v, np.ones((n, 1))], 1)
    return q / np.linalg.norm(q, axis=1, keepdims=True)


def _lowest(he, q):
    """How far a box's lowest corner lies below its centre."""
    x, y, z, w = np.moveaxis(q, -1, 0)
    row = np.stack([2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)], -1)
    return (np.abs(row) * he).sum(-1)


def _stacks(seed, worlds, low, high):
    """Worlds of boxes and spheres on their own floors: single bodies, stacks of two to five, rows of
    stacks that touch, one body in five lying as it fell and still moving."""
    rng = np.random.default_rng(4)  # how many bodies each world holds goes with the case, not with the seed
    counts = np.clip(np.rint(np.exp(rng.uniform(math.log(low), math.log(high), worlds))).astype(np.int64), low, high)
    crowded = rng.uniform(0.1, 0.9, worlds)  # how many of a world's stacks touch the next one
    rng = np.random.default_rng(seed)
    n = int(counts.sum())
    world = np.repeat(np.arange(worlds), counts)
    first = np.concatenate([[0], np.cumsum(counts)[:-1]])
    he = rng.uniform(0.2, 0.8, (n, 3))
    radius = rng.uniform(0.2, 0.6, n)
    sphere = rng.random(n) < 0.5
    loose = rng.random(n) < 0.2
    # a body starts a new stack unless it sits on the one before it
    on_top = (rng.random(n) < 0.4) & ~loose
    on_top[first] = False
    below = np.concatenate([[False], (~sphere & ~loose)[:-1]])
    on_top &= below
    level = np.zeros(n, np.int64)
    for _ in range(4):  # stacks are at most five high
        prev = np.concatenate([[0], level[:-1]])
        level = np.where(on_top, prev + 1, 0)
    on_top &= level < 5
    stack = np.cumsum(~on_top) - 1
    start = np.flatnonzero(~on_top)
    q = _small_turns(rng, n, 0.004)
    tumbled = scenes.random_quaternions(rng, n).astype(np.float64)
    q[loose] = tumbled[loose]
    half = np.where(sphere, radius, np.where(loose, _lowest(he, q), he[:, 1]))
    # heights: each body 4 to 16 mm into what carries it
    sink = rng.uniform(0.004, 0.016, n)
    rise = 2 * half - sink
    total = np.cumsum(rise)
    y = total - total[start][stack] + rise[start][stack] - half
    # stacks in rows of 24 along x, each clear of the one before it or 2 to 8 mm into it
    reach = np.where(sphere, radius, np.where(loose, np.linalg.norm(he, axis=1), he[:, 0]))
    wide = np.maximum.reduceat(reach, start)
    s_world = world[start]
    s_first = np.searchsorted(s_world, np.arange(worlds))
    nth = np.arange(len(start)) - s_first[s_world]
    gap = np.where(rng.random(len(start)) < crowded[s_world], rng.uniform(-0.008, -0.002, len(start)),
                   rng.uniform(0.06, 0.4, len(start)))
    run = np.cumsum(2 * wide + gap)
    row_start = np.maximum.accumulate(np.where(nth % 24 == 0, np.arange(len(start)), 0))
    x = run - run[row_start] + wide[row_start] - wide - 24.0
    z = (nth // 24) * 2.1 - 24.0
    pos = np.stack([x[stack], y, z[stack]], 1)
    b = scenes.blank_bodies(n + worlds)
    at = np.arange(n) + world + 1
    floors = first + np.arange(worlds)
    b["shape_type"][at] = np.where(sphere, _lib.SHAPE_SPHERE, _lib.SHAPE_BOX)
    b["shape_params"][at, 0] = np.where(sphere, radius, he[:, 0])
    b["shape_params"][at, 1] = np.where(sphere, 0.0, he[:, 1])
    b["shape_params"][at, 2] = np.where(sphere, 0.0, he[:, 2])
    b["shape_params"][at, 3] = np.where(sphere, 0.0, scenes.DEFAULT_CONVEX_RADIUS)
    b["position"][at] = pos
    b["quaternion"][at] = q
    b["world"][at] = world
    b["friction"][at] = 0.5
    b["linear_velocity"][at] = rng.normal(0, 1, (n, 3)) * np.where(loose, 0.4, 0.01)[:, None]
    b["angular_velocity"][at] = rng.normal(0, 1, (n, 3)) * np.where(loose, 0.8, 0.01)[:, None]
    scenes.set_box(b, floors, (30.0, 0.5, 30.0))
    b["motion_type"][floors] = _lib.STATIC
    b["object_layer"][floors] = scenes.LAYER_NOT_MOVING
    b["position"][floors] = (0.0, -0.5, 0.0)
    b["friction"][floors] = 0.5
    b["world"][floors] = np.arange(worlds)
    return b


def _heap(seed, side):
    """side^3 unit boxes packed on a floor, each a few millimetres into the one below and within the
    contact distance of its neighbours: one island."""
    rng = np.random.default_rng(seed)
    n = side ** 3
    b = scenes.blank_bodies(n + 1)
    scenes.static_floor(b, 0, half=(100.0, 0.5, 100.0), friction=0.5)
    idx = np.arange(1, n + 1)
    scenes.set_box(b, idx, (0.5, 0.5, 0.5))
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3).astype(np.float64)
    pos = g * (1.004, 0.994, 1.004) + (-side / 2, 0.495, -side / 2)
    pos += rng.uniform(-1, 1, (n, 3)) * (0.006, 0.002, 0.006)
    b["position"][idx] = pos
    b["quaternion"][idx] = _small_turns(rng, n, 0.004)
    b["linear_velocity"][idx] = rng.normal(0, 0.02, (n, 3))
    b["friction"][idx] = 0.5
    return b


def _terrain(seed, bodies, cells):
    """Spheres, boxes, capsules, cylinders and hulls lying on a rolling heightfield, a fifth of them in
    the air at 20 to 60 m/s with continuous collision.  Returns (bodies, hull points, mesh)."""
    rng = np.random.default_rng(seed)
    verts, tris = scenes.heightfield(cells, 1.0, 4.0, seed)
    n = bodies
    b = scenes.blank_bodies(n + 1)
    b["shape_type"][0] = _lib.SHAPE_TRIANGLE_MESH
    b["motion_type"][0] = _lib.STATIC
    b["object_layer"][0] = scenes.LAYER_NOT_MOVING
    b["friction"][0] = 0.5
    kind = rng.integers(0, 5, n)
    he = rng.uniform(0.2, 0.8, (n, 3))
    r = rng.uniform(0.2, 0.5, n)
    h = rng.uniform(0.3, 0.8, n)
    num_hulls = max(1, min(256, n // 8))  # a program's props share their shapes
    hulls = [scenes.ellipsoid_hull_points(rng, int(rng.integers(16, 33)), rng.uniform(0.3, 0.8, 3))
             for _ in range(num_hulls)]
    reach = np.zeros(n)
    for k, (make, args, out) in enumerate((
            (scenes.set_sphere, lambda s: (r[s],), lambda s: r[s]),
            (scenes.set_box, lambda s: (he[s],), lambda s: he[s].min(1)),
            (scenes.set_capsule, lambda s: (r[s], h[s]), lambda s: r[s]),
            (scenes.set_cylinder, lambda s: (h[s], r[s]), lambda s: np.minimum(r[s], h[s])),
            (None, None, None))):
        s = np.flatnonzero(kind == k)
        if make is not None:
            make(b, s + 1, *args(s))
            reach[s] = out(s)
        else:
            which = rng.integers(0, num_hulls, len(s))
            b["shape_type"][s + 1] = _lib.SHAPE_CONVEX_HULL
            b["shape_params"][s + 1] = 0.0
            b["shape_params"][s + 1, 0] = which
            reach[s] = np.array([np.linalg.norm(p, axis=1).min() for p in hulls])[which]
    # on a jittered grid over the terrain, each as high as its smallest reach above the nearest vertex
    side = int(math.ceil(math.sqrt(n)))
    pitch = 0.86 * cells / side
    cell = rng.permutation(side * side)[:n]
    x = (cell % side - (side - 1) / 2) * pitch + rng.uniform(-0.3, 0.3, n)
    z = (cell // side - (side - 1) / 2) * pitch + rng.uniform(-0.3, 0.3, n)
    grid = verts[:, 1].reshape(cells + 1, cells + 1)
    ground = grid[np.clip(np.rint(x + cells / 2).astype(int), 0, cells), np.clip(np.rint(z + cells / 2).astype(int), 0,
                                                                                cells)]
    fast = rng.random(n) < 0.2
    up = np.where(fast, rng.uniform(0.6, 4.0, n), rng.uniform(0.0, 0.1, n))
    b["position"][1:] = np.stack([x, ground + reach + up, z], 1)
    b["quaternion"][1:] = scenes.random_quaternions(rng, n)
    d = rng.normal(size=(n, 3))
    d[:, 1] = -np.abs(d[:, 1]) - 0.5
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    speed = np.where(fast, rng.uniform(20.0, 60.0, n), 0.3)
    b["linear_velocity"][1:] = d * speed[:, None]
    b["motion_quality"][1:] = np.where(fast, _lib.MOTION_LINEAR_CAST, _lib.MOTION_DISCRETE)
    b["friction"][1:] = 0.5
    return b, hulls, (verts, tris)


def _world(case, seed):
    """(world, body records) of the case's scene, every body added."""
    scene = case["scene"]
    sc, hulls, mesh = None, [], None
    if scene == "stacks":
        bodies = _stacks(seed, case["worlds"], case["low"], case["high"])
    elif scene == "heap":
        bodies = _heap(seed, case["side"])
    elif scene == "ragdolls":
        sc = scenes.ragdolls(case["ragdolls"], seed=seed, random_poses=False)
        bodies = sc.bodies
        bodies["position"][0, 1] += 1.7  # the floor comes up to the lowest layer's limbs
    else:
        bodies, hulls, mesh = _terrain(seed, case["bodies"], case["cells"])
    settings = standard_settings(velocity_iterations=case.get("velocity", 8),
                                 position_iterations=case.get("position", 2),
                                 num_worlds=case.get("worlds", 1), allow_sleeping=False)
    w = GpuWorld(settings, len(bodies))
    for points in hulls:
        w.add_convex_hull(points)
    if mesh is not None:
        w.add_triangle_mesh(*mesh)
    w.add_bodies(bodies)
    if sc is not None:
        w.set_skip_joint_pairs(True)
        w.add_hinges(sc.hinges)
        w.add_swing_twists(sc.swings)
    return w, bodies


def _pinned(shape):
    t = torch.zeros(shape, dtype=torch.float32, pin_memory=True)
    return t, t.numpy()


# ---------------------------------------------------------------------------
# queries
# ---------------------------------------------------------------------------
def _query_rows(case, seed, count):
    """Origins, unit directions, reach and world of ``count`` queries in the case's scene."""
    rng = np.random.default_rng(seed + 7)
    if case["scene"] == "stacks":
        origin = rng.uniform((-24.0, 0.1, -24.0), (4.0, 3.0, -14.0), (count, 3))
        d = rng.normal(size=(count, 3)) * (1.0, 0.35, 1.0)
        reach = rng.uniform(5.0, 40.0, count)
        world = rng.integers(0, case["worlds"], count)
    else:
        half = 0.43 * case["cells"]
        origin = rng.uniform((-half, 10.0, -half), (half, 30.0, half), (count, 3))
        d = rng.normal(size=(count, 3)) * 0.5
        d[:, 1] = -np.abs(d[:, 1]) - 0.5
        reach = rng.uniform(40.0, 100.0, count)
        world = np.zeros(count, np.int64)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return origin, d, reach, world


def _rays(case, seed):
    origin, d, reach, world = _query_rows(case, seed, case["rays"])
    rays = np.zeros(case["rays"], _lib.RAY_DTYPE)
    rays["origin"], rays["direction"], rays["length"], rays["world"] = origin, d, reach, world
    return rays


def _shapes(rng, count, dtype):
    out = np.zeros(count, dtype)
    kind = rng.integers(0, 4, count)
    out["shape_type"] = np.array([_lib.SHAPE_SPHERE, _lib.SHAPE_BOX, _lib.SHAPE_CAPSULE, _lib.SHAPE_CYLINDER])[kind]
    p = rng.uniform(0.15, 0.5, (count, 4)).astype(np.float32)
    p[:, 3] = np.where(kind == 1, scenes.DEFAULT_CONVEX_RADIUS, 0.0)
    p[:, 2] = np.where(kind == 3, scenes.DEFAULT_CONVEX_RADIUS, np.where(kind == 1, p[:, 2], 0.0))
    p[:, 1] = np.where(kind == 0, 0.0, p[:, 1])
    out["shape_params"] = p
    out["quaternion"] = scenes.random_quaternions(rng, count)
    return out


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def prepare(case, seed):
    torch.cuda.init()
    s = {"case": dict(case)}
    kind = case["kind"]
    if kind == "grad":
        sc, targets = scenes.diff_rollout_worlds(case["worlds"], seed=seed, boxes=case["boxes"])
        w = GpuWorld(standard_settings(velocity_iterations=10, position_iterations=2, num_worlds=case["worlds"],
                                       allow_sleeping=False), len(sc.bodies))
        w.add_bodies(sc.bodies)
        s.update(world=w, rows=w.get_state()[0], targets=targets, dt=1.0 / 60.0)
        return s
    w, bodies = _world(case, seed)
    s["world"] = w
    if kind in ("step", "substeps"):
        s["dt"] = 1.0 / case["hz"]
        rows = w.get_state()[0]
        w.step(s["dt"], 3)
        s["keep"], s["rows"] = _pinned((w.n, _lib.STATE_FLOATS))
        s["keep_out"], s["out"] = _pinned((w.n, _lib.STATE_FLOATS))
        s["rows"][:] = rows
        return s
    if kind == "rays":
        rays = _rays(case, seed)
        if case["device"]:
            s["rays"] = torch.from_numpy(rays.view(np.float32).reshape(len(rays), -1)).cuda()
            s["hits"] = torch.zeros((len(rays), 4), dtype=torch.int32, device="cuda")
            s["filter"] = _lib.QueryFilter(0xFFFFFFFF, 0xFFFFFFFF, 0xFFFFFFFF, _lib.CAST_RAY_TREAT_CONVEX_AS_SOLID)
        else:
            s["rays"] = rays
    elif kind == "casts":
        origin, d, reach, _ = _query_rows(case, seed, case["casts"])
        casts = _shapes(np.random.default_rng(seed + 8), case["casts"], _lib.SHAPE_CAST_DTYPE)
        casts["position"], casts["displacement"] = origin, d * reach[:, None]
        s["casts"] = casts
    else:
        origin, _, _, world = _query_rows(case, seed, case["shapes"])
        shapes = _shapes(np.random.default_rng(seed + 8), case["shapes"], _lib.COLLIDE_SHAPE_DTYPE)
        shapes["position"], shapes["world"] = origin, world
        origin, _, _, world = _query_rows(case, seed + 100, case["points"])
        points = np.zeros(case["points"], _lib.POINT_DTYPE)
        points["position"], points["world"] = origin, world
        s.update(shapes=shapes, points=points)
    w.step(0.0, 1)
    return s


def run(s):
    case, w = s["case"], s["world"]
    kind = case["kind"]
    if kind == "step":
        w.step_host(s["dt"], s["rows"], s["out"])
        return s["out"]
    if kind == "substeps":
        w.set_state(s["rows"])
        w.step(s["dt"], case["steps"])
        return w.get_state()[0]
    if kind == "grad":
        w.set_state(s["rows"])
        loss, gv, gw, gm = w.rollout_grad(s["dt"], case["steps"], s["targets"], checkpoint_every=10)
        return {"loss": loss, "linear": gv, "angular": gw, "friction": gm}
    if kind == "rays":
        if case["device"]:
            _lib.check(_lib.load().cc_world_cast_rays_device(
                w.handle, C.c_void_p(s["rays"].data_ptr()), len(s["rays"]), C.byref(s["filter"]),
                C.c_void_p(s["hits"].data_ptr())), "cc_world_cast_rays_device")
            h = s["hits"]
            return {"body": h[:, 0], "fraction": h[:, 1].view(torch.float32), "sub_shape": h[:, 2]}
        h = w.cast_rays(s["rays"])
        return {"body": h["body"], "fraction": h["fraction"], "sub_shape": h["sub_shape_id"].view(np.int32)}
    if kind == "casts":
        h = w.cast_shapes(s["casts"])
        return {"body": h["body"], "fraction": h["fraction"], "normal": h["normal"], "point": h["point"],
                "sub_shape": h["sub_shape_id"].view(np.int32)}
    hits, counts = w.collide_shapes(s["shapes"], collector=_lib.COLLECT_ALL, max_hits=24)
    inside = w.collide_points(s["points"])
    return {"counts": counts, "body": hits["body"], "penetration": hits["penetration"], "point_a": hits["point_a"],
            "point_b": hits["point_b"], "axis": hits["axis"], "inside": inside["count"], "holder": inside["body"]}


def _body_count(case):
    kind = case["kind"]
    if kind == "grad":
        return case["worlds"] * (case["boxes"] + 1)
    scene = case["scene"]
    if scene == "heap":
        return case["side"] ** 3 + 1
    if scene == "ragdolls":
        return case["ragdolls"] * 11 + 6
    if scene == "terrain":
        return case["bodies"] + 1
    lo, hi = case["low"], case["high"]
    return int(case["worlds"] * (1 + (lo if hi == lo else (hi - lo) / math.log(hi / lo))))


def work(case):
    """Bytes that a pass cannot do without.  A step reads and writes every body's state row (64 bytes
    each way) and reads its constants (shape, mass, inertia, material, damping, filters: 100 bytes); the
    substeps between the first and the last need no bytes of their own.  Queries read each query and
    write each hit once, and read the bodies they are cast against."""
    n, kind = _body_count(case), case["kind"]
    if kind in ("step", "substeps"):
        return {"bytes": n * (64 + 64 + 100), "flops": 0}
    if kind == "grad":
        return {"bytes": n * (64 + 100 + 28) + 16 * case["worlds"], "flops": 0}
    mesh = 2 * case["cells"] ** 2 * 28 if case["scene"] == "terrain" else 0
    bodies = n * 48 + mesh
    if kind == "rays":
        return {"bytes": bodies + case["rays"] * (32 + 16), "flops": 0}
    if kind == "casts":
        return {"bytes": bodies + case["casts"] * (64 + 40), "flops": 0}
    return {"bytes": bodies + case["shapes"] * (56 + 4 + 24 * 48) + case["points"] * 32, "flops": 0}


def exact(case, seed):
    """Ray fractions in 64 bits in the scenes of boxes and spheres; None elsewhere."""
    if case["kind"] != "rays" or case["scene"] != "stacks":
        return None
    b = _stacks(seed, case["worlds"], case["low"], case["high"])
    if case["rays"] * len(b) / case["worlds"] > 2e8:
        return None
    rays = _rays(case, seed)
    o_all = rays["origin"].astype(np.float64)
    v_all = rays["direction"].astype(np.float64) * rays["length"].astype(np.float64)[:, None]
    best = np.ones(len(rays))
    x, y, z, w = np.moveaxis(b["quaternion"].astype(np.float64), -1, 0)
    rot = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                    2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                    2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], -1).reshape(-1, 3, 3)
    by_world = [np.flatnonzero(rays["world"] == k) for k in range(case["worlds"])]
    for i in range(len(b)):
        s = by_world[b["world"][i]]
        o = (o_all[s] - b["position"][i].astype(np.float64)) @ rot[i]  # into the body's frame
        v = v_all[s] @ rot[i]
        p = b["shape_params"][i].astype(np.float64)
        with np.errstate(divide="ignore", invalid="ignore"):
            if b["shape_type"][i] == _lib.SHAPE_SPHERE:
                a2, a1, a0 = (v * v).sum(1), (o * v).sum(1), (o * o).sum(1) - p[0] ** 2
                disc = a1 * a1 - a2 * a0
                t = np.where(a0 <= 0, 0.0, np.where(disc >= 0, (-a1 - np.sqrt(np.maximum(disc, 0))) / a2, np.inf))
            else:
                t0, t1 = (-p[:3] - o) / v, (p[:3] - o) / v
                enter, leave = np.minimum(t0, t1).max(1), np.maximum(t0, t1).min(1)
                t = np.where((enter <= leave) & (leave >= 0), np.maximum(enter, 0.0), np.inf)
        t = np.where(t >= 0, t, np.inf)
        best[s] = np.minimum(best[s], t)
    return {"body": None, "fraction": best, "sub_shape": None}
