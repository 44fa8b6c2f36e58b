"""The island tiers, queries and bounds off the sizes that the other tests meet: where a rule hands a
call from one kernel to another, and inputs at the ends of what the entry points take.

Tolerances: islands on lanes against one thread 1e-6 over three steps, as the other tests of the tiers; piles on one tier against another after
one step 1e-5 m/s and, up to 92 m tall, 2e-5 m (a position near 64-128 m is held to 4e-6 m and written twice); a ray's fraction 1e-4 of 40 m (the cast's tolerance is 1 mm).
"""
import numpy as np
import pytest
from scipy.sparse import coo_matrix
from scipy.sparse.csgraph import connected_components

from crashcat_gb300 import _lib, scenes, world
from oracle import pyoracle

pytestmark = pytest.mark.gpu


def make(sc, **settings):
    ws = world.standard_settings(**settings)
    ws.num_worlds = sc.num_worlds
    g = world.GpuWorld(ws, sc.n + 16)
    for p in sc.hull_points or ():
        g.add_convex_hull(p)
    if sc.mesh is not None:
        g.add_triangle_mesh(*sc.mesh)
    g.add_bodies(sc.bodies)
    return g


@pytest.mark.parametrize("n", [1, 2, 15, 16, 31])
def test_lane_islands_that_hand_one_body_on(gpu_lib, n, monkeypatch):
    """n boxes on a slab: every contact's visit waits for the one before it on the slab, up to a
    full warp of them."""
    b = scenes.blank_bodies(n + 2)
    scenes.static_floor(b, 0)
    k = np.arange(n)
    scenes.set_box(b, 1 + k, (0.2, 0.2, 0.2))
    b["position"][1 + k] = np.stack([(k % 6 - 2.5) * 0.6, np.full(n, 0.5 + 0.2 - 0.005), (k // 6 - 2.5) * 0.6], 1)
    b["linear_velocity"][1 + k] = np.random.default_rng(n).normal(scale=0.3, size=(n, 3))
    scenes.set_box(b, n + 1, (2.0, 0.25, 2.0))
    b["position"][n + 1] = (0.0, 0.25 - 0.005, 0.0)
    sc = scenes.Scene("slab", b, dt=1.0 / 60.0, steps=1)
    g = make(sc)
    monkeypatch.setenv("CRASHCAT_SMALL_ISLAND_MAX", "64")  # past the size buckets: one thread each
    ref = make(sc)
    for _ in range(3):
        g.step(sc.dt, 1)
        ref.step(sc.dt, 1)
        assert g.stats()["max_island_constraints"] == n + 1
    np.testing.assert_allclose(g.get_state()[0], ref.get_state()[0], atol=1e-6)


@pytest.mark.parametrize("base,threshold,grid", [  # 8,855 and 12,650 contacts
    (77, None, 0), (77, "8192", 1),  # the default keeps islands of contacts on a CTA past 8,192
    (92, None, 1), (92, "20000", 0), (92, "2147483647", 0),  # a set threshold holds past the CTA tier's reach
])
def test_islands_above_and_below_the_grid_threshold(gpu_lib, base, threshold, grid, monkeypatch):
    sc = scenes.box_pyramid(base)
    scenes.static_floor(sc.bodies, 0, half=(120.0, 0.5, 30.0), friction=0.5)
    if threshold:
        monkeypatch.setenv("CRASHCAT_GIANT_MIN", threshold)
    g = make(sc, velocity_iterations=2)
    monkeypatch.setenv("CRASHCAT_GIANT_MIN", "64")
    ref = make(sc, velocity_iterations=2)
    g.step(sc.dt, 1)
    ref.step(sc.dt, 1)
    assert (g.stats()["num_giant_islands"], ref.stats()["num_giant_islands"]) == (grid, 1)
    a, b = g.get_state()[0], ref.get_state()[0]
    assert np.abs(a[:, 7:13] - b[:, 7:13]).max() < 1e-5
    assert np.abs(a[:, 0:7] - b[:, 0:7]).max() < 2e-5


@pytest.mark.parametrize("length", [0.25, 1.0, 2.0, 10.0])
def test_rays_with_a_direction_of_any_length(gpu_lib, length):
    """A ray reaches length x direction, whatever the direction's length: the same hits as along the
    unit direction."""
    b = scenes.blank_bodies(4)
    scenes.set_sphere(b, 0, 1.0)
    scenes.set_box(b, 1, (1.0, 1.0, 1.0))
    scenes.set_capsule(b, 2, 1.0, 0.5)
    scenes.set_cylinder(b, 3, 0.5, 1.0)
    y = 10.0 * np.arange(4)[:, None]
    b["position"][:, 1] = y[:, 0]
    b["motion_type"] = _lib.STATIC
    b["object_layer"] = scenes.LAYER_NOT_MOVING
    g = make(scenes.Scene("shapes", b, dt=1.0 / 60.0, steps=1))
    x = np.array([0.0, 0.5, 0.9, 1.1, 3.0])
    rays = np.zeros((4, 5, 7))
    rays[..., 0], rays[..., 1], rays[..., 2] = x, y, -20.0
    hits = []
    for d in (1.0, length):
        rays[..., 5], rays[..., 6] = d, 40.0 / d
        hits.append(g.cast_rays(rays.reshape(-1, 7)))
    assert (hits[0]["body"].reshape(4, 5) == np.where(x < 1, np.arange(4)[:, None], -1)).all()
    np.testing.assert_array_equal(hits[1]["body"], hits[0]["body"])
    np.testing.assert_allclose(hits[1]["fraction"], hits[0]["fraction"], atol=1e-4)


def quad():
    """A static 10 m square of two triangles at y = 0, facing up."""
    b = scenes.blank_bodies(1)
    b["shape_type"][0] = _lib.SHAPE_TRIANGLE_MESH
    b["motion_type"][0] = _lib.STATIC
    b["object_layer"][0] = scenes.LAYER_NOT_MOVING
    sc = scenes.Scene("quad", b, dt=1.0 / 60.0, steps=1)
    sc.mesh = (np.array([[-5, 0, -5], [5, 0, -5], [5, 0, 5], [-5, 0, 5]], np.float32),
               np.array([[0, 2, 1], [0, 3, 2]], np.int32))
    return sc


@pytest.mark.parametrize("dy", [np.nan, np.inf, 0.0, -1.0])
def test_sphere_casts_that_touch_at_the_start(gpu_lib, dy):
    """A sphere that touches a mesh where it starts hits it at fraction 0, whatever it is moved by;
    one 2.5 m above does not."""
    g = make(quad())
    c = np.zeros(2, _lib.SHAPE_CAST_DTYPE)
    c["shape_type"] = _lib.SHAPE_SPHERE
    c["shape_params"][:, 0] = 0.5
    c["position"] = [(1.0, 0.4, 1.0), (1.0, 3.0, 1.0)]
    c["quaternion"][:, 3] = 1.0
    c["displacement"][:, 1] = dy
    h = g.cast_shapes(c)
    assert h["body"].tolist() == [0, -1] and h["fraction"][0] == 0.0


@pytest.mark.parametrize("turned", [False, True])
@pytest.mark.parametrize("shape", ["empty", "empty_moved"])
def test_bounds_of_extents_below_zero(gpu_lib, shape, turned):
    """The world box of a body is the extremes of its corners, so half extents of either sign give the
    same pairs."""
    n = 40
    pairs = []
    for sign in (1.0, -1.0):
        b = scenes.blank_bodies(n + 1)
        for i in range(n):
            scenes.set_sphere(b, i, 0.4)
        b["position"][:n] = np.random.default_rng(3).uniform(-2, 2, (n, 3))
        scenes.set_empty(b, n)
        b["shape_params"][n, 0] = sign
        if shape == "empty_moved":
            b["shape_position"][n] = (0.5, 0.0, 0.0)
        if turned:
            b["quaternion"][n] = (0.0, 0.6, 0.0, 0.8)
        b["motion_type"][n] = _lib.STATIC
        b["object_layer"][n] = scenes.LAYER_NOT_MOVING
        g = make(scenes.Scene("one of no surface", b, dt=1.0 / 60.0, steps=1))
        g.step(0.0, 1)
        pairs.append(sorted(tuple(sorted(p)) for p in g.get_pairs().tolist()))
    assert any(n in p for p in pairs[0])
    assert pairs[0] == pairs[1]


@pytest.mark.parametrize("chains,length", [(1, 4000), (16, 1000), (1000, 30)])
def test_every_body_is_in_the_island_of_its_contacts(gpu_lib, chains, length):
    """Chains of touching spheres numbered at random, so that the links of an island race for its root:
    bodies share an island exactly when contacts join them, in every one of 20 steps."""
    n = chains * length
    b = scenes.blank_bodies(n)
    order = np.random.default_rng(length).permutation(n)
    scenes.set_sphere(b, np.arange(n), 0.5)
    k = np.arange(n)
    b["position"][order] = np.stack([0.999 * (k % length), np.zeros(n), 3.0 * (k // length)], 1)
    b["gravity_factor"] = 0.0
    b["allow_sleeping"] = 0
    g = make(scenes.Scene("chains", b, dt=1.0 / 60.0, steps=1), velocity_iterations=1, position_iterations=0)
    rows = g.get_state()[0]
    for _ in range(20):
        g.set_state(rows)
        g.step(1.0 / 60.0, 1)
        island, contacts = g.debug_islands()
        assert len(contacts) == chains * (length - 1)
        joined = coo_matrix((np.ones(len(contacts)), (contacts[:, 0], contacts[:, 1])), shape=(n, n))
        count, label = connected_components(joined, directed=False)
        assert count == chains == g.stats()["num_islands"]
        assert len(np.unique(np.stack([label, island]), axis=1).T) == count
        np.testing.assert_array_equal(contacts[:, 2], island[contacts[:, 0]])


@pytest.mark.parametrize("base", [20, 53])  # 590 and 4,187 contacts: the CTA tier's two sizes
def test_turn_of_a_cta_island_runs_out_with_a_status(gpu_lib, base, monkeypatch):
    """With a warp's finished chunks not reported, the other warps' wait for their turn runs out after
    the polls that the settings allow: the step returns CC_ERR_TIMEOUT with OVF_TIMEOUT in the counters,
    and the device keeps answering."""
    monkeypatch.setenv("CRASHCAT_TEST_WITHHOLD_BARRIER", "1")
    sc = scenes.box_pyramid(base)
    scenes.static_floor(sc.bodies, 0, half=(120.0, 0.5, 30.0), friction=0.5)
    g = make(sc, device_wait_polls=2000)
    with pytest.raises(_lib.CCError) as e:
        g.step(sc.dt, 1)
    assert e.value.status == _lib.CC_ERR_TIMEOUT
    assert g.stats()["num_giant_islands"] == 0 and g.stats()["overflow_flags"] & 64
    monkeypatch.delenv("CRASHCAT_TEST_WITHHOLD_BARRIER")
    ok = make(sc)
    assert ok.step(sc.dt, 3) == _lib.CC_OK
    assert np.isfinite(ok.get_state()[0]).all()


def bullet_worlds(worlds, k):
    """`worlds` worlds, in each k swept spheres: in three, one hits a wall, one the sphere before it
    (cast too), and one meets nothing."""
    b = scenes.blank_bodies(2 * k)
    i = np.arange(k)
    scenes.set_box(b, i, (0.05, 1.0, 1.0))
    scenes.set_sphere(b, k + i, 0.2)
    at = np.stack([np.zeros(k), np.zeros(k), 4.0 * (i // 3)], 1)
    b["position"][:k] = at + (5.0, 0.0, 0.0)
    b["position"][:k][i % 3 != 0] += (0.0, 500.0, 0.0)  # no wall for these
    b["position"][k:] = at
    b["position"][k:][i % 3 == 1] += (-2.0, 0.1, 0.0)
    b["position"][k:][i % 3 == 2] += (0.0, 50.0, 0.0)
    b["motion_type"][:k] = _lib.STATIC
    b["object_layer"][:k] = scenes.LAYER_NOT_MOVING
    b["linear_velocity"][k:, 0] = np.where(i % 3 == 1, 450.0, 320.0) + i % 7
    b["motion_quality"][k:] = 1
    b["gravity_factor"][k:] = 0.0
    out = np.tile(b, worlds)
    out["world"] = np.repeat(np.arange(worlds), 2 * k)
    return scenes.Scene("bullets", out, dt=1.0 / 60.0, steps=1, num_worlds=worlds)


@pytest.mark.parametrize("k", [1, 2, 15, 16, 25])  # threads up to 15 records of 700 worlds
def test_swept_bodies_of_many_worlds(gpu_lib, k):
    """More worlds than CTAs at once: worlds of few records take a thread, the others a CTA.  Every
    world ends as the same bodies do in a world handle of their own, which take a CTA."""
    worlds = 700
    many, one = make(bullet_worlds(worlds, k)), make(bullet_worlds(1, k))
    for step in range(2):
        many.step(1.0 / 60.0, 1)
        one.step(1.0 / 60.0, 1)
        s, t = many.stats(), one.stats()
        assert (s["num_ccd"], s["num_ccd_hits"]) == (worlds * t["num_ccd"], worlds * t["num_ccd_hits"])
        assert step > 0 or t["num_ccd_hits"] >= (k + 2) // 3
    a, b = many.get_state()[0].reshape(worlds, 2 * k, -1), one.get_state()[0]
    np.testing.assert_array_equal(a, np.broadcast_to(b, a.shape))


@pytest.mark.parametrize("kind", ["falling", "stack", "pairs"])
def test_autotune_of_a_small_world(gpu_lib, kind):
    """A small world starts with fewer EPA blocks than SMs.  Whether or not the tuner finds a shape that
    is faster, the world steps on, and as without the tuner."""
    sc = {"falling": lambda: scenes.free_fall(n=8), "stack": lambda: scenes.box_stack(height=5),
          "pairs": lambda: scenes.random_pairs_scene(n=40)}[kind]()
    tuned, plain = make(sc), make(sc)
    for g in (tuned, plain):
        g.step(sc.dt, 5)
    rep = tuned.autotune(sc.dt, 1)
    assert rep["epa_blocks_per_sm"] >= 0 and rep["giant_min"] == 12288
    for g in (tuned, plain):
        assert g.step(sc.dt, 5) == _lib.CC_OK
    np.testing.assert_allclose(tuned.get_state()[0], plain.get_state()[0], atol=1e-4)


@pytest.mark.parametrize("extra", [0, 1])
def test_islands_at_the_count_that_ends_the_lanes(gpu_lib, extra):
    """Pyramids of 1, 5, 12, 22 and 35 contacts among falling boxes, 16,384 islands (contacts on lanes) or
    one more (threads and both per-warp sizes): the pyramids end as they do alone."""
    parts, alone = [], []
    for base in (1, 2, 3, 4, 5):
        sc = scenes.box_pyramid(base)
        g = make(sc)
        for _ in range(3):
            g.step(sc.dt, 1)
        alone.append(g.get_state()[0])
        b = sc.bodies.copy()
        b["world"] = base
        parts.append(b)
    lone = 16384 - len(parts) + extra
    k = np.arange(lone)
    b = scenes.blank_bodies(lone)
    scenes.set_box(b, k, (0.2, 0.2, 0.2))
    b["position"] = np.stack([2.0 * (k % 128), np.full(lone, 30.0), 2.0 * (k // 128)], 1)
    sc = scenes.Scene("many", np.concatenate(parts + [b]), dt=1.0 / 60.0, steps=3, num_worlds=6)
    g = make(sc)
    for _ in range(3):
        g.step(sc.dt, 1)
        assert g.stats()["num_islands"] == 16384 + extra
    rows, at = g.get_state()[0], 0
    for a in alone:
        np.testing.assert_allclose(rows[at:at + len(a)], a, atol=1e-6)
        at += len(a)


def snake(n):
    """n spheres numbered at random, each touching the next, in rows of 63 joined at their ends: n - 1
    contacts, no gravity."""
    k = np.arange(n)
    row, at = k // 64, k % 64
    x = np.where(row % 2 == 0, np.minimum(at, 62), 62 - np.minimum(at, 62))
    z = 2.0 * row + (at == 63)
    rng = np.random.default_rng(n)
    order = rng.permutation(n)
    b = scenes.blank_bodies(n)
    scenes.set_sphere(b, k, 0.5)
    b["position"][order] = 0.999 * np.stack([x, np.zeros(n), z], 1)
    b["linear_velocity"] = rng.normal(scale=0.3, size=(n, 3))
    b["gravity_factor"] = 0.0
    return scenes.Scene("snake", b, dt=1.0 / 60.0, steps=1)


@pytest.mark.parametrize("n,grid", [(127, 0), (128, 0), (129, 0), (2047, 0), (2048, 0), (2049, 0), (6144, 0), (6145, 1)])
def test_islands_at_the_body_limits(gpu_lib, n, grid, monkeypatch):
    """The tiers' limits of bodies, with half as many contacts as they take: 128 on a warp, 2,048 and
    6,144 on a CTA; against the grid, and the grid against one CTA."""
    sc = snake(n)
    g = make(sc)
    monkeypatch.setenv("CRASHCAT_GIANT_MIN", "2147483647" if grid else "64")
    ref = make(sc)
    g.step(sc.dt, 1)
    ref.step(sc.dt, 1)
    s, t = g.stats(), ref.stats()
    assert s["max_island_constraints"] == t["max_island_constraints"] == n - 1 and s["num_islands"] == 1
    assert (s["num_giant_islands"], t["num_giant_islands"]) == (grid, 1 - grid)
    a, b = g.get_state()[0], ref.get_state()[0]
    assert np.abs(a[:, 7:13] - b[:, 7:13]).max() < 1e-5
    assert np.abs(a[:, 0:7] - b[:, 0:7]).max() < 3e-5  # up to 192 m from the origin


@pytest.mark.parametrize("iterations", [12, 13, 30])
def test_position_sweeps_past_one_schedule(gpu_lib, iterations, monkeypatch):
    sc = scenes.box_pyramid(20)
    sc.bodies["position"][1:, 1] -= 0.02  # pressed in by more than the slop: every sweep moves something
    g = make(sc, position_iterations=iterations)
    monkeypatch.setenv("CRASHCAT_GIANT_MIN", "64")
    ref = make(sc, position_iterations=iterations)
    g.step(sc.dt, 1)
    ref.step(sc.dt, 1)
    a, b = g.get_state()[0], ref.get_state()[0]
    assert np.abs(a[:, 7:13] - b[:, 7:13]).max() < 1e-5
    assert np.abs(a[:, 0:7] - b[:, 0:7]).max() < 2e-5


def test_cta_tiers_side_by_side(gpu_lib, monkeypatch):
    """Islands of both sizes of the CTA tier and jointed ones of the coloured solve in one step, on their
    streams over the shared scratch: each ends as it does in a world handle of its own."""
    monkeypatch.setenv("CRASHCAT_SMALL_JOINTS_MAX", "0")

    def build(scs):
        b, hinges, swings, at = [], [], [], 0
        for k, sc in enumerate(scs):
            rows = sc.bodies.copy()
            rows["world"] = k
            b.append(rows)
            for joints, of in ((hinges, sc.hinges), (swings, sc.swings)):
                if of is not None:
                    j = of.copy()
                    j["body_a"] += at
                    j["body_b"] += at
                    joints.append(j)
            at += len(rows)
        ws = world.standard_settings()
        ws.num_worlds = len(scs)
        g = world.GpuWorld(ws, at + 16)
        g.add_bodies(np.concatenate(b))
        if hinges:
            g.add_hinges(np.concatenate(hinges))
            g.add_swing_twists(np.concatenate(swings))
        g.set_skip_joint_pairs(True)
        return g

    big = scenes.box_pyramid(55)  # 4,510 contacts
    scenes.static_floor(big.bodies, 0, half=(120.0, 0.5, 30.0), friction=0.5)
    scs = [scenes.ragdolls(num=4, arena=12.0), scenes.box_pyramid(15), big, scenes.box_pyramid(20)]
    together = build(scs)
    for _ in range(3):
        together.step(1.0 / 60.0, 1)
    rows, at = together.get_state()[0], 0
    for sc in scs:
        g = build([sc])
        for _ in range(3):
            g.step(1.0 / 60.0, 1)
        np.testing.assert_allclose(rows[at:at + sc.n], g.get_state()[0], atol=1e-6)
        at += sc.n


def triples(groups, extra):
    """Groups of three swept spheres and a wall: sphere A would hit the wall half way through the step;
    B meets A at 0.3 of it, which cancels A's hit; C meets A at 0.8, after A's turn.  `extra` more meet
    nothing."""
    n = 3 * groups + extra
    b = scenes.blank_bodies(groups + n)
    wall, s = np.arange(groups), groups + np.arange(n)
    scenes.set_box(b, wall, (0.05, 0.8, 0.5))
    scenes.set_sphere(b, s, 0.2)
    b["motion_type"][wall] = _lib.STATIC
    b["object_layer"][wall] = scenes.LAYER_NOT_MOVING
    lane = np.stack([40.0 * (wall % 16), np.zeros(groups), 3.0 * (wall // 16)], 1)
    b["position"][wall] = lane + (2.25, 0.0, 0.0)
    for k, (y, vy) in enumerate(((-1.6, 240.0), (3.6, -240.0), (0.0, 0.0))):  # B, C, A
        i = groups + 3 * wall + k
        b["position"][i] = lane + (0.0, y, 0.0)
        b["linear_velocity"][i] = (240.0, vy, 0.0)
    b["position"][s[3 * groups:]] = np.stack([np.arange(extra), np.full(extra, 300.0), np.zeros(extra)], 1)
    b["linear_velocity"][s[3 * groups:], 2] = 240.0
    b["motion_quality"][s] = 1
    b["gravity_factor"][s] = 0.0
    return scenes.Scene("triples", b, dt=1.0 / 60.0, steps=1)


@pytest.mark.parametrize("groups", [1, 11, 1365])  # 1,365: 4,096 and 4,097 records, on chip and on one thread
def test_swept_bodies_that_hit_one_another(gpu_lib, oracle_lib, groups):
    """A record whose hit was cancelled moves at its turn, before a later record hits it."""
    rows = []
    for extra in (1, 2):
        sc = triples(groups, extra)
        g = make(sc)
        g.step(sc.dt, 1)
        assert (g.stats()["num_ccd"], g.stats()["num_ccd_hits"]) == (3 * groups + extra, 3 * groups)
        rows.append(g.get_state()[0][:4 * groups])
    np.testing.assert_array_equal(rows[0], rows[1])
    if groups < 100:
        o = pyoracle.OracleWorld(world.standard_settings(), sc.bodies)
        o.step(sc.dt, 1)
        st = o.state()[:4 * groups]
        np.testing.assert_allclose(rows[0][:, 0:3], st[:, 0:3], atol=5e-3)
        np.testing.assert_allclose(rows[0][:, 7:10], st[:, 7:10], atol=5e-2)


@pytest.mark.parametrize("offset", [0.0, 2000.0])
def test_sphere_casts_far_from_the_origin(gpu_lib, oracle_lib, offset):
    """Long sphere sweeps onto a terrain whose vertices lie `offset` from the mesh's origin, against the
    oracle: as many hits, 99 % of the distances within 2e-3 m and ten times the spacing of FP32 there, all
    within 0.1 m (as the other test of casts onto a terrain)."""
    verts, tris = scenes.heightfield(24, 1.0, 2.0, 5)
    b = scenes.blank_bodies(1)
    b["shape_type"][0] = _lib.SHAPE_TRIANGLE_MESH
    b["motion_type"][0] = _lib.STATIC
    b["object_layer"][0] = scenes.LAYER_NOT_MOVING
    sc = scenes.Scene("far", b, dt=1.0 / 60.0, steps=1)
    sc.mesh = ((np.asarray(verts).reshape(-1, 3) + (offset, 0.0, -offset)).astype(np.float32), tris)
    g = make(sc)
    o = pyoracle.OracleWorld(world.standard_settings(), b, (), [g.get_triangle_mesh(0)])
    rng = np.random.default_rng(7)
    n = 512
    q = np.zeros((n, 15), np.float32)
    q[:, 0] = _lib.SHAPE_SPHERE
    q[:, 1] = rng.uniform(0.05, 1.5, n)
    q[:, 5:8] = np.stack([rng.uniform(-9, 9, n) + offset, rng.uniform(4, 9, n), rng.uniform(-9, 9, n) - offset], 1)
    q[:, 11] = 1.0
    q[:, 12:15] = np.stack([rng.uniform(-12, 12, n), rng.uniform(-14, -3, n), rng.uniform(-12, 12, n)], 1)
    c = np.zeros(n, _lib.SHAPE_CAST_DTYPE)
    c["shape_type"] = _lib.SHAPE_SPHERE
    c["shape_params"], c["position"], c["quaternion"], c["displacement"] = q[:, 1:5], q[:, 5:8], q[:, 8:12], q[:, 12:15]
    h = g.cast_shapes(c)
    out, bo = o.cast_shapes(q.astype(np.float64))
    hit = (h["body"] == 0) & (bo == 0)
    assert (bo == 0).sum() > 300 and ((h["body"] == 0) == (bo == 0)).mean() >= 0.99
    err = np.abs(h["fraction"][hit] - out[hit, 0]) * np.linalg.norm(q[hit, 12:15], axis=1)
    assert np.quantile(err, 0.99) < 2e-3 + 10 * np.spacing(np.float32(offset)) and err.max() < 0.1


@pytest.mark.parametrize("worlds,per", [(341, 3), (256, 4), (205, 5), (11, 93), (2, 512)])  # 1,023 to 1,025 bodies
def test_queries_of_many_worlds_at_the_small_tree_sizes(gpu_lib, worlds, per):
    """Every world holds the same row of spheres; a ray along a world's row, a cast and a point meet
    that world's bodies only."""
    n = worlds * per
    b = scenes.blank_bodies(n)
    k = np.arange(n)
    scenes.set_sphere(b, k, 0.4)
    b["position"][:, 0] = 2.0 + 2.0 * (k % per)
    b["world"] = k // per
    b["motion_type"] = _lib.STATIC
    b["object_layer"] = scenes.LAYER_NOT_MOVING
    g = make(scenes.Scene("rows", b, dt=1.0 / 60.0, steps=1, num_worlds=worlds))
    w = np.arange(worlds)
    rays = np.zeros((worlds, 8))
    rays[:, 3], rays[:, 6], rays[:, 7] = 1.0, 4.0 * per, w
    h = g.cast_rays(rays)
    np.testing.assert_array_equal(h["body"], w * per)
    np.testing.assert_allclose(h["fraction"] * rays[:, 6], 1.6, atol=2e-3)
    c = np.zeros(worlds, _lib.SHAPE_CAST_DTYPE)
    c["shape_type"], c["shape_params"][:, 0], c["quaternion"][:, 3], c["world"] = _lib.SHAPE_SPHERE, 0.1, 1.0, w
    c["position"][:, 0], c["displacement"][:, 0] = 2.0 * per + 4.0, -4.0 * per  # from the row's far end
    np.testing.assert_array_equal(g.cast_shapes(c)["body"], w * per + per - 1)
    p = np.zeros(worlds, _lib.POINT_DTYPE)
    p["position"][:, 0], p["world"] = 2.0 * per, w
    inside = g.collide_points(p)
    np.testing.assert_array_equal(inside["body"], w * per + per - 1)
    assert (inside["count"] == 1).all()


@pytest.mark.parametrize("worlds", [1, 2, 3, 7])
@pytest.mark.parametrize("scene", [("pyramid", 3), ("stack", 9), ("stack", 16), ("pyramid", 4)])  # 12, 9, 16, 22 contacts
def test_lane_islands_that_share_a_warp(gpu_lib, scene, worlds, monkeypatch):
    """Islands of 9 to 16 contacts go two to a warp, the last one alone; against one thread each."""
    kind, size = scene
    sc = scenes.box_pyramid(size) if kind == "pyramid" else scenes.box_stack(height=size)
    b = np.tile(sc.bodies, worlds)
    b["world"] = np.repeat(np.arange(worlds), sc.n)
    b["linear_velocity"][b["motion_type"] == 2] += np.random.default_rng(worlds).normal(
        scale=0.1, size=((b["motion_type"] == 2).sum(), 3))  # no two islands alike
    sc = scenes.Scene("tiled", b, dt=1.0 / 60.0, steps=1, num_worlds=worlds)
    g = make(sc)
    monkeypatch.setenv("CRASHCAT_SMALL_ISLAND_MAX", "64")
    ref = make(sc)
    for _ in range(3):
        g.step(sc.dt, 1)
        ref.step(sc.dt, 1)
    np.testing.assert_allclose(g.get_state()[0], ref.get_state()[0], atol=1e-6)
