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
