"""The size rules that choose a kernel, at their edges: every path on either side of a line gives
what the general path or the oracle gives.

Tolerances: a solve of one step against another tier in the same order 1e-5 m/s (as the tiers'
other tests) and, for piles up to 91 m tall, 2e-5 m (positions near 64-128 m are held to 4e-6 m and
are written twice a step); islands on lanes against one thread 1e-6 over three steps; pairs exactly;
swept bodies exactly, and 5e-3 m and 5e-2 m/s against the oracle (as the other tests of them); contacts
of the two EPA passes as the passes' other test (1e-5, 1e-4); a ray against an exact surface: it hits
5 mm inside and misses 50 mm outside (the cast's tolerance is 1 mm).
"""
import numpy as np
import pytest

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


@pytest.mark.parametrize("base,iterations", [
    (13, 10), (14, 10),  # 247 and 287 contacts: one warp, one CTA
    (52, 10), (53, 10),  # 4,030 and 4,187: the two sizes of the CTA tier
    (64, 4),             # 2,080 bodies, past the smaller size's 2,048
    (90, 2), (91, 2),    # 12,105 and 12,376: the CTA tier's largest, the whole grid
    (20, 12), (20, 13), (20, 30),  # 12 sweeps are scheduled at a time
])
def test_block_tier_against_the_grid(gpu_lib, base, iterations, monkeypatch):
    sc = scenes.box_pyramid(base)
    scenes.static_floor(sc.bodies, 0, half=(120.0, 0.5, 30.0), friction=0.5)
    g = make(sc, velocity_iterations=iterations)
    monkeypatch.setenv("CRASHCAT_GIANT_MIN", "64")
    ref = make(sc, velocity_iterations=iterations)
    g.step(sc.dt, 1)
    ref.step(sc.dt, 1)
    a, b = g.get_state()[0], ref.get_state()[0]
    assert g.stats()["max_island_constraints"] == base + 3 * base * (base - 1) // 2
    assert np.abs(a[:, 7:13] - b[:, 7:13]).max() < 1e-5
    assert np.abs(a[:, 0:7] - b[:, 0:7]).max() < 2e-5


@pytest.mark.parametrize("base", [1, 2, 3, 4, 5])  # 1, 5, 12 and 22 contacts on lanes, 35 on a warp
def test_lane_islands_against_one_thread(gpu_lib, base, monkeypatch):
    sc = scenes.box_pyramid(base)
    g = make(sc)
    monkeypatch.setenv("CRASHCAT_SMALL_ISLAND_MAX", "64")  # past the size buckets: one thread each
    ref = make(sc)
    for _ in range(3):
        g.step(sc.dt, 1)
        ref.step(sc.dt, 1)
    np.testing.assert_allclose(g.get_state()[0], ref.get_state()[0], atol=1e-6)


@pytest.mark.parametrize("n", [2, 33, 1023, 1024, 1025, 9216, 9217, 16384, 16385])
def test_pairs_at_the_tree_sort_and_scan_sizes(gpu_lib, oracle_lib, n):
    sc = scenes.random_pairs_scene(n=n - 1, seed=n, extent=float(np.sqrt(n)))
    g = make(sc)
    o = pyoracle.OracleWorld(world.standard_settings(), sc.bodies)
    g.step(0.0, 1)
    o.step(0.0, 1)
    canon = lambda p: sorted(tuple(sorted(q)) for q in p.tolist())  # noqa: E731
    assert canon(g.get_pairs()) == canon(o.pairs())


@pytest.mark.parametrize("n", [1, 33, 4095])  # up to 4,096 records of a world are sorted on chip
def test_swept_bodies_of_a_world(gpu_lib, oracle_lib, n):
    """n bullets onto n walls, with one and with two more that meet nothing: 4,096 and 4,097 records
    take the two paths, and the bullets end the same to the bit (hits are resolved in the same order)."""
    def bullets(m):
        b = scenes.blank_bodies(2 * n + m)
        k = np.arange(n + m)
        for i in range(n):
            scenes.set_box(b, i, (0.05, 1.0, 1.0))
        for i in k:
            scenes.set_sphere(b, n + i, 0.2)
        at = np.stack([np.zeros(n + m), 4.0 * (k // 64), 4.0 * (k % 64)], 1)
        b["position"][:n] = at[:n] + (5.0, 0.0, 0.0)
        b["position"][n:] = at
        b["motion_type"][:n] = _lib.STATIC
        b["object_layer"][:n] = scenes.LAYER_NOT_MOVING
        b["linear_velocity"][n:, 0] = 320.0 + k % 7  # past the wall within a step
        b["motion_quality"][n:] = 1
        b["gravity_factor"][n:] = 0.0
        return scenes.Scene("bullets", b, dt=1.0 / 60.0, steps=1)

    rows = []
    for m in (1, 2):
        g = make(bullets(m))
        g.step(1.0 / 60.0, 1)
        assert (g.stats()["num_ccd"], g.stats()["num_ccd_hits"]) == (n + m, n)
        rows.append(g.get_state()[0][n:2 * n])
    np.testing.assert_array_equal(rows[0], rows[1])
    assert (rows[0][:, 0] < 5.0).all()
    if n <= 33:
        o = pyoracle.OracleWorld(world.standard_settings(), bullets(1).bodies)
        o.step(1.0 / 60.0, 1)
        st = o.state()[n:2 * n]
        np.testing.assert_allclose(rows[0][:, 0:3], st[:, 0:3], atol=5e-3)
        np.testing.assert_allclose(rows[0][:, 7:10], st[:, 7:10], atol=5e-2)


@pytest.mark.parametrize("n", [1, 31, 33, 120])
def test_mesh_items_of_the_two_epa_passes(gpu_lib, n, monkeypatch):
    sc = scenes.mesh_drop(n=n, n_cells=16, seed=5, heights=(-0.2, 0.2))  # deep in the triangles

    def contacts():
        g = make(sc)
        g.step(0.0, 1)
        return g.stats()["num_epa"], g.get_manifolds()

    n_epa, packed = contacts()
    monkeypatch.setenv("CRASHCAT_EPA_PACKED_POINTS", "5")
    _, fallback = contacts()
    assert n_epa > 0 or n == 1
    assert len(packed) == len(fallback)
    for p in packed:  # manifolds come in no fixed order
        q = fallback[(fallback[:, 0] == p[0]) & (fallback[:, 1] == p[1])]
        err = np.maximum(np.abs(q[:, 2:7] - p[2:7]).max(1) * 10, np.abs(q[:, 8:] - p[8:]).max(1))
        assert len(q) and err.min() < 1e-4


@pytest.mark.parametrize("n", [1, 31, 33, 100])
@pytest.mark.parametrize("kind", ["sphere", "box", "capsule", "cylinder"])
def test_rays_along_a_surface(gpu_lib, kind, n):
    """Rays from 2 and from 20 m parallel to z pass the shape's side at x = 1, inside it or outside; some
    lanes of their warps have no ray (length 0)."""
    b = scenes.blank_bodies(1)
    {"sphere": lambda: scenes.set_sphere(b, 0, 1.0), "box": lambda: scenes.set_box(b, 0, (1.0, 1.0, 1.0)),
     "capsule": lambda: scenes.set_capsule(b, 0, 1.0, 0.5),
     "cylinder": lambda: scenes.set_cylinder(b, 0, 0.5, 1.0)}[kind]()
    b["motion_type"][0] = _lib.STATIC
    b["object_layer"][0] = scenes.LAYER_NOT_MOVING
    g = make(scenes.Scene("one", b, dt=1.0 / 60.0, steps=1))
    k = np.arange(n)
    inside, far, none = k % 2 == 0, k % 3 == 0, k % 5 == 4
    rays = np.zeros((n, 7))
    rays[:, 0] = np.where(inside, 1.0 - 5e-3, 1.0 + 5e-2)
    rays[:, 2] = np.where(far, -20.0, -2.0)
    rays[:, 5] = 1.0
    rays[:, 6] = np.where(none, 0.0, np.where(far, 40.0, 4.0))
    assert ((g.cast_rays(rays)["body"] == 0) == (inside & ~none)).all()
