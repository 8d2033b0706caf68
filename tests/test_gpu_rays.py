"""GPU: RayCastSingle against the smallest fraction of RayCast (every hit),
bit for bit, where the ordered walks could leave a hit out or take another:
rays that start in a shape's surface, fractions without an order, long rays
that only just touch their shapes, triangles outside their boxes.

The batch sizes lie on both sides of the two walks' border (a warp per ray up
to 23,680 rays)."""
import numpy as np
import pytest

from bounce_b200 import _native as N
from bounce_b200 import scene as S
from bounce_b200.pipeline import CollisionPipeline

pytestmark = pytest.mark.gpu

NONE = 0xFFFFFFFF
BATCHES = [700, 23681]


def same_first_hit(sc, rays):
    """ray_cast_single(rays) is the first of ray_cast(rays); returns its hits' fractions."""
    pipe = CollisionPipeline(sc, max_contacts=max(32 * sc.n_fixtures, 80000))
    pipe.collide(S.KinematicDriver(sc).state17())
    rays = np.ascontiguousarray(rays, np.float32)
    fix, hit = pipe.ray_cast_single(rays)
    idx, hits = pipe.ray_cast(rays)
    pipe.close()
    # A fraction that is not a number is below no other (world.cpp:500-566).
    ordered = hits[:, 6] == hits[:, 6]
    idx, hits = idx[ordered].astype(np.int64), hits[ordered]
    # Of equal fractions (-0 and 0 among them) the smaller fixture.
    order = np.lexsort((idx[:, 1], hits[:, 6], idx[:, 0]))
    ray, first = np.unique(idx[order, 0], return_index=True)
    want = order[first]
    assert np.array_equal(np.nonzero(fix != NONE)[0], ray)
    assert np.array_equal(fix[ray], idx[want, 1])
    assert hit[ray].tobytes() == hits[want].tobytes()
    return hits[want, 6]


def surface_rays(points, directions, n, rng):
    p1 = points[rng.integers(0, len(points), n)]
    return np.concatenate([p1, p1 + directions[rng.integers(0, len(directions), n)]], axis=1)


# From points of a ground at y = 0 up and down, with spheres on both sides: the
# plane's fraction is 0 or -0, and either is before the spheres'.
@pytest.mark.parametrize("n", BATCHES)
@pytest.mark.parametrize("ground", ["mesh", "triangles"])
def test_from_the_ground(ground, n):
    rng = np.random.default_rng(n)
    sc = S.Scene()
    g = sc.add_body(0, N.BODY_STATIC, (0, 0, 0), (0, 0, 0, 1))
    if ground == "mesh":
        V, T = S.grid_mesh(9, 9, 1.0, 3, amplitude=0.0)
        sc.mesh_arrays = dict(desc=np.array([0, len(V), 0, len(T)], np.uint32), verts=np.ascontiguousarray(V.reshape(-1)),
                              tris=np.ascontiguousarray(T.reshape(-1), np.uint32), max_pairs=20000)
        sc.add_fixture(g, N.SHAPE_MESH, [1.0, 1.0, 1.0, 0.0])
    else:
        params, _ = S.terrain_triangles(9, 9, 1.0, 3, amplitude=0.0)
        for p in params:
            sc.add_fixture(g, N.SHAPE_TRIANGLE, list(p[:9]) + [0.0])
    for y in (-3.0, 3.0):
        for x in (-3.0, -1.0, 1.0, 3.0):
            for z in (-3.0, -1.0, 1.0, 3.0):
                b = sc.add_body(0, N.BODY_DYNAMIC, (x, y, z), (0, 0, 0, 1))
                sc.add_fixture(b, N.SHAPE_SPHERE, [0, 0, 0, 0.9])
    sc.finalize()
    points = rng.uniform(-3.5, 3.5, (400, 3))
    points[::3] = rng.integers(-3, 4, (len(points[::3]), 3))  # vertices
    points[:, 1] = 0.0
    directions = rng.uniform(-2, 2, (50, 3))
    directions[:, 1] = np.where(np.arange(50) & 1, 6.0, -6.0)
    directions[::5, ::2] = 0.0
    fractions = same_first_hit(sc, surface_rays(points, directions, n, rng))
    assert (fractions == 0.0).mean() > 0.9 and np.signbit(fractions[fractions == 0.0]).any()


# From a point of a capsule's side along its tangent (a fraction of -0), and
# rays whose lengths overflow (fractions that are no numbers).
@pytest.mark.parametrize("n", BATCHES)
def test_tangent_and_endless(n):
    rng = np.random.default_rng(n)
    sc = S.Scene()
    for z in (0.0, 4.0, -4.0):
        b = sc.add_body(0, N.BODY_DYNAMIC, (0, 0, z), (0, 0, 0, 1))
        sc.add_fixture(b, N.SHAPE_CAPSULE, [0, -0.5, 0, 0, 0.5, 0, 0.5])
    sc.finalize()
    points = np.array([[0.5, 0.0, 0.0], [-0.5, 0.25, 0.0], [0.5, -0.25, 4.0]])
    directions = np.array([[0.0, 0.0, 8.0], [0.0, 0.0, -8.0], [-0.125, 0.0, 8.0], [0.0, 1.0, 4.0]])
    rays = surface_rays(points, directions, n, rng)
    rays[::4] = rng.normal(size=(len(rays[::4]), 6)) * 1e25
    same_first_hit(sc, rays)


def tangent_rays(sc, n, rng):
    """Rays of 50 to 1,000 m that pass the fixtures' bounding spheres, a
    capsule's hemispheres or a hull's vertices at their surface."""
    pick = rng.integers(0, sc.n_fixtures, n)
    params = sc.fix_params.reshape(-1, 12)[pick]
    kind = sc.fix_type[pick]
    verts, desc = sc.hull_arrays["verts"].reshape(-1, 3), sc.hull_arrays["desc"].reshape(-1, 6)
    local = np.zeros((n, 3), np.float32)
    radius = np.where(kind == N.SHAPE_SPHERE, params[:, 3], np.where(kind == N.SHAPE_CAPSULE, params[:, 6], 0.0))
    ends = np.where(rng.random(n)[:, None] < 0.5, params[:, 0:3], params[:, 3:6])
    local[kind == N.SHAPE_CAPSULE] = ends[kind == N.SHAPE_CAPSULE]
    for i in np.nonzero(kind == N.SHAPE_HULL)[0]:
        d = desc[sc.fix_hull[pick[i]]]
        local[i] = verts[d[0] + rng.integers(d[1])]
    c = S.xf_apply(sc.body_pos[sc.fix_body[pick]], sc.body_quat[sc.fix_body[pick]], local)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    side = np.cross(d, rng.normal(size=(n, 3)))
    side /= np.linalg.norm(side, axis=1)[:, None]
    length = np.exp(rng.uniform(np.log(50.0), np.log(1000.0), n))
    # As far outside as the rounding of a cast reaches: about a part in a
    # million of the squared length over the radius.
    off = radius + rng.uniform(-0.2, 1.0, n) * 1e-6 * length**2 / np.maximum(radius, 0.3)
    p1 = c + side * off[:, None] - d * (length * rng.uniform(0.05, 0.95, n))[:, None]
    return np.concatenate([p1, p1 + d * length[:, None]], axis=1)


@pytest.mark.parametrize("n", BATCHES)
def test_long_tangent_rays(n):
    rng = np.random.default_rng(n)
    sc = S.mixed_scene(seed=n, n=400, side=24.0).finalize()
    same_first_hit(sc, tangent_rays(sc, n, rng))


# Hulls with faces that meet at a sharp edge, and plates.
@pytest.mark.parametrize("n", BATCHES)
def test_long_rays_past_sharp_hulls(n):
    rng = np.random.default_rng(n)
    sc = S.Scene()
    shapes = []
    for w, t in ((4.0, 0.004), (3.0, 0.05), (2.0, 0.4)):
        x = np.array([[-w, 0, -0.5], [-w, 0, 0.5], [w, -t, -0.5], [w, -t, 0.5], [w, t, -0.5], [w, t, 0.5]])
        shapes.append(sc.hulls.add_points(x.astype(np.float32)))
    q = S.random_quats(rng, 60)
    for i in range(60):
        b = sc.add_body(0, N.BODY_DYNAMIC, rng.uniform(-15, 15, 3), q[i])
        sc.add_fixture(b, N.SHAPE_HULL, [0.0], hull=shapes[i % 3])
    sc.finalize()
    same_first_hit(sc, tangent_rays(sc, n, rng))


# Triangles of a body away from the identity are not where their boxes are
# (triangle_shape.cpp:59-67): a ray can hit one, then a body, and only then
# meet the triangle's box.
@pytest.mark.parametrize("n", BATCHES)
@pytest.mark.parametrize("shift", [(0.3, 2.0, -0.2), (0.0, -1.5, 0.0)])
def test_triangles_outside_their_boxes(shift, n):
    rng = np.random.default_rng(n)
    sc = S.terrain_scene(seed=5, n=300)
    sc.body_pos[0] = shift
    sc.finalize()
    p1 = rng.uniform(-8, 8, (n, 3))
    p1[:, 1] = np.where(rng.random(n) < 0.5, 7.0, -7.0)
    d = rng.normal(size=(n, 3)) * (1.0, 0.0, 1.0)
    d[:, 1] = -2.0 * p1[:, 1]
    same_first_hit(sc, np.concatenate([p1, p1 + d], axis=1))
