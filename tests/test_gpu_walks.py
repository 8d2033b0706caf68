"""GPU: the ordered walks of the single-hit queries against the every-hit
queries (whose walks and casts they do not share), and the pairs of a world
that is wide on one axis only against all pairs of its fat AABBs."""
import ctypes

import numpy as np
import pytest

from bounce_b200 import _native as N
from bounce_b200 import scene as S
from bounce_b200 import serving as V
from bounce_b200.pipeline import CollisionPipeline

pytestmark = pytest.mark.gpu

NONE = 0xFFFFFFFF


def stepped(scene, passes=3, **kw):
    pipe = CollisionPipeline(scene, **kw)
    drv = S.KinematicDriver(scene)
    for k in range(passes):
        if k:
            drv.advance()
        pipe.collide(drv.state17())
    return pipe


def first_of(index, value, n):
    """Per query the row of its smallest value, the smaller fixture on a tie (-1: none)."""
    out = np.full(n, -1, np.int64)
    order = np.lexsort((index[:, 1], value, index[:, 0]))
    q, first = np.unique(index[order, 0], return_index=True)
    out[q] = order[first]
    return out


def world(kind, n):
    rng = np.random.default_rng(n)
    if kind == "mixed":
        return S.mixed_scene(seed=n, n=n, side=max(3.0, 49.0 * (n / 65536.0) ** (1 / 3))).finalize()
    if kind == "mesh":
        return S.mesh_terrain_scene(seed=n, n=n).finalize()
    if kind == "triangles":
        return S.terrain_scene(seed=n, n=n).finalize()
    s, _ = S.batched_scene(seed=int(rng.integers(100)), n_worlds=n, lo=4, hi=200)
    return s.finalize()


# One fixture, two, a few; the ends of a warp, of the warp-per-ray range and of
# a block's share of rays.
@pytest.mark.parametrize("kind,n,rays", [
    ("mixed", 1, 40), ("mixed", 2, 33), ("mixed", 3, 1), ("mixed", 700, 31), ("mixed", 3000, 23681),
    ("mixed", 3000, 23680), ("mixed", 5000, 70001), ("mesh", 600, 500), ("mesh", 600, 30011), ("triangles", 400, 700),
    ("triangles", 400, 24001), ("worlds", 9, 900), ("worlds", 9, 24500)])
def test_first_hit(kind, n, rays):
    sc = world(kind, n)
    pipe = stepped(sc, max_contacts=max(32 * sc.n_fixtures, 80000))
    rng = np.random.default_rng(rays)
    span = np.abs(sc.body_pos).max(axis=0) + 1
    p1 = rng.uniform(-span, span, (rays, 3))
    d = rng.normal(size=(rays, 3)) * rng.uniform(0, 8, (rays, 1))
    d[::17] = np.eye(3)[rng.integers(0, 3, len(d[::17]))] * 6.0  # along one axis
    d[5::101] = 0.0
    r = np.concatenate([p1, p1 + d], axis=1).astype(np.float32)
    worlds = rng.integers(0, sc.n_worlds, rays).astype(np.uint32)
    fix, hit = pipe.ray_cast_single(r, worlds)
    idx, hits = pipe.ray_cast(r, worlds)
    want = first_of(idx.astype(np.int64), hits[:, 6], rays)
    got = want >= 0
    assert np.array_equal(fix != NONE, got)
    if rays > 400:
        assert got.any()
    assert np.array_equal(fix[got], idx[want[got], 1])
    assert np.array_equal(hit[got], hits[want[got]])
    assert not hit[~got].any()
    pipe.close()


def casts_of(sc, n, seed):
    rng = np.random.default_rng(seed)
    pick = rng.integers(0, sc.n_fixtures, n)
    pick = pick[sc.fix_type[pick] != N.SHAPE_MESH]
    pick = rng.choice(pick, n)
    c = np.zeros(n, N.SHAPE_CAST_DTYPE)
    c["type"], c["hull"], c["params"] = sc.fix_type[pick], sc.fix_hull[pick], sc.fix_params.reshape(-1, 12)[pick]
    span = np.abs(sc.body_pos).max(axis=0) + 0.5
    c["position"] = rng.uniform(-span, span, (n, 3))
    c["rotation"] = S.random_quats(rng, n)
    c["displacement"] = rng.normal(size=(n, 3)) * rng.uniform(0, 2.5, (n, 1))
    c["displacement"][::29] = 0.0
    c["world"] = rng.integers(0, sc.n_worlds, n)
    return c


# Lanes per cast go from 32 to 1 over these counts; triangle fixtures on bodies
# away from the identity lie outside their boxes (the reference's quirk).
@pytest.mark.parametrize("kind,n,casts", [
    ("mixed", 1, 3), ("mixed", 2, 33), ("mixed", 700, 1), ("mixed", 2000, 2368), ("mixed", 2000, 2369),
    ("mixed", 2000, 9500), ("mixed", 2000, 40001), ("mixed", 500, 80001), ("mesh", 500, 300), ("mesh", 500, 20000),
    ("triangles", 300, 500), ("turned", 300, 500), ("turned", 300, 9000), ("worlds", 7, 6000)])
def test_first_cast(kind, n, casts):
    sc = world("triangles" if kind == "turned" else kind, n)
    if kind == "turned":
        sc.body_pos[0] = (0.4, 0.3, -0.2)
    pipe = stepped(sc, max_contacts=max(32 * sc.n_fixtures, 90000))
    c = casts_of(sc, casts, n + casts)
    fix, hit = pipe.shape_cast_single(c)
    idx, hits = pipe.shape_cast(c)
    key = idx.astype(np.int64)
    # Of equal fractions the smaller fixture, then triangle.
    order = np.lexsort((key[:, 2], key[:, 1], hits[:, 6], key[:, 0]))
    q, first = np.unique(key[order, 0], return_index=True)
    want = np.full(casts, -1, np.int64)
    want[q] = order[first]
    got = want >= 0
    assert np.array_equal(fix[:, 0] != NONE, got)
    if casts > 400:
        assert got.any()
    assert np.array_equal(fix[got], idx[want[got], 1:])
    assert np.array_equal(hit[got], hits[want[got]])
    assert not hit[~got].any()
    pipe.close()


# Spheres whose box covers none, some, more than a warp's row (128) and all of
# a fine mesh's triangles: a work item per triangle whose box the sphere's fat
# box in mesh space overlaps, and no other.
@pytest.mark.parametrize("radius", [0.05, 0.6, 1.2, 2.5, 9.0])
def test_mesh_items(radius):
    V, T = S.grid_mesh(41, 41, 0.25, 3)
    sc = S.Scene()
    sc.mesh_arrays = dict(desc=np.array([0, len(V), 0, len(T)], np.uint32), verts=np.ascontiguousarray(V.reshape(-1)),
                          tris=np.ascontiguousarray(T.reshape(-1), np.uint32), max_pairs=200000)
    g = sc.add_body(0, N.BODY_STATIC, (0, 0, 0), (0, 0, 0, 1))
    sc.add_fixture(g, N.SHAPE_MESH, [1.0, 1.0, 1.0, 0.0])
    rng = np.random.default_rng(7)
    p = np.concatenate([rng.uniform(-5, 5, (30, 1)), rng.uniform(-1, 1, (30, 1)), rng.uniform(-5, 5, (30, 1))], 1)
    for x in p:
        b = sc.add_body(0, N.BODY_DYNAMIC, x, (0, 0, 0, 1))
        sc.add_fixture(b, N.SHAPE_SPHERE, [0, 0, 0, radius])
    sc.finalize()
    pipe = CollisionPipeline(sc)
    pipe.collide(S.KinematicDriver(sc).state17())
    F = np.float32
    lo, hi = V[T].min(axis=1) - F(0.005), V[T].max(axis=1) + F(0.005)
    want = 0
    for x in sc.body_pos[1:]:
        l, h = (x - F(radius)) - F(0.2), (x + F(radius)) + F(0.2)
        want += int(np.all((lo <= h) & (hi >= l), axis=1).sum())
    assert pipe.pass_stats()["mesh_items"] == want
    pipe.close()


def overlapping(pipe, sc):
    """Contacts every pass must hold: overlapping fat AABBs of two bodies, one of them dynamic."""
    box = pipe.fat_aabbs()
    pairs = set()
    for a in range(len(box)):
        b = np.arange(a + 1, len(box))
        hit = np.all((box[b, :3] <= box[a, 3:]) & (box[b, 3:] >= box[a, :3]), axis=1)
        dyn = (sc.body_type[sc.fix_body[b]] == N.BODY_DYNAMIC) | (sc.body_type[sc.fix_body[a]] == N.BODY_DYNAMIC)
        tri = (sc.fix_type[a] >= N.SHAPE_MESH) & (sc.fix_type[b] >= N.SHAPE_MESH)
        pairs.update((a, int(x)) for x in b[hit & dyn & ~tri])
    return pairs


@pytest.mark.parametrize("scale", [(1.0, 0.02, 1.0), (0.05, 0.05, 1.0), (1.0, 1.0, 1.0)])
def test_pairs_of_flat_and_narrow_worlds(scale):
    sc = S.mixed_scene(seed=8, n=900, side=30.0).finalize()
    sc.body_pos = np.ascontiguousarray(sc.body_pos * np.array(scale, np.float32))
    pipe = stepped(sc, passes=4, max_contacts=400000)
    got = {(min(a, b), max(a, b)) for a, b, _ in pipe.contacts().tolist()}
    assert got == overlapping(pipe, sc)
    pipe.close()


def prism(n, radius, height):
    """A prism over a regular n-gon as packed hull arrays, its caps one face each."""
    a = 2 * np.pi * np.arange(n) / n
    ring = radius * np.stack([np.cos(a), np.zeros(n), np.sin(a)], -1)
    v = np.concatenate([ring + [0, height, 0], ring - [0, height, 0]]).astype(np.float32)
    # Outward loops: the top, the bottom, then the sides.
    loops = [list(range(n))[::-1], [n + i for i in range(n)]]
    loops += [[i, (i + 1) % n, n + (i + 1) % n, n + i] for i in range(n)]
    at, edges = {}, []
    for loop in loops:
        for k, x in enumerate(loop):
            y = loop[(k + 1) % len(loop)]
            if (y, x) in at:
                at[(x, y)] = at[(y, x)] ^ 1
            else:
                at[(x, y)] = len(edges)
                edges += [None, None]
    for f, loop in enumerate(loops):
        ids = [at[(x, loop[(k + 1) % len(loop)])] for k, x in enumerate(loop)]
        for k, e in enumerate(ids):
            edges[e] = [loop[k], e ^ 1, f, ids[k - 1], ids[(k + 1) % len(ids)]]
    faces = [at[(loop[0], loop[1])] for loop in loops]
    planes = []
    for loop in loops:
        p = v[loop].astype(np.float64)
        nrm = np.cross(p[1] - p[0], p[2] - p[1])
        nrm /= np.linalg.norm(nrm)
        planes.append([*nrm, nrm @ p[0]])
    return dict(desc=np.array([0, 2 * n, 0, len(edges), 0, len(loops)], np.uint32), verts=v.reshape(-1),
                edges=np.array(edges, np.uint32).reshape(-1), faces=np.array(faces, np.uint32),
                planes=np.array(planes, np.float32).reshape(-1), centroids=np.zeros(3, np.float32))


# A pair at rest: the pass that finds the contact builds it from the separating
# axes (a warp per contact), the next rebuilds it from the feature cache (a
# lane per contact, rings of a few clip vertices), and both give the same points.
# Faces below, at and beyond what a ring holds; more pairs than a block takes.
@pytest.mark.parametrize("sides", [(3, 3), (4, 4), (4, 9), (3, 15), (15, 3), (16, 4), (8, 16), (17, 4), (30, 30),
                                   (4, 40)])
@pytest.mark.parametrize("pairs", [1, 33, 700])
def test_rebuilt_face_contacts(sides, pairs):
    rng = np.random.default_rng(sides[0] * 100 + sides[1])
    sc = S.Scene()
    low, top = (sc.hulls.extend(prism(n, r, 0.5)) for n, r in zip(sides, (1.0, 0.9)))
    for k in range(pairs):
        x = np.array([5.0 * (k % 30), 0, 5.0 * (k // 30)])
        b = sc.add_body(0, N.BODY_STATIC, x, (0, 0, 0, 1))
        sc.add_fixture(b, N.SHAPE_HULL, [0.02], hull=low)
        turn = rng.uniform(-3, 3) / 2
        x = x + [rng.uniform(-0.6, 0.6), 0.98 + rng.uniform(0, 0.05), rng.uniform(-0.6, 0.6)]
        tilt = np.array([rng.uniform(-0.01, 0.01), np.sin(turn), rng.uniform(-0.01, 0.01), np.cos(turn)])
        b = sc.add_body(0, N.BODY_DYNAMIC, x, tilt / np.linalg.norm(tilt))
        sc.add_fixture(b, N.SHAPE_HULL, [0.02], hull=top)
    sc.finalize()
    pipe = CollisionPipeline(sc, max_contacts=4096)
    state = S.KinematicDriver(sc).state17()
    rounds = []
    for _ in range(2):
        pipe.collide(state)
        index, m = pipe.touching()
        order = np.argsort(index)
        rounds.append((pipe.contacts()[index][order], m[order]))
    assert pipe.pass_stats()["hull_miss"] < len(rounds[0][0])
    (f0, m0), (f1, m1) = rounds
    assert len(f0) >= 0.9 * pairs
    assert np.array_equal(f0[:, :2], f1[:, :2])
    assert np.array_equal(m0["pointCount"], m1["pointCount"])
    for field in ("n", "p1", "p2", "triangleKey", "key", "edgeContact"):
        for i in range(4):
            has = m0["pointCount"] > i
            assert np.array_equal(m0["points"][field][has, i], m1["points"][field][has, i]), field
    pipe.close()


# More overlapping nodes than a warp's stack holds (every box meets every other,
# the lanes go on along the ropes), the fewest leaves, and several worlds whose
# boxes lie on top of one another.
@pytest.mark.parametrize("n,worlds", [(1, 1), (2, 1), (3, 2), (5, 1), (129, 1), (1500, 1), (1200, 7)])
def test_pairs_of_heaped_worlds(n, worlds):
    sc = S.Scene()
    rng = np.random.default_rng(n)
    for k in range(n):
        b = sc.add_body(k % worlds, N.BODY_DYNAMIC, rng.uniform(-0.2, 0.2, 3), (0, 0, 0, 1))
        sc.add_fixture(b, N.SHAPE_SPHERE, [0, 0, 0, 0.5])
    sc.finalize()
    pipe = CollisionPipeline(sc, max_contacts=max(64, n * n))
    state = S.KinematicDriver(sc).state17()
    for _ in range(2):
        pipe.collide(state)
    got = pipe.contacts()[:, :2].astype(np.int64)
    world = np.arange(n) % worlds
    a, b = np.triu_indices(n, 1)
    same = world[a] == world[b]
    want = a[same] * n + b[same]
    assert np.array_equal(np.sort(got.min(axis=1) * n + got.max(axis=1)), np.sort(want))
    per_leaf = 32
    over = sum(max(0, c - 1 - i - per_leaf) for w in range(worlds) for c in [np.sum(world == w)] for i in range(c))
    assert pipe.pass_stats()["trav_overflow"] == over
    pipe.close()


# The packed results and the impulses of worlds on both sides of what travels
# through the small pinned buffers (256 KB), to pageable and to pinned memory;
# mesh contacts bring contacts of several manifolds.
@pytest.mark.parametrize("kind,n", [("mixed", 1), ("mixed", 40), ("mixed", 900), ("mixed", 9000), ("mesh", 700)])
@pytest.mark.parametrize("pinned", [False, True])
def test_results_through_small_buffers(kind, n, pinned):
    torch = pytest.importorskip("torch")
    sc = world(kind, n)
    pipe = CollisionPipeline(sc, max_contacts=max(40 * sc.n_fixtures, 64))
    drv = S.KinematicDriver(sc)
    cap = 4 * sc.n_fixtures + 64
    make = lambda shape, dt: torch.zeros(shape, dtype=dt, pin_memory=pinned).numpy()
    contacts = make((40 * sc.n_fixtures + 64, 3), torch.int32).view(np.uint32)
    index, packed = make((cap,), torch.int32).view(np.uint32), make((cap * 320,), torch.uint8)
    rng = np.random.default_rng(n)
    for k in range(3):
        pipe.collide(drv.state17())
        c = pipe.fetch_results_packed_async(contacts, index, packed)
        pipe.wait_results()
        assert np.array_equal(contacts[: c["contacts"]], pipe.contacts())
        want_index, want = pipe.touching()
        assert np.array_equal(index[: c["manifolds"]], want_index)
        at = 0
        for m in want:
            points = int(m["pointCount"])
            assert packed[at : at + 32].tobytes() == m.tobytes()[288:]
            assert packed[at + 32 : at + 32 + 72 * points].tobytes() == m["points"][:points].tobytes()
            at += 32 + 72 * points
        assert at == 32 * c["manifolds"] + 72 * c["points"]
        # What the solver hands back reaches the next pass's first manifolds.
        c0 = pipe.contacts()[:, :2]
        imp = rng.uniform(0, 1, len(c0)).astype(np.float32)
        pipe.load_impulses(np.zeros((len(c0), 4), np.float32), np.zeros((len(c0), 2), np.float32), imp)
        pipe.collide(drv.state17())
        flags = pipe.contacts()
        man = pipe.manifolds()
        old = {tuple(p): float(x) for p, x in zip(c0.tolist(), imp)}
        both = [(float(m["motorImpulse"]), old[tuple(p[:2])]) for p, m in zip(flags.tolist(), man)
                if tuple(p[:2]) in old and not p[2] & 2 and m["pointCount"] and sc.fix_type[p[0]] != N.SHAPE_MESH
                and sc.fix_type[p[1]] != N.SHAPE_MESH]
        assert all(a == b for a, b in both) and (both or n < 100)
        drv.advance()
    pipe.close()


def flush_by_lists(e, torch):
    """ServingEngine._flush_updates through b3g_update_scene_device's index lists."""
    adm, ret = e.pending_admit, e.pending_retire
    dev = lambda x, dt: torch.from_numpy(np.ascontiguousarray(x, dt)).to(e.dev)
    cat = lambda xs: np.concatenate(xs) if xs else np.zeros(0)
    slots = cat([r.start + np.arange(r.tmpl.n) for r in adm])
    a = [dev(slots, np.int32), dev(cat([np.full(r.tmpl.n, r.world) for r in adm]), np.int32),
         dev(cat([r.tmpl.body_type for r in adm]), np.int32), dev(cat([r.start + r.tmpl.fix_body for r in adm]), np.int32),
         dev(cat([r.tmpl.fix_type for r in adm]), np.int32), dev(cat([r.tmpl.fix_hull for r in adm]), np.int32),
         dev(cat([r.tmpl.fix_params.reshape(-1) for r in adm]), np.float32),
         dev(cat([r.tmpl.fix_flags for r in adm]), np.int32),
         dev(cat([np.arange(s, s + n) for s, n in ret]), np.int32)]
    for r in adm:
        rows = slice(r.tmpl.offset, r.tmpl.offset + r.tmpl.n)
        e.state[r.start:r.start + r.tmpl.n] = e.st_state[rows]
        e.motion[r.start:r.start + r.tmpl.n] = e.st_motion[rows]
    torch.cuda.synchronize()
    b, w, bt, fb, ft, fh, fp, ff, rx = [ctypes.c_void_p(x.data_ptr()) for x in a]
    e._check(e.lib.b3g_update_scene_device(e.ctx, len(a[0]), b, w, bt, len(a[0]), b, fb, ft, fh, fp, ff, len(a[8]), rx,
                                           ctypes.c_void_p(e.sptr)))
    torch.cuda.synchronize()
    e.pending_admit, e.pending_retire = [], []


# More worlds in and out at once than one launch takes (64), and sizes around a
# block's 256 slots, against the same update through index lists.
@pytest.mark.parametrize("sizes", [[2], [255, 256, 257, 700], [4] * 130])
def test_swapped_worlds(sizes):
    torch = pytest.importorskip("torch")
    results = []
    for lists in (False, True):
        e = V.ServingEngine(capacity=4096, max_worlds=256, active_quantum=4096, graph=False)
        if lists:
            e._flush_updates = lambda e=e: flush_by_lists(e, torch)
        t = e.load_templates([V.WorldTemplate(7 + n, n - 1, e.box_hull, e.ground_hull, e.hull_arrays)
                              for n in sorted(set(sizes))])
        rows = []
        for step in range(4):
            for k in range(len(sizes)):
                e.admit(V.Request(step * 1000 + k, t[(k + step) % len(t)], 1 + k % 2, 0.0))
            slot = e.slot
            e.step()
            c = e.counts()
            rows += [np.array(list(c.values())), e.state.cpu().numpy(), e.motion.cpu().numpy(),
                     e.counts_dev[slot].cpu().numpy()]
        results.append(rows)
        e.close()
    assert len(sizes) == 1 or any(r.any() for r in results[0][3::4])
    for a, b in zip(*results):
        assert np.array_equal(a, b)


# Hull-capsule pairs at a distance, touching and deep, one pair a world: however
# many there are (a lane group takes 1 to 8), each is the pair alone.
@pytest.mark.parametrize("worlds", [9, 31, 4737, 9475, 40001])
def test_many_hull_capsule_pairs(worlds):
    rng = np.random.default_rng(3)
    kinds = 9
    where = np.concatenate([rng.uniform(-0.5, 0.5, (kinds, 1)), np.linspace(0.1, 0.85, kinds)[:, None],
                            rng.uniform(-0.5, 0.5, (kinds, 1))], 1)
    turn = S.random_quats(rng, kinds)

    def manifolds(n):
        sc = S.Scene()
        hull = sc.hulls.add_points(S.ellipsoid_points(np.random.default_rng(1), 20, np.array([0.6, 0.5, 0.7])))
        box = sc.hulls.add_box(0.5, 0.4, 0.6)
        for w in range(n):
            b = sc.add_body(w, N.BODY_DYNAMIC, (0, 0, 0), (0, 0, 0, 1))
            sc.add_fixture(b, N.SHAPE_HULL, [0.0], hull=(hull, box)[w % 2])
            b = sc.add_body(w, N.BODY_DYNAMIC, where[w % kinds], turn[w % kinds])
            sc.add_fixture(b, N.SHAPE_CAPSULE, [0, -0.5, 0, 0, 0.5, 0, 0.2])
        sc.finalize()
        pipe = CollisionPipeline(sc, max_contacts=2 * n + 64)
        pipe.collide(S.KinematicDriver(sc).state17())
        c, m = pipe.contacts(), pipe.manifolds()
        pipe.close()
        out = {}
        for (a, _, _), x in zip(c, m):
            points = int(x["pointCount"])
            out[int(a) // 2] = (points, x["points"][:points].tobytes())
        return out

    few = manifolds(2 * kinds)
    assert len(few) >= kinds and any(k for k, _ in few.values())
    many = manifolds(worlds)
    for w, m in many.items():
        assert m == few[w % (2 * kinds)]
    assert len(many) == sum(w % (2 * kinds) in few for w in range(worlds))
