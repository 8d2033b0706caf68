"""Performance cases: the calls a program built on this library makes, over the
sizes it makes them at.

A case is a dict of plain values. ``call`` names what is run:

``step``   one collision pass and its results. ``io`` says how the program
           exchanges data with it: "host" (body state from host memory, contact
           list and touching manifolds back to host memory, as the engine's
           contact manager does every step) or "device" (body state in device
           memory, the solver's contact constraints built into device memory,
           as a device solver does).
``serve``  one step of the serving loop: requests admitted and retired, bodies
           moved, one pass over every resident world, the per-world counts back.
``rays``   RayCastSingle for a batch of rays, from host or device memory.
``casts``  ShapeCastSingle for a batch of shape casts on device memory.
``toi``    b3TimeOfImpact for a batch of sweep pairs on device memory.

``scene`` is the world of a case: "mixed" (40 % spheres, 30 % capsules, 30 %
convex hulls of 8-32 points at the density of the 65,536-body benchmark world),
"plain" (unit boxes and spheres over a ground box, the density of the
2,000-body scene), "terrain" (mixed bodies over a triangle mesh), "pile"
(columns of touching hulls of 12-64 points over a triangle mesh), "batched"
(independent plain worlds of 16-4,096 bodies). Bodies move back and forth along
the first MOVES poses of their kinematic motion, so any number of passes meets
the same contact density.

The collision pass, the shape casts and the time of impact have no value in 64
bits that a pass in 32 bits could be held to (feature choices, iteration counts
and iterative tolerances decide their results), so ``exact`` gives one only for
the ray casts, whose hit points are closed forms.
"""
import ctypes
import math

import numpy as np
import torch

from bounce_b200 import _native as N
from bounce_b200 import scene as S
from bounce_b200 import serving as V
from bounce_b200.pipeline import CollisionPipeline

F = np.float32
DT = 1.0 / 60.0
MOVES = 8  # poses away from the start before the bodies turn back
HULL_POOL = 512  # distinct hulls a world's bodies share


def listed():
    return [
        # A small game scene stepped with the defaults: state in ordinary host
        # memory, the solver's impulses handed back each step. Latency only.
        dict(name="step_host_mixed_64", call="step", io="host", scene="mixed", bodies=64, graph=False, pinned=False,
             impulses=True, asleep=0.0),
        # The 2,000-body falling-objects scene with part of the bodies asleep
        # (awake flags in, wake-ups resolved in the pass).
        dict(name="step_host_plain_2001_sleep", call="step", io="host", scene="plain", bodies=2001, graph=True,
             pinned=True, impulses=False, asleep=0.4),
        # Mixed bodies on a mesh ground, impulses handed back each step.
        dict(name="step_host_terrain_3001", call="step", io="host", scene="terrain", bodies=3001, graph=True,
             pinned=True, impulses=True, asleep=0.0),
        # The benchmark world through host memory.
        dict(name="step_host_mixed_65536", call="step", io="host", scene="mixed", bodies=65536, graph=True,
             pinned=True, impulses=False, asleep=0.0),
        # The benchmark world resident on the device.
        dict(name="step_device_mixed_65536", call="step", io="device", scene="mixed", bodies=65536, graph=True),
        # Many independent worlds in one pass (a batched simulator).
        dict(name="step_device_batched_512", call="step", io="device", scene="batched", worlds=512, graph=True),
        # A settled pile of large hulls over a mesh.
        dict(name="step_device_pile_24064", call="step", io="device", scene="pile", bodies=24064, graph=True),
        # The serving loop at a steady load.
        dict(name="serve_192", call="serve", worlds=192),
        # The few rays of one game tick, through host memory.
        dict(name="rays_host_100", call="rays", io="host", rays=100, bodies=5000),
        # A sensor simulator's batch of rays.
        dict(name="rays_device_524288", call="rays", io="device", rays=524288, bodies=65536),
        # A planner's batch of swept shapes.
        dict(name="casts_device_16384", call="casts", casts=16384, bodies=20001),
        # Continuous collision of a batch of body pairs.
        dict(name="toi_device_262144", call="toi", queries=262144),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "host", "host", "device", "device", "pile", "batched", "serve", "rays_host",
                       "rays_device", "casts", "toi"])
    if kind == "host":
        scene = rng.choice(["mixed", "plain", "terrain"])
        n = _log_int(rng, 16, {"mixed": 65536, "plain": 16384, "terrain": 8192}[scene])
        pinned = rng.random() < 0.75
        return dict(call="step", io="host", scene=scene, bodies=n, graph=pinned, pinned=pinned,
                    impulses=rng.random() < 0.5, asleep=rng.choice([0.0, 0.0, 0.3]))
    if kind == "device":
        return dict(call="step", io="device", scene=rng.choice(["mixed", "mixed", "plain"]),
                    bodies=_log_int(rng, 256, 65536), graph=True)
    if kind == "pile":
        return dict(call="step", io="device", scene="pile", bodies=_log_int(rng, 1024, 24064), graph=True)
    if kind == "batched":
        return dict(call="step", io="device", scene="batched", worlds=_log_int(rng, 8, 512), graph=True)
    if kind == "serve":
        return dict(call="serve", worlds=_log_int(rng, 16, 192))
    if kind == "rays_host":
        return dict(call="rays", io="host", rays=_log_int(rng, 1, 4096), bodies=_log_int(rng, 500, 20000))
    if kind == "rays_device":
        return dict(call="rays", io="device", rays=_log_int(rng, 8192, 524288), bodies=_log_int(rng, 2000, 65536))
    if kind == "casts":
        return dict(call="casts", casts=_log_int(rng, 512, 16384), bodies=_log_int(rng, 2000, 20001))
    return dict(call="toi", queries=_log_int(rng, 2048, 262144))


# ---------------------------------------------------------------------------
# Worlds.


def _hulls(rng, pool, count, pts, axes):
    while len(pool) < count:
        m = int(rng.integers(pts[0], pts[1] + 1))
        try:
            pool.add_points(S.ellipsoid_points(rng, m, rng.uniform(axes[0], axes[1], 3)))
        except ValueError:
            continue
    return pool


def _assemble(pool, world, btype, pos, quat, lin, ang, ftype, hull, params, mesh=None):
    """A Scene from arrays, one fixture per body."""
    s = S.Scene()
    n = len(pos)
    s.hull_arrays = pool.arrays()
    s.body_world = np.ascontiguousarray(world, np.uint32)
    s.body_type = np.ascontiguousarray(btype, np.uint32)
    s.body_pos = np.ascontiguousarray(pos, F)
    s.body_quat = np.ascontiguousarray(quat, F)
    s.body_lin = np.ascontiguousarray(lin, F)
    s.body_ang = np.ascontiguousarray(ang, F)
    s.fix_body = np.arange(n, dtype=np.uint32)
    s.fix_type = np.ascontiguousarray(ftype, np.uint32)
    s.fix_hull = np.ascontiguousarray(hull, np.uint32)
    s.fix_params = np.ascontiguousarray(params, F).reshape(-1)
    s.fix_flags = np.zeros(n, np.uint32)
    # Centres of mass: only the hulls' lie off their bodies' origins.
    cents = s.hull_arrays["centroids"].reshape(-1, 3)
    own = (s.fix_type == N.SHAPE_HULL) & (s.body_type == N.BODY_DYNAMIC)
    s.local_center = np.where(own[:, None], cents[s.fix_hull * own], F(0)).astype(F)
    if mesh is not None:
        verts, tris = mesh
        s.mesh_arrays = dict(desc=np.array([0, len(verts), 0, len(tris)], np.uint32),
                             verts=np.ascontiguousarray(verts.reshape(-1), F),
                             tris=np.ascontiguousarray(tris.reshape(-1), np.uint32))
    return s


def _mixed_shapes(rng, n, hulls, ranges):
    """Types, hulls and params of n mixed bodies."""
    (s0, s1), (r0, r1), (h0, h1) = ranges
    kind = rng.random(n)
    ftype = np.where(kind < 0.4, N.SHAPE_SPHERE, np.where(kind < 0.7, N.SHAPE_CAPSULE, N.SHAPE_HULL)).astype(np.uint32)
    params = np.zeros((n, 12), F)
    sph, cap = ftype == N.SHAPE_SPHERE, ftype == N.SHAPE_CAPSULE
    params[sph, 3] = rng.uniform(s0, s1, n)[sph]
    h, r = rng.uniform(h0, h1, n), rng.uniform(r0, r1, n)
    params[cap, 1], params[cap, 4], params[cap, 6] = -h[cap], h[cap], r[cap]
    hull = np.where(ftype == N.SHAPE_HULL, rng.integers(0, hulls, n), 0)
    return ftype, hull, params


def _prepend(ground, arrays):
    """A first body in front of the others' arrays."""
    return [np.concatenate([np.asarray(g, a.dtype).reshape((1,) + a.shape[1:]), a]) for g, a in zip(ground, arrays)]


def _velocities(rng, n, down=0.0):
    lin, ang = rng.normal(0, 1, (n, 3)).astype(F), rng.normal(0, 1, (n, 3)).astype(F)
    lin[:, 1] -= F(down)
    return lin, ang


def _mixed(rng, n):
    pool = _hulls(rng, S.HullPool(), min(HULL_POOL, max(8, n // 4)), (8, 32), (0.3, 1.2))
    side = 49.0 * (n / 65536.0) ** (1.0 / 3.0)
    pos = rng.uniform(-side / 2, side / 2, (n, 3)).astype(F)
    lin, ang = _velocities(rng, n)
    ftype, hull, params = _mixed_shapes(rng, n, len(pool), ((0.2, 1.0), (0.1, 0.5), (0.2, 1.0)))
    return _assemble(pool, np.zeros(n), np.full(n, N.BODY_DYNAMIC), pos, S.random_quats(rng, n), lin, ang, ftype, hull,
                     params)


def _plain(rng, counts):
    """Plain worlds of counts[w] bodies each, one ground box per world first."""
    pool = S.HullPool()
    box, ground = pool.add_box(0.5, 0.5, 0.5), pool.add_box(50.0, 0.5, 50.0)
    counts = np.asarray(counts)
    total = int(counts.sum()) + len(counts)
    world = np.repeat(np.arange(len(counts)), counts + 1)
    first = np.concatenate([[0], np.cumsum(counts + 1)[:-1]])
    local = np.arange(total) - first[world]
    is_ground = local == 0
    side = np.maximum(20.0 * (counts / 2000.0) ** (1.0 / 3.0), 4.0)[world]
    pos = rng.uniform(-0.5, 0.5, (total, 3)) * side[:, None]
    pos[:, 1] += 0.5 + side / 2
    pos[is_ground] = (0.0, -0.5, 0.0)
    quat = S.random_quats(rng, total)
    quat[is_ground] = (0, 0, 0, 1)
    lin, ang = _velocities(rng, total)
    lin[is_ground] = ang[is_ground] = 0
    hulls = is_ground | (local <= counts[world] // 2)
    params = np.zeros((total, 12), F)
    params[~hulls, 3] = 0.5
    return _assemble(pool, world, np.where(is_ground, N.BODY_STATIC, N.BODY_DYNAMIC), pos, quat, lin, ang,
                     np.where(hulls, N.SHAPE_HULL, N.SHAPE_SPHERE), np.where(is_ground, ground, np.where(hulls, box, 0)),
                     params)


def _with_ground(pool, mesh, pos, quat, lin, ang, ftype, hull, params):
    n = len(pos)
    scale = np.zeros(12, F)
    scale[:3] = 1.0
    pos, quat, lin, ang, ftype, hull, params = _prepend(
        ((0, 0, 0), (0, 0, 0, 1), (0, 0, 0), (0, 0, 0), N.SHAPE_MESH, 0, scale),
        (pos, quat, lin, ang, ftype, hull, params))
    btype = np.full(n + 1, N.BODY_DYNAMIC)
    btype[0] = N.BODY_STATIC
    return _assemble(pool, np.zeros(n + 1), btype, pos, quat, lin, ang, ftype, hull, params, mesh)


def _terrain(rng, n):
    grid = max(6, int(round(14 * math.sqrt(n / 800.0))))
    mesh = S.grid_mesh(grid, grid, 1.5, int(rng.integers(1 << 30)))
    pool = _hulls(rng, S.HullPool(), min(HULL_POOL, max(8, n // 4)), (8, 20), (0.3, 0.8))
    half = 0.75 * (grid - 1)
    pos = np.stack([rng.uniform(-half, half, n), rng.uniform(-0.5, 4.0, n), rng.uniform(-half, half, n)], -1).astype(F)
    lin, ang = _velocities(rng, n, down=1.0)
    ftype, hull, params = _mixed_shapes(rng, n, len(pool), ((0.2, 0.6), (0.1, 0.4), (0.2, 0.7)))
    return _with_ground(pool, mesh, pos, S.random_quats(rng, n), lin, ang, ftype, hull, params)


def _pile(rng, n):
    per = 64
    columns = max(1, n // per)
    n = columns * per
    pool = _hulls(rng, S.HullPool(), HULL_POOL, (12, 64), (0.3, 1.0))
    arrays = pool.arrays()
    desc, verts = arrays["desc"].reshape(-1, 6), arrays["verts"].reshape(-1, 3)
    hull, quat = rng.integers(0, len(pool), n), S.random_quats(rng, n)
    # Vertical extent of each rotated hull (vertices padded by their first).
    pad = np.minimum(np.arange(desc[:, 1].max())[None], desc[:, 1:2].astype(int) - 1) + desc[:, 0:1]
    y = S.quat_rotate(quat[:, None, :], verts[pad][hull])[..., 1]
    top, bottom = y.max(axis=1).reshape(columns, per), y.min(axis=1).reshape(columns, per)
    # Stacked a little closer than their extents, which the hulls reach at
    # different places: most neighbours touch.
    pitch = np.zeros((columns, per))
    pitch[:, 1:] = 0.72 * (top[:, :-1] - bottom[:, 1:])
    cols = int(math.ceil(math.sqrt(columns)))
    grid = max(8, 5 * cols + 8)
    mesh_seed = int(rng.integers(1 << 30))
    mesh = S.sines_mesh(grid, 0.5, mesh_seed)
    c = np.arange(columns)
    cx, cz = (c % cols - (cols - 1) / 2.0) * 2.5, (c // cols - (cols - 1) / 2.0) * 2.5
    base = S.sines_heights(cx, cz, mesh_seed) + 0.1 - 0.72 * bottom[:, 0]
    height = base[:, None] + np.cumsum(pitch, axis=1)
    pos = np.stack([np.repeat(cx, per), height.reshape(-1), np.repeat(cz, per)], -1).astype(F)
    lin = rng.normal(0, 0.02, (n, 3)).astype(F)
    ang = rng.normal(0, 0.05, (n, 3)).astype(F)
    return _with_ground(pool, mesh, pos, quat, lin, ang, np.full(n, N.SHAPE_HULL, np.uint32), hull,
                        np.zeros((n, 12), F))


def _batched(rng, worlds):
    sizes = np.exp(np.log(16) + (np.arange(worlds) + 0.5) / worlds * np.log(4096 / 16))
    return _plain(rng, rng.permutation(np.round(sizes).astype(int)))


def _scene(case, rng):
    kind = case["scene"]
    if kind == "batched":
        return _batched(rng, case["worlds"])
    if kind == "plain":
        return _plain(rng, [case["bodies"]])
    return {"mixed": _mixed, "terrain": _terrain, "pile": _pile}[kind](rng, case["bodies"])


# Contacts, touching contacts and manifold points per body of each world.
DENSITY = {"mixed": (10.8, 2.1, 2.6), "plain": (4.2, 0.9, 1.5), "batched": (4.2, 0.9, 1.5), "terrain": (6.0, 1.6, 3.0),
           "pile": (2.0, 1.0, 2.5)}
# Contact capacity per body.
CAPACITY = {"mixed": 24, "plain": 16, "batched": 10, "terrain": 32, "pile": 12}


def _states(scene, moving=None):
    """Body states (2 * MOVES, 17 * bodies) of the motion out and back."""
    drv = S.KinematicDriver(scene, dt=DT)
    poses = [(drv.p.copy(), drv.q.copy(), drv.c.copy())]
    for _ in range(MOVES):
        drv.advance(moving)
        poses.append((drv.p.copy(), drv.q.copy(), drv.c.copy()))
    way = list(range(MOVES + 1)) + list(range(MOVES - 1, -1, -1))
    out = np.empty((2 * MOVES, scene.n_bodies, 17), F)
    for k in range(2 * MOVES):
        (_, q0, c0), (p1, q1, _) = poses[way[k]], poses[way[k + 1]]
        out[k, :, 0:3], out[k, :, 3:7], out[k, :, 7:10], out[k, :, 10:14] = p1, q1, c0, q0
        out[k, :, 14:17] = scene.local_center
    return out.reshape(2 * MOVES, -1)


def _pinned(shape, dtype):
    return torch.zeros(shape, dtype=dtype, pin_memory=True)


def _solver_bodies(rng, scene):
    """b3g_solver_body records: the state of the bodies at rest in their first pose."""
    n = scene.n_bodies
    b = np.zeros(n, N.SOLVER_BODY_DTYPE)
    b["x"], b["q"] = S.xf_apply(scene.body_pos, scene.body_quat, scene.local_center), scene.body_quat
    b["v"], b["w"], b["localCenter"] = scene.body_lin, scene.body_ang, scene.local_center
    dyn = scene.body_type == N.BODY_DYNAMIC
    b["invMass"] = np.where(dyn, 1.0 / rng.uniform(0.5, 5.0, n), 0.0)
    inertia = rng.uniform(0.5, 2.0, (n, 3))
    for k in range(3):
        b["invI"][:, 4 * k] = np.where(dyn, inertia[:, k], 0.0)
    return b


def _prepare_step(case, rng):
    scene = _scene(case, rng)
    nb, nf = scene.n_bodies, scene.n_fixtures
    cap = max(1024, CAPACITY[case["scene"]] * nf)
    pipe = CollisionPipeline(scene, max_contacts=cap, graph=bool(case["graph"]))
    asleep = case.get("asleep", 0.0)
    awake = None
    if asleep:
        awake = (rng.random(nb) >= asleep).astype(np.uint8)
    states = _states(scene, awake)
    st = dict(case=case, pipe=pipe, at=0, awake=awake)
    if case["io"] == "host":
        if case["pinned"]:
            t = _pinned(states.shape, torch.float32)
            t.numpy()[...] = states
            st["keep"] = t
            states = t.numpy()
        st["states"] = states
        # Result buffers: room for 4 touching manifolds and 7 points a body.
        touch = max(1024, 4 * nb)
        make = _pinned if case["pinned"] else (lambda shape, dtype: torch.zeros(shape, dtype=dtype))
        st["out"] = [make((cap, 3), torch.int32), make((touch,), torch.int32), make((touch * 158,), torch.uint8)]
        st["np"] = [t.numpy().view(np.uint32) if t.dtype == torch.int32 else t.numpy() for t in st["out"]]
        if case["impulses"]:
            st["impulses"] = [rng.uniform(0, 1, (cap, 4)).astype(F), rng.normal(0, 0.2, (cap, 2)).astype(F),
                              rng.normal(0, 0.2, cap).astype(F)]
        st["contacts"] = 0
    else:
        st["states"] = torch.from_numpy(states).cuda()
        st["bodies"] = torch.from_numpy(_solver_bodies(rng, scene).view(np.uint8).reshape(nb, 112)).cuda()
        rows = max(1024, 4 * nb)
        st["con"] = torch.zeros((rows, 32), dtype=torch.float32, device="cuda")
        st["man"] = torch.zeros((rows, 116), dtype=torch.float32, device="cuda")
        st["counts"] = torch.zeros(2, dtype=torch.int32, device="cuda")
    # The passes of a program's first frames: proxies created, passes captured.
    for _ in range(4):
        _run_step(st)
    torch.cuda.synchronize()
    pipe.counts()
    return st


def _run_step(st):
    case, pipe = st["case"], st["pipe"]
    state = st["states"][st["at"]]
    st["at"] = (st["at"] + 1) % (2 * MOVES)
    if case["io"] == "host":
        if case["impulses"] and st["contacts"]:
            n = st["contacts"]
            pipe.load_impulses(*[a[:n] for a in st["impulses"]])
        if st["awake"] is not None:
            pipe.set_awake(st["awake"])
        pipe.collide(state)
        contacts, index, packed = st["np"]
        c = pipe.fetch_results_packed_async(contacts, index, packed)
        pipe.wait_results()
        st["contacts"] = c["contacts"]
        return dict(contacts=contacts, index=index, packed=packed, counts=np.array(list(c.values()), np.int64))
    pipe.collide(state.data_ptr(), on_device=True)
    con, man = st["con"], st["man"]
    pipe._check(pipe.lib.b3g_contact_constraints_device(
        pipe.ctx, 0, None, ctypes.c_void_p(st["bodies"].data_ptr()), 1.0, 1, ctypes.c_void_p(con.data_ptr()), len(con),
        ctypes.c_void_p(man.data_ptr()), len(man), ctypes.c_void_p(st["counts"].data_ptr()), None))
    ci, mi = con.view(torch.int32), man.view(torch.int32)
    # The records' fields by type (the rest of a record is padding).
    return dict(counts=st["counts"], bodies=ci[:, 0:4], masses=con[:, 4:28], contact=ci[:, 28], manifold=man[:, 0:26],
                points=mi[:, 26:28], rows=man[:, 32:116])


# ---------------------------------------------------------------------------
# Serving.


def _prepare_serve(case, rng):
    worlds = case["worlds"]
    engine = V.ServingEngine(capacity=max(4096, 512 * worlds), max_worlds=max(64, 2 * worlds), active_quantum=4096)
    templates = V.make_templates(engine, 24, int(rng.integers(1 << 30)), lo=32, hi=1024)
    picks = rng.integers(0, len(templates), 4096)
    passes = rng.integers(1, 17, 4096)
    st = dict(case=case, engine=engine, templates=templates, picks=picks, passes=passes, next=0)
    for _ in range(12):
        _run_serve(st)
    return st


def _run_serve(st):
    e = st["engine"]
    while len(e.resident) < st["case"]["worlds"]:
        k = st["next"]
        r = V.Request(k, st["templates"][st["picks"][k % 4096]], int(st["passes"][k % 4096]), 0.0)
        if not e.admit(r):
            break
        st["next"] = k + 1
    # At most two steps under way; which further steps poll() finds finished
    # depends on the moment, so the per-world counts are the outputs.
    while e.in_flight() >= 2:
        e.poll(block=True)
    slot = e.slot
    e.step()
    return dict(counts=e.counts_dev[slot], state=e.state)


# ---------------------------------------------------------------------------
# World queries.


def _query_world(case, rng):
    return _mixed(rng, case["bodies"])


def _query_pipe(scene, queries):
    pipe = CollisionPipeline(scene, max_contacts=max(24 * scene.n_fixtures, queries, 1024))
    drv = S.KinematicDriver(scene, dt=DT)
    pipe.collide(drv.state17())
    pipe.counts()
    return pipe


def _rays(rng, n, bodies):
    half = 24.5 * (bodies / 65536.0) ** (1.0 / 3.0)
    p1 = rng.uniform(-half, half, (n, 3))
    d = rng.normal(size=(n, 3))
    d *= 10.0 / np.linalg.norm(d, axis=1, keepdims=True)
    return np.ascontiguousarray(np.concatenate([p1, p1 + d], axis=1), F)


def _prepare_rays(case, rng):
    scene = _query_world(case, rng)
    pipe = _query_pipe(scene, case["rays"])
    rays = _rays(rng, case["rays"], case["bodies"])
    st = dict(case=case, pipe=pipe, rays=rays)
    if case["io"] == "device":
        st["rays"] = torch.from_numpy(rays).cuda()
        st["fixture"] = torch.zeros(case["rays"], dtype=torch.int32, device="cuda")
        st["hit"] = torch.zeros((case["rays"], 7), dtype=torch.float32, device="cuda")
    return st


def _run_rays(st):
    pipe = st["pipe"]
    if st["case"]["io"] == "host":
        fixture, hit = pipe.ray_cast_single(st["rays"])
        return dict(fixture=fixture, hit=hit)
    p = [ctypes.c_void_p(st[k].data_ptr()) for k in ("rays", "fixture", "hit")]
    pipe._check(pipe.lib.b3g_ray_cast_single_device(pipe.ctx, len(st["rays"]), p[0], None, p[1], p[2], None))
    return dict(fixture=st["fixture"], hit=st["hit"])


def _prepare_casts(case, rng):
    scene = _query_world(case, rng)
    n = case["casts"]
    pipe = _query_pipe(scene, n)
    half = 24.5 * (case["bodies"] / 65536.0) ** (1.0 / 3.0)
    pick = rng.integers(0, scene.n_fixtures, n)
    c = np.zeros(n, N.SHAPE_CAST_DTYPE)
    c["type"], c["hull"], c["params"] = scene.fix_type[pick], scene.fix_hull[pick], scene.fix_params.reshape(-1, 12)[pick]
    c["position"] = rng.uniform(-half, half, (n, 3))
    c["rotation"] = S.random_quats(rng, n)
    d = rng.normal(size=(n, 3))
    c["displacement"] = d * (rng.uniform(1.0, 4.0, (n, 1)) / np.linalg.norm(d, axis=1, keepdims=True))
    return dict(case=case, pipe=pipe, casts=torch.from_numpy(c.view(np.uint8).reshape(n, 112)).cuda(),
                fixture=torch.zeros((n, 2), dtype=torch.int32, device="cuda"),
                hit=torch.zeros((n, 7), dtype=torch.float32, device="cuda"))


def _run_casts(st):
    pipe = st["pipe"]
    p = [ctypes.c_void_p(st[k].data_ptr()) for k in ("casts", "fixture", "hit")]
    pipe._check(pipe.lib.b3g_shape_cast_single_device(pipe.ctx, len(st["casts"]), *p, None))
    return dict(fixture=st["fixture"], hit=st["hit"])


def _convex_shapes(rng, n, hulls):
    types = rng.choice(np.array([N.SHAPE_SPHERE, N.SHAPE_CAPSULE, N.SHAPE_TRIANGLE, N.SHAPE_HULL]), n,
                       p=[0.25, 0.25, 0.15, 0.35])
    params = np.zeros((n, 12), F)
    sph, cap, tri = (types == t for t in (N.SHAPE_SPHERE, N.SHAPE_CAPSULE, N.SHAPE_TRIANGLE))
    params[sph, :3], params[sph, 3] = rng.uniform(-0.1, 0.1, (sph.sum(), 3)), rng.uniform(0.2, 0.8, sph.sum())
    h = rng.uniform(0.2, 0.8, cap.sum())
    params[cap, 1], params[cap, 4], params[cap, 6] = -h, h, rng.uniform(0.1, 0.4, cap.sum())
    params[tri, :9] = rng.uniform(-0.8, 0.8, (tri.sum(), 9))
    return types, params, np.where(types == N.SHAPE_HULL, rng.integers(0, hulls, n), 0)


def _toi_queries(rng, n, hulls):
    """Sweep pairs as S.toi_queries makes them: A moves toward the middle and
    turns a little, B drifts near the middle."""
    q = np.zeros(n, N.TOI_INPUT_DTYPE)
    for side in "ab":
        q["type_" + side], q["params_" + side], q["hull_" + side] = _convex_shapes(rng, n, hulls)
        sw = q["sweep_" + side]
        sw[:, 0:3] = rng.uniform(-0.1, 0.1, (n, 3))
        q0 = S.unit_quats(rng, n)
        turn = np.concatenate([rng.normal(0, 0.3, (n, 3)), np.ones((n, 1))], axis=1)
        q1 = S.qmul(q0, turn / np.linalg.norm(turn, axis=1, keepdims=True))
        sw[:, 3:7], sw[:, 11:15] = q0, np.where(rng.random((n, 1)) < 0.3, -q1, q1)
        if side == "a":
            c0 = rng.uniform(-3, 3, (n, 3))
            c1 = c0 + (rng.uniform(-1, 1, (n, 3)) - c0) * rng.uniform(0.5, 2.5, (n, 1))
        else:
            c0 = rng.uniform(-0.5, 0.5, (n, 3))
            c1 = c0 + rng.normal(0, 0.3, (n, 3))
        sw[:, 7:10], sw[:, 15:18] = c0, c1
    q["t_max"] = 1.0
    return q


def _prepare_toi(case, rng):
    n = case["queries"]
    pool = _hulls(rng, S.HullPool(), 256, (8, 32), (0.3, 1.0))
    one = np.ones((1, 4), F)
    scene = _assemble(pool, [0], [N.BODY_DYNAMIC], [(0, 0, 0)], 0.5 * one, [(0, 0, 0)], [(0, 0, 0)], [N.SHAPE_HULL], [0],
                      np.zeros((1, 12), F))
    pipe = CollisionPipeline(scene, max_contacts=1024)
    q = _toi_queries(rng, n, len(pool))
    return dict(case=case, pipe=pipe, queries=torch.from_numpy(q.view(np.uint8).reshape(n, 272)).cuda(),
                out=torch.zeros((n, 4), dtype=torch.int32, device="cuda"))


def _run_toi(st):
    pipe, out = st["pipe"], st["out"]
    pipe._check(pipe.lib.b3g_time_of_impact_device(pipe.ctx, len(out), ctypes.c_void_p(st["queries"].data_ptr()),
                                                   ctypes.c_void_p(out.data_ptr()), None))
    return dict(state=out[:, 0], t=out.view(torch.float32)[:, 1], iterations=out[:, 2])


PREPARE = dict(step=_prepare_step, serve=_prepare_serve, rays=_prepare_rays, casts=_prepare_casts, toi=_prepare_toi)
RUN = dict(step=_run_step, serve=_run_serve, rays=_run_rays, casts=_run_casts, toi=_run_toi)


def prepare(case, seed):
    return PREPARE[case["call"]](case, np.random.default_rng(seed))


def run(state):
    return RUN[state["case"]["call"]](state)


def work(case):
    """Bytes: each input read once (body states, fixtures, hulls, the previous
    contacts' manifolds), each output written once. Flops: the closed-form and
    iterative routines per contact or query, roughly."""
    call = case["call"]
    if call == "step":
        n = case["bodies"] if "bodies" in case else 713 * case["worlds"]
        contacts, touching, points = (n * d for d in DENSITY[case["scene"]])
        size = n * (17 * 4 + 60 + 64) + contacts * (12 + 8) + 2 * (32 * touching + 72 * points)
        if case["io"] == "device":
            size += n * 112 + touching * (128 + 464)
        return {"bytes": size, "flops": 800.0 * contacts}
    if call == "serve":
        n = 285 * case["worlds"]
        return {"bytes": n * (17 * 4 * 3 + 60 + 64) + 4.2 * n * 20 + n * (32 * 0.9 + 72 * 1.5) * 2, "flops": 3500.0 * n}
    if call == "rays":
        return {"bytes": case["rays"] * (24 + 32) + case["bodies"] * 150, "flops": 500.0 * case["rays"]}
    if call == "casts":
        return {"bytes": case["casts"] * (112 + 36) + case["bodies"] * 150, "flops": 5000.0 * case["casts"]}
    return {"bytes": case["queries"] * (272 + 16), "flops": 10000.0 * case["queries"]}


# ---------------------------------------------------------------------------
# Ray casts in 64 bits.


def _rotate(q, v):
    u, s = q[..., :3], q[..., 3:]
    t = 2 * torch.linalg.cross(u, v)
    return v + s * t + torch.linalg.cross(u, t)


def _ray_sphere(m, d, r):
    """Entry fraction of rays from m (relative to the centre) along d; inf for a miss or a start inside."""
    a, b, c = (d * d).sum(-1), (m * d).sum(-1), (m * m).sum(-1) - r * r
    disc = b * b - a * c
    t = (-b - disc.clamp(min=0).sqrt()) / a
    return torch.where((disc >= 0) & (t > 0) & (t <= 1), t, torch.inf)


def exact(case, seed):
    if case["call"] != "rays":
        return None
    rng = np.random.default_rng(seed)
    sc = _query_world(case, rng)
    rays = torch.from_numpy(_rays(rng, case["rays"], case["bodies"])).cuda().double()
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    pos, quat = dev(sc.body_pos).double(), dev(sc.body_quat).double()
    params, ftype = dev(sc.fix_params.reshape(-1, 12)).double(), dev(sc.fix_type.astype(np.int64))
    ha = sc.hull_arrays
    desc = ha["desc"].reshape(-1, 6).astype(np.int64)
    vpad = np.minimum(np.arange(desc[:, 1].max())[None], desc[:, 1:2] - 1) + desc[:, 0:1]
    reach = np.linalg.norm(ha["verts"].reshape(-1, 3)[vpad].astype(np.float64), axis=2).max(axis=1)
    ppad = dev(np.minimum(np.arange(desc[:, 5].max())[None], desc[:, 5:6] - 1) + desc[:, 4:5])
    planes = dev(ha["planes"].reshape(-1, 4)).double()
    hull = dev(sc.fix_hull.astype(np.int64))
    # Distance from its origin that each fixture stays within.
    bound = torch.where(ftype == N.SHAPE_SPHERE, params[:, 3], torch.where(
        ftype == N.SHAPE_CAPSULE, params[:, 4] + params[:, 6], dev(reach)[hull])) * 1.001 + 1e-3
    n, nf = len(rays), len(pos)
    best = torch.full((n,), torch.inf, dtype=torch.float64, device="cuda")
    normal = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
    pos32, bound32 = pos.float(), bound.float()
    step = max(1, (1 << 26) // nf)
    for i0 in range(0, n, step):
        a, d = rays[i0:i0 + step, :3], rays[i0:i0 + step, 3:] - rays[i0:i0 + step, :3]
        # Fixtures whose bounding sphere comes near the segment.
        a32, d32 = a.float(), d.float()
        dd = (d32 * d32).sum(-1, keepdim=True)
        t = ((d32 @ pos32.T) - (a32 * d32).sum(-1, keepdim=True)) / dd
        t = t.clamp(0, 1)
        gap = torch.zeros_like(t)
        for k in range(3):
            gap += (a32[:, k, None] + t * d32[:, k, None] - pos32[None, :, k]).square()
        ri, fi = torch.nonzero(gap <= (bound32 + 0.02).square()[None], as_tuple=True)
        A, D, q, p, prm = a[ri], d[ri], quat[fi], pos[fi], params[fi]
        frac = torch.full((len(ri),), torch.inf, dtype=torch.float64, device="cuda")
        nrm = torch.zeros((len(ri), 3), dtype=torch.float64, device="cuda")
        k = torch.nonzero(ftype[fi] == N.SHAPE_SPHERE)[:, 0]
        m = A[k] - p[k]
        frac[k] = _ray_sphere(m, D[k], prm[k, 3])
        hit = torch.where(frac[k].isfinite(), frac[k], 0.0)[:, None]
        nrm[k] = m + hit * D[k]
        k = torch.nonzero(ftype[fi] == N.SHAPE_CAPSULE)[:, 0]
        P, Q, r = p[k] + _rotate(q[k], prm[k, 0:3]), p[k] + _rotate(q[k], prm[k, 3:6]), prm[k, 6]
        ax, m, v = Q - P, A[k] - P, D[k]
        dd2, nn, nd = (ax * ax).sum(-1), (v * v).sum(-1), (v * ax).sum(-1)
        md, mn, mm = (m * ax).sum(-1), (m * v).sum(-1), (m * m).sum(-1)
        ca, cb, cc = dd2 * nn - nd * nd, dd2 * mn - nd * md, dd2 * (mm - r * r) - md * md
        disc = cb * cb - ca * cc
        tc = (-cb - disc.clamp(min=0).sqrt()) / ca
        ok = (disc >= 0) & (tc >= 0) & (tc <= 1)
        along = md + tc * nd
        end = torch.where((along < 0)[:, None], P, Q)
        side = ok & (along >= 0) & (along <= dd2)
        cap = torch.where(ok & ~side, _ray_sphere(A[k] - end, v, r), torch.inf)
        frac[k] = torch.where(side, tc, cap)
        hit = torch.where(frac[k].isfinite(), frac[k], 0.0)[:, None]
        point = A[k] + hit * v
        on = P + ((point - P) * ax).sum(-1, keepdim=True).div(dd2[:, None]).clamp(0, 1) * ax
        nrm[k] = point - on
        k = torch.nonzero(ftype[fi] == N.SHAPE_HULL)[:, 0]
        inv = q[k] * torch.tensor([-1.0, -1.0, -1.0, 1.0], dtype=torch.float64, device="cuda")
        lp, ld = _rotate(inv, A[k] - p[k]), _rotate(inv, D[k])
        lo, hi = torch.zeros(len(k), dtype=torch.float64, device="cuda"), torch.ones(len(k), dtype=torch.float64, device="cuda")
        face = torch.full((len(k),), -1, dtype=torch.int64, device="cuda")
        miss = torch.zeros(len(k), dtype=torch.bool, device="cuda")
        pl = ppad[hull[fi[k]]]
        for j in range(pl.shape[1]):
            w = planes[pl[:, j]]
            num, den = w[:, 3] - (w[:, :3] * lp).sum(-1), (w[:, :3] * ld).sum(-1)
            ratio = num / den
            miss |= (den == 0) & (num < 0)
            enter = (den < 0) & (ratio > lo)
            face = torch.where(enter, pl[:, j], face)
            lo = torch.where(enter, ratio, lo)
            hi = torch.where((den > 0) & (ratio < hi), ratio, hi)
        got = ~miss & (face >= 0) & (lo <= hi)
        frac[k] = torch.where(got, lo, torch.inf)
        nrm[k] = _rotate(q[k], planes[face.clamp(min=0), :3])
        # The first hit of each ray.
        least = torch.full((len(a),), torch.inf, dtype=torch.float64, device="cuda").scatter_reduce(
            0, ri, frac, "amin", include_self=True)
        first = torch.nonzero((frac == least[ri]) & frac.isfinite())[:, 0]
        best[i0:i0 + step] = least
        normal[i0 + ri[first]] = nrm[first] / nrm[first].norm(dim=-1, keepdim=True)
    found = best.isfinite()
    t = torch.where(found, best, 0.0)[:, None]
    point = torch.where(found[:, None], (1 - t) * rays[:, :3] + t * rays[:, 3:], 0.0)
    return dict(fixture=None, hit=torch.cat([point, normal, t], dim=1))
