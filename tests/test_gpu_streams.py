"""GPU: one context's calls over several streams and under capture: what a call
leaves under way when it returns may not be overtaken by the next one, and what
could be captured or run asynchronously still can."""
import numpy as np
import pytest

from bounce_b200 import _native as N
from bounce_b200 import scene as S
from bounce_b200.pipeline import CollisionPipeline

pytestmark = pytest.mark.gpu


def mixed(n):
    return S.mixed_scene(seed=n, n=n, side=max(3.0, 49.0 * (n / 65536.0) ** (1 / 3))).finalize()


def states_of(sc, passes):
    drv = S.KinematicDriver(sc)
    out = []
    for _ in range(passes):
        out.append(drv.state17().copy())
        drv.advance()
    return out


def packed_of(manifolds):
    return b"".join(m.tobytes()[288:] + m["points"][: int(m["pointCount"])].tobytes() for m in manifolds)


# The results of a pass are packed while the next pass already runs on the
# caller's stream; the largest packs for longer than that pass takes to clear
# its counters. Spheres apart: contacts, but nothing to pack.
@pytest.mark.parametrize("kind,n", [("mixed", 30), ("mixed", 3000), ("mixed", 30000), ("apart", 2000)])
@pytest.mark.parametrize("graph", [False, True])
def test_packed_results_beside_the_next_pass(kind, n, graph):
    torch = pytest.importorskip("torch")
    if kind == "mixed":
        sc = mixed(n)
    else:
        sc = S.Scene()
        for i in range(n):
            b = sc.add_body(0, N.BODY_DYNAMIC, (1.1 * (i % 50), 1.1 * (i // 50), 0), (0, 0, 0, 1), lin=(0, 0, 1 + i % 3))
            sc.add_fixture(b, N.SHAPE_SPHERE, [0, 0, 0, 0.5])
        sc.finalize()
    states = states_of(sc, 8)
    ref = CollisionPipeline(sc)
    want = []
    for st in states:
        ref.collide(st)
        index, man = ref.touching()
        want.append((ref.contacts(), index, packed_of(man)))
    ref.close()
    pipe = CollisionPipeline(sc, graph=graph)
    s = torch.cuda.Stream()
    on_device = [torch.from_numpy(st).cuda() for st in states]
    room = max(len(w[2]) for w in want) + 8
    make = lambda shape, dt: torch.zeros(shape, dtype=dt, pin_memory=True).numpy()
    contacts = make((max(len(w[0]) for w in want), 3), torch.int32).view(np.uint32)
    index = make((max(len(w[1]) for w in want) + 1,), torch.int32).view(np.uint32)
    packed = make((room,), torch.uint8)
    torch.cuda.synchronize()
    pipe.collide(on_device[0].data_ptr(), on_device=True, stream=s.cuda_stream)
    for k, (c, i, p) in enumerate(want):
        s.synchronize()
        counts = pipe.fetch_results_packed_async(contacts, index, packed)
        if k + 1 < len(states):
            pipe.collide(on_device[k + 1].data_ptr(), on_device=True, stream=s.cuda_stream)
        pipe.wait_results()
        assert counts["contacts"] == len(c) and counts["manifolds"] == len(i)
        assert np.array_equal(contacts[: len(c)], c)
        assert np.array_equal(index[: len(i)], i)
        assert packed[: len(p)].tobytes() == p
    pipe.close()


# A pass on the context's own stream, its results being packed, then a pass on a
# caller's.
def test_packed_results_before_a_pass_on_another_stream():
    torch = pytest.importorskip("torch")
    sc = mixed(30000)
    states = states_of(sc, 6)
    ref = CollisionPipeline(sc)
    pipe = CollisionPipeline(sc)
    s = torch.cuda.Stream()
    on_device = [torch.from_numpy(st).cuda() for st in states]
    torch.cuda.synchronize()
    make = lambda shape, dt: torch.zeros(shape, dtype=dt, pin_memory=True).numpy()
    contacts = make((40 * sc.n_fixtures, 3), torch.int32).view(np.uint32)
    index, packed = make((8 * sc.n_fixtures,), torch.int32).view(np.uint32), make((8 * sc.n_fixtures * 320,), torch.uint8)
    for k in range(0, len(states), 2):
        ref.collide(states[k])
        want_index, man = ref.touching()
        want, p = ref.contacts(), packed_of(man)
        pipe.collide(on_device[k].data_ptr(), on_device=True)
        counts = pipe.fetch_results_packed_async(contacts, index, packed)
        pipe.collide(on_device[k + 1].data_ptr(), on_device=True, stream=s.cuda_stream)
        pipe.wait_results()
        assert np.array_equal(contacts[: counts["contacts"]], want)
        assert np.array_equal(index[: counts["manifolds"]], want_index)
        assert packed[: len(p)].tobytes() == p
        ref.collide(states[k + 1])
        s.synchronize()
        assert np.array_equal(pipe.contacts(), ref.contacts())
    ref.close()
    pipe.close()


# Two passes (one of each buffer parity) captured by the caller, after and before
# flags and impulses have been handed in.
@pytest.mark.parametrize("n", [40, 3000])
def test_captured_passes(n):
    torch = pytest.importorskip("torch")
    sc = mixed(n)
    states = states_of(sc, 12)
    ref = CollisionPipeline(sc)
    pipe = CollisionPipeline(sc)
    awake = np.ones(sc.n_bodies, np.uint8)

    def impulses(p, seed):
        k = p.counts()["contacts"]
        motor = np.random.default_rng(seed).uniform(0, 1, k).astype(np.float32)
        p.load_impulses(np.zeros((k, 4), np.float32), np.zeros((k, 2), np.float32), motor)

    for st in states[:2]:
        for p in (ref, pipe):
            p.set_awake(awake)
            p.collide(st)
    for p in (ref, pipe):
        impulses(p, 0)
        p.collide(states[2])
        p.set_awake(awake)
    slots = [torch.from_numpy(states[3]).cuda() for _ in range(2)]
    graph = torch.cuda.CUDAGraph()
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        for x in slots:
            pipe.collide(x.data_ptr(), on_device=True, stream=stream.cuda_stream)
    for k in range(3, 11, 2):
        for p in (ref, pipe):
            p.set_awake(awake)
        for j, x in enumerate(slots):
            x.copy_(torch.from_numpy(states[k + j]))
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        ref.collide(states[k])
        ref.collide(states[k + 1])
        assert np.array_equal(pipe.contacts(), ref.contacts())
        assert pipe.manifolds().tobytes() == ref.manifolds().tobytes()
        assert np.array_equal(pipe.caches(), ref.caches())
    graph.reset()
    ref.close()
    pipe.close()


# Flags handed in between the halves of a filtered pass, on a caller's stream
# as on the context's.
def test_flags_between_the_halves_of_a_pass():
    torch = pytest.importorskip("torch")
    sc = mixed(20000)
    states = states_of(sc, 5)
    rng = np.random.default_rng(1)
    flags = [(rng.random(sc.n_bodies) < 0.7).astype(np.uint8) for _ in states]
    s = torch.cuda.Stream()
    make = lambda shape, dt: torch.zeros(shape, dtype=dt, pin_memory=True).numpy()
    contacts = make((40 * sc.n_fixtures, 3), torch.int32).view(np.uint32)
    index, packed = make((8 * sc.n_fixtures,), torch.int32).view(np.uint32), make((8 * sc.n_fixtures * 320,), torch.uint8)
    out = []
    for stream in (None, s.cuda_stream):
        pipe = CollisionPipeline(sc, contact_filter=True)
        got = []
        for st, awake in zip(states, flags):
            x = torch.from_numpy(st).cuda()
            torch.cuda.synchronize()
            pipe.collide(x.data_ptr(), on_device=True, stream=stream)
            pipe.new_pairs()
            pipe.set_awake(awake)
            pipe.finish_pass()
            s.synchronize()
            pipe.fetch_results_packed_async(contacts, index, packed)
            got.append((pipe.contacts(), pipe.manifolds().tobytes(), pipe.awake()))
        out.append(got)
        pipe.close()
    for a, b in zip(*out):
        assert np.array_equal(a[0], b[0]) and a[1] == b[1] and np.array_equal(a[2], b[2])


# Scene updates after a pass with sleeping bodies: asynchronous on their stream
# (they wait for no work of others), and the next pass sees their bodies awake.
@pytest.mark.parametrize("how", ["host", "device", "swap"])
def test_updates_after_a_pass_with_sleepers(how):
    torch = pytest.importorskip("torch")
    sc = mixed(600)
    states = states_of(sc, 4)
    rng = np.random.default_rng(3)
    awake = (rng.random(sc.n_bodies) < 0.5).astype(np.uint8)
    first, count = 100, 30
    b = np.arange(first, first + count, dtype=np.uint32)
    world, btype = sc.body_world[b], sc.body_type[b]
    ftype, fhull, fflags = sc.fix_type[b], sc.fix_hull[b], sc.fix_flags[b]
    fparams = np.ascontiguousarray(sc.fix_params.reshape(-1, 12)[b])
    assert np.array_equal(sc.fix_body[b], b)
    other, mine = torch.cuda.Stream(), torch.cuda.Stream()
    results = []
    for busy in (False, True):
        pipe = CollisionPipeline(sc)
        pipe.collide(states[0])
        pipe.set_awake(awake)
        pipe.collide(states[1])
        p = lambda a: a.ctypes.data_as(N.ctypes.c_void_p)
        dev = [torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1)).cuda()
               for a in (b, world, btype, b, b, ftype, fhull, fparams, fflags, b - first)]
        d = [N.ctypes.c_void_p(x.data_ptr()) for x in dev]
        rows = torch.zeros((sc.n_bodies, 17), device="cuda")
        torch.cuda.synchronize()
        if busy:
            with torch.cuda.stream(other):
                torch.cuda._sleep(400_000_000)
        s = N.ctypes.c_void_p(mine.cuda_stream)
        if how == "host":
            u32, u8, f32 = N.ctypes.c_uint32, N.ctypes.c_uint8, N.ctypes.c_float
            on = np.ones(count, np.uint8)
            pipe._check(pipe.lib.b3g_update_scene(
                pipe.ctx, count, N.ptr(b, u32), N.ptr(world, u32), N.ptr(btype, u32), N.ptr(on, u8), count,
                N.ptr(b, u32), N.ptr(b, u32), N.ptr(ftype, u32), N.ptr(fhull, u32), N.ptr(fparams, f32),
                N.ptr(fflags, u32), 0, None, s))
        elif how == "device":
            pipe._check(pipe.lib.b3g_update_scene_device(
                pipe.ctx, count, d[0], d[1], d[2], count, d[3], d[4], d[5], d[6], d[7], d[8], 0, None, s))
        else:
            admit = np.array([[first, count, 0, 0]], np.uint32)
            t = N.WorldTemplates(*(x.value for x in (d[2], d[9], d[5], d[6], d[8], d[7])), rows.data_ptr(), rows.data_ptr())
            pipe._check(pipe.lib.b3g_swap_worlds(
                pipe.ctx, 0, None, 1, p(admit), N.ctypes.byref(t), N.ctypes.c_void_p(rows.data_ptr()),
                N.ctypes.c_void_p(rows.data_ptr()), s))
        assert not busy or not other.query()
        torch.cuda.synchronize()
        assert pipe.awake()[b].all()
        for st in states[2:]:
            pipe.collide(st)
        results.append((pipe.contacts(), pipe.awake(), pipe.pass_stats()["asleep"]))
        assert results[-1][2] == int(((results[-1][1] == 0) & (sc.body_type != N.BODY_STATIC)).sum())
        pipe.close()
    assert np.array_equal(results[0][0], results[1][0]) and np.array_equal(results[0][1], results[1][1])


# The constraints of a scene without sensors are captured; then some fixtures
# become sensors, and the replay leaves their contacts out.
def test_captured_constraints_see_new_sensors():
    torch = pytest.importorskip("torch")
    sc = mixed(1500)
    states = states_of(sc, 6)
    pipe = CollisionPipeline(sc)
    bodies = np.zeros(sc.n_bodies, N.SOLVER_BODY_DTYPE)
    bodies["x"], bodies["q"], bodies["invMass"] = sc.body_pos, sc.body_quat, 1.0
    room = 8 * sc.n_fixtures
    vp = N.ctypes.c_void_p
    dev = [torch.from_numpy(bodies.view(np.uint8).copy()).cuda(), torch.zeros(room * 128, dtype=torch.uint8, device="cuda"),
           torch.zeros(room * 464, dtype=torch.uint8, device="cuda"), torch.zeros(2, dtype=torch.int32, device="cuda")]
    b, con, man, counts = (vp(x.data_ptr()) for x in dev)
    stream = torch.cuda.Stream()

    def build(s):
        pipe._check(pipe.lib.b3g_contact_constraints_device(pipe.ctx, 0, None, b, 1.0, 1, con, room, man, room, counts, s))

    for st in states[:2]:
        pipe.collide(st)
    torch.cuda.synchronize()
    build(vp(stream.cuda_stream))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        build(vp(stream.cuda_stream))
    before, _ = pipe.contact_constraints(bodies)
    f = np.arange(0, sc.n_fixtures, 3, dtype=np.uint32)
    u32, f32 = N.ctypes.c_uint32, N.ctypes.c_float
    flags = np.full(len(f), N.FIXTURE_SENSOR, np.uint32)
    arrays = [np.ascontiguousarray(a) for a in (sc.fix_body[f], sc.fix_type[f], sc.fix_hull[f])]
    params = np.ascontiguousarray(sc.fix_params.reshape(-1, 12)[f])
    pipe._check(pipe.lib.b3g_update_scene(
        pipe.ctx, 0, None, None, None, None, len(f), N.ptr(f, u32), *(N.ptr(a, u32) for a in arrays),
        N.ptr(params, f32), N.ptr(flags, u32), 0, None, None))
    for st in states[2:4]:
        pipe.collide(st)
    want, want_man = pipe.contact_constraints(bodies)
    assert 0 < len(want) < len(before)
    graph.replay()
    torch.cuda.synchronize()
    n, m = dev[3].cpu().numpy().tolist()
    assert (n, m) == (len(want), len(want_man))
    assert dev[1].cpu().numpy()[: n * 128].tobytes() == want.tobytes()
    assert dev[2].cpu().numpy()[: m * 464].tobytes() == want_man.tobytes()
    graph.reset()
    pipe.close()


# The first sensors of a scene come with an update, after its passes have been
# captured.
def test_first_sensors_after_captured_passes():
    torch = pytest.importorskip("torch")
    sc = mixed(1500)
    states = states_of(sc, 10)
    f = np.arange(0, sc.n_fixtures, 2, dtype=np.uint32)
    u32, f32 = N.ctypes.c_uint32, N.ctypes.c_float
    flags = np.full(len(f), N.FIXTURE_SENSOR, np.uint32)
    arrays = [np.ascontiguousarray(a) for a in (sc.fix_body[f], sc.fix_type[f], sc.fix_hull[f])]
    params = np.ascontiguousarray(sc.fix_params.reshape(-1, 12)[f])
    out = []
    for graph in (False, True):
        pipe = CollisionPipeline(sc, graph=graph)
        got = []
        for k, st in enumerate(states):
            if k == 5:
                pipe._check(pipe.lib.b3g_update_scene(
                    pipe.ctx, 0, None, None, None, None, len(f), N.ptr(f, u32), *(N.ptr(a, u32) for a in arrays),
                    N.ptr(params, f32), N.ptr(flags, u32), 0, None, None))
            x = torch.from_numpy(st).cuda()
            torch.cuda.synchronize()
            pipe.collide(x.data_ptr(), on_device=True)
            got.append((pipe.contacts(), pipe.manifolds().tobytes()))
        assert (pipe.totals()["graph_passes"] > 0) == graph
        out.append(got)
        pipe.close()
    for a, b in zip(*out):
        assert np.array_equal(a[0], b[0]) and a[1] == b[1]


# An update from device memory captured after a pass with sleeping bodies, and
# replayed (once: the tree is rebuilt for the call, the host sees no replay).
@pytest.mark.parametrize("graph_passes", [False, True])
def test_captured_update(graph_passes):
    torch = pytest.importorskip("torch")
    sc = mixed(600)
    states = states_of(sc, 8)
    pipe, ref = CollisionPipeline(sc, graph=graph_passes), CollisionPipeline(sc)
    awake = np.ones(sc.n_bodies, np.uint8)
    awake[::3] = 0
    on_device = [torch.from_numpy(st).cuda() for st in states]
    torch.cuda.synchronize()
    for p in (pipe, ref):
        for x in on_device[:3]:
            p.collide(x.data_ptr(), on_device=True)
        p.set_awake(awake)
        p.collide(on_device[3].data_ptr(), on_device=True)
    b = np.arange(0, 60, 2, dtype=np.uint32)
    fixtures = [sc.fix_type[b], sc.fix_hull[b], np.ascontiguousarray(sc.fix_params.reshape(-1, 12)[b]), sc.fix_flags[b]]
    dev = [torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1)).cuda()
           for a in (b, sc.body_world[b], sc.body_type[b], *fixtures)]
    idx, world, btype, ftype, fhull, fparams, fflags = (N.ctypes.c_void_p(x.data_ptr()) for x in dev)

    def update(p, s):
        p._check(p.lib.b3g_update_scene_device(p.ctx, len(b), idx, world, btype, len(b), idx, idx, ftype, fhull, fparams,
                                               fflags, 0, None, s))

    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        update(pipe, N.ctypes.c_void_p(stream.cuda_stream))
    graph.replay()
    update(ref, None)
    torch.cuda.synchronize()
    assert pipe.awake()[b].all()
    for x in on_device[4:]:
        pipe.collide(x.data_ptr(), on_device=True)
        ref.collide(x.data_ptr(), on_device=True)
        assert np.array_equal(pipe.contacts(), ref.contacts())
        assert np.array_equal(pipe.awake(), ref.awake())
        assert pipe.manifolds().tobytes() == ref.manifolds().tobytes()
    graph.reset()
    pipe.close()
    ref.close()


# The fetches wait for a pass on a caller's stream by themselves.
@pytest.mark.parametrize("packed_form", [False, True])
@pytest.mark.parametrize("how", ["launched", "graphs", "captured", "filtered"])
def test_results_of_a_pass_under_way(packed_form, how):
    torch = pytest.importorskip("torch")
    sc = mixed(20000)
    states = states_of(sc, 8)
    ref = CollisionPipeline(sc)
    pipe = CollisionPipeline(sc, graph=how == "graphs", contact_filter=how == "filtered")
    make = lambda shape, dt: torch.zeros(shape, dtype=dt, pin_memory=True).numpy()
    contacts = make((40 * sc.n_fixtures, 3), torch.int32).view(np.uint32)
    index = make((4 * sc.n_fixtures,), torch.int32).view(np.uint32)
    packed = make((4 * sc.n_fixtures * 320,), torch.uint8)
    full = packed.view(N.MANIFOLD_DTYPE)
    s = torch.cuda.Stream()
    on_device = [torch.from_numpy(st).cuda() for st in states]
    slots = [x.clone() for x in on_device[:2]]
    torch.cuda.synchronize()

    def check():
        c = (pipe.fetch_results_packed_async(contacts, index, packed) if packed_form else
             pipe.fetch_results_async(contacts, index, full))
        pipe.wait_results()
        want_index, man = ref.touching()
        assert np.array_equal(contacts[: c["contacts"]], ref.contacts())
        assert np.array_equal(index[: c["manifolds"]], want_index)
        got = packed[: len(packed_of(man))].tobytes() if packed_form else packed_of(full[: c["manifolds"]])
        assert got == packed_of(man)

    graph = None
    for k, (st, x) in enumerate(zip(states, on_device)):
        ref.collide(st)
        if how == "captured" and k >= 2:
            if graph is None:
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, stream=s):
                    for y in slots:
                        pipe.collide(y.data_ptr(), on_device=True, stream=s.cuda_stream)
            if k & 1:
                slots[0].copy_(on_device[k - 1])
                slots[1].copy_(x)
                torch.cuda.synchronize()
                with torch.cuda.stream(s):
                    graph.replay()
                check()
            continue
        pipe.collide(x.data_ptr(), on_device=True, stream=s.cuda_stream)
        if how == "filtered":
            pipe.new_pairs()
            pipe.finish_pass()
        check()
    if graph is not None:
        graph.reset()
    ref.close()
    pipe.close()
