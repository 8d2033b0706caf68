"""GPU: single-hit ray and shape casts on several streams at once, and captured,
give what the same calls give one after another on the context's stream."""
import ctypes

import numpy as np
import pytest

from bounce_b200 import _native as N
from bounce_b200 import scene as S
from bounce_b200.pipeline import CollisionPipeline
from tests.test_gpu_walks import casts_of

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

vp = ctypes.c_void_p


class Query:
    """One batch of rays or casts in device memory."""

    def __init__(self, pipe, sc, kind, n, seed):
        self.pipe, self.kind, self.n = pipe, kind, n
        rng = np.random.default_rng(seed)
        if kind == "rays":
            p = rng.uniform(-8, 8, (n, 3))
            self.host = np.concatenate([p, p + rng.normal(size=(n, 3)) * 5], axis=1).astype(np.float32)
        else:
            self.host = casts_of(sc, n, seed)
        self.data = torch.from_numpy(self.host.view(np.uint8).reshape(-1)).cuda()
        self.fix = torch.zeros(n * (1 if kind == "rays" else 2), dtype=torch.int32, device="cuda")
        self.hit = torch.zeros((n, 7), device="cuda")

    def run(self, stream):
        a, f, h = vp(self.data.data_ptr()), vp(self.fix.data_ptr()), vp(self.hit.data_ptr())
        if self.kind == "rays":
            rc = self.pipe.lib.b3g_ray_cast_single_device(self.pipe.ctx, self.n, a, None, f, h, vp(stream.cuda_stream))
        else:
            rc = self.pipe.lib.b3g_shape_cast_single_device(self.pipe.ctx, self.n, a, f, h, vp(stream.cuda_stream))
        self.pipe._check(rc)

    def check(self):
        want = self.pipe.ray_cast_single(self.host) if self.kind == "rays" else self.pipe.shape_cast_single(self.host)
        assert np.array_equal(self.fix.cpu().numpy().view(np.uint32), want[0].reshape(-1))
        assert self.hit.cpu().numpy().tobytes() == want[1].tobytes()
        self.fix.zero_()
        self.hit.zero_()


def setup(kind):
    if kind == "mixed":
        sc = S.mixed_scene(seed=3, n=3000, side=18.0).finalize()
    else:
        sc = S.terrain_scene(seed=3, n=500)
        sc.body_pos[0] = (0.3, 1.0, -0.2)  # triangles outside their boxes
        sc.finalize()
    pipe = CollisionPipeline(sc, max_contacts=120000)
    drv = S.KinematicDriver(sc)
    pipe.collide(drv.state17())
    queries = [Query(pipe, sc, k, n, i) for i, (k, n) in enumerate(
        [("rays", 100), ("casts", 300), ("rays", 40000), ("casts", 9000), ("rays", 5000), ("casts", 50)])]
    torch.cuda.synchronize()
    return pipe, drv, queries


@pytest.mark.parametrize("kind", ["mixed", "turned"])
def test_queries_side_by_side(kind):
    pipe, drv, queries = setup(kind)
    streams = [torch.cuda.Stream() for _ in queries]
    for _ in range(4):
        for _ in range(3):
            for q, s in zip(queries, streams):
                q.run(s)
        torch.cuda.synchronize()
        for q in queries:
            q.check()
        drv.advance()
        pipe.collide(drv.state17())
        torch.cuda.synchronize()
    pipe.close()


@pytest.mark.parametrize("kind", ["mixed", "turned"])
def test_captured_queries(kind):
    pipe, drv, queries = setup(kind)
    graphs, streams = [], [torch.cuda.Stream() for _ in queries]
    for q, s in zip(queries, streams):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            q.run(s)
            q.run(s)
        graphs.append(g)
    for _ in range(3):
        for g, s in zip(graphs, streams):
            with torch.cuda.stream(s):
                g.replay()
        torch.cuda.synchronize()
        for q in queries:
            q.check()
        drv.advance()
        pipe.collide(drv.state17())  # the replays after it walk its tree
        torch.cuda.synchronize()
    for g in graphs:
        g.reset()
    pipe.close()
