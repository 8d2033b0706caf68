"""GPU: contacts of hulls with small and with large faces in one scene: the pass
that finds a contact (from the separating axes, a warp each) and the next (from
the feature cache, in rings of 8 clip vertices or on a thread each) give the same
points, and without the cache every pass gives the first one's."""
import numpy as np
import pytest

from bounce_b200 import _native as N
from bounce_b200 import scene as S
from bounce_b200.pipeline import CollisionPipeline
from tests.test_gpu_walks import prism

pytestmark = pytest.mark.gpu


# 4 and 4 vertices just fit the rings, 4 and 5 do not.
@pytest.mark.parametrize("sides", [(4, 5), (3, 5), (3, 6), (4, 12), (3, 4, 6, 8, 24)])
@pytest.mark.parametrize("pairs", [2, 129, 2000])
def test_small_and_large_faces(sides, pairs):
    rng = np.random.default_rng(sum(sides) + pairs)
    sc = S.Scene()
    hulls = [sc.hulls.extend(prism(n, 1.0, 0.5)) for n in sides]
    for k in range(pairs):
        x = np.array([5.0 * (k % 50), 0, 5.0 * (k // 50)])
        b = sc.add_body(0, N.BODY_STATIC, x, (0, 0, 0, 1))
        sc.add_fixture(b, N.SHAPE_HULL, [0.02], hull=hulls[rng.integers(len(hulls))])
        turn = rng.uniform(-3, 3) / 2
        x = x + [rng.uniform(-0.5, 0.5), 0.98 + rng.uniform(0, 0.05), rng.uniform(-0.5, 0.5)]
        tilt = np.array([rng.uniform(-0.01, 0.01), np.sin(turn), rng.uniform(-0.01, 0.01), np.cos(turn)])
        b = sc.add_body(0, N.BODY_DYNAMIC, x, tilt / np.linalg.norm(tilt))
        sc.add_fixture(b, N.SHAPE_HULL, [0.02], hull=hulls[rng.integers(len(hulls))])
    sc.finalize()
    state = S.KinematicDriver(sc).state17()
    rounds = []
    for cache in (True, False):
        pipe = CollisionPipeline(sc, max_contacts=4 * pairs + 64, convex_cache=cache)
        for k in range(2):
            pipe.collide(state)
            index, m = pipe.touching()
            order = np.argsort(index)
            rounds.append((pipe.contacts()[index][order], m[order]))
            if k == 1:
                assert (pipe.pass_stats()["hull_miss"] < len(index)) == cache
        pipe.close()
    f0, m0 = rounds[0]
    assert len(f0) >= 0.9 * pairs
    for f, m in rounds[1:]:
        assert np.array_equal(f0[:, :2], f[:, :2])
        assert np.array_equal(m0["pointCount"], m["pointCount"])
        for field in ("n", "p1", "p2", "triangleKey", "key", "edgeContact"):
            for i in range(4):
                has = m0["pointCount"] > i
                assert np.array_equal(m0["points"][field][has, i], m["points"][field][has, i]), field
