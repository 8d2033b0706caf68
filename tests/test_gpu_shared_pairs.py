"""GPU: hull pairs whose edge query 1, 2 or 4 warps share give the same contacts.

148 blocks an SM's worth of 1 with 2 warps are 296 warps: 148 pairs and fewer are
shared by 2 of them; 8 blocks of 4 warps share up to 1,184 pairs by 4."""
import numpy as np
import pytest

from bounce_b200 import scene as S
from bounce_b200 import _native as N
from bounce_b200.pipeline import CollisionPipeline

pytestmark = pytest.mark.gpu

# (warps a block, blocks an SM)
SHAPES = [(4, 8), (2, 1), (2, 2), (4, 1), (8, 1), (8, 2)]


@pytest.mark.parametrize("pairs", [1, 36, 74, 75, 148, 149, 297, 1184])
def test_shared_pairs(pairs):
    rng = np.random.default_rng(pairs)
    sc = S.Scene()
    hulls = [sc.hulls.add_points(S.ellipsoid_points(rng, m, rng.uniform(0.5, 0.9, 3))) for m in (6, 12, 20, 40, 64)]
    q = S.random_quats(rng, 2 * pairs)
    for k in range(pairs):
        x = np.array([6.0 * (k % 40), 0.0, 6.0 * (k // 40)])
        for j in range(2):
            b = sc.add_body(0, N.BODY_DYNAMIC, x + j * rng.uniform(-0.7, 0.7, 3), q[2 * k + j])
            sc.add_fixture(b, N.SHAPE_HULL, [0.01], hull=hulls[rng.integers(5)])
    sc.finalize()
    state = S.KinematicDriver(sc).state17()
    first = None
    for warps, blocks in SHAPES:
        pipe = CollisionPipeline(sc, max_contacts=8192)
        table = pipe.tuning()
        table[10], table[11] = warps, blocks
        pipe.set_tuning(table)
        pipe.collide(state)
        got = (pipe.contacts(), pipe.manifolds().tobytes(), pipe.caches())
        pipe.close()
        assert len(got[0]) == pairs
        if first is None:
            first = got
        assert np.array_equal(got[0], first[0]) and got[1] == first[1] and np.array_equal(got[2], first[2])
