"""GPU: b3TimeOfImpact in batches: a query's answer does not depend on the
others of its batch, and two translating spheres meet where their distance is
the target separation."""
import numpy as np
import pytest

from bounce_b200 import _native as N
from bounce_b200 import scene as S
from bounce_b200.pipeline import CollisionPipeline

pytestmark = pytest.mark.gpu

SLOP = 0.005
FAILED, OVERLAPPED, TOUCHING, SEPARATED = 1, 2, 3, 4


def hull_pipe():
    sc = S.Scene()
    rng = np.random.default_rng(4)
    for n in (4, 5, 8, 13, 32, 64):
        sc.hulls.add_points(S.ellipsoid_points(rng, n, np.array([0.5, 0.7, 0.9])))
    b = sc.add_body(0, N.BODY_DYNAMIC, (0, 0, 0), (0, 0, 0, 1))
    sc.add_fixture(b, N.SHAPE_HULL, [0.0], hull=0)
    return CollisionPipeline(sc.finalize())


# One query, the ends of a warp, of the queries that get a warp each (1,776)
# and of a full warp's share, and a batch whose warps refill their lanes.
@pytest.mark.parametrize("n", [1, 31, 33, 1775, 1777, 20011, 120001])
def test_batches(n):
    pipe = hull_pipe()
    rng = np.random.default_rng(n)
    q = S.toi_queries(rng, min(n, 3000), len(pipe.scene.hull_arrays["desc"]) // 6)
    q = q[rng.integers(0, len(q), n)] if n > len(q) else q
    out = pipe.time_of_impact(q)
    assert set(np.unique(out[:, 0])) <= {FAILED, OVERLAPPED, TOUCHING, SEPARATED}
    order = rng.permutation(n)
    assert np.array_equal(pipe.time_of_impact(q[order]), out[order])
    for i in range(0, n, max(1, n // 7)):
        assert np.array_equal(pipe.time_of_impact(q[i:i + 1]), out[i:i + 1])
    if n > 1000:
        assert {TOUCHING, SEPARATED} <= set(np.unique(out[:, 0]))
    pipe.close()


def test_spheres_meet_at_the_target():
    pipe = hull_pipe()
    rng = np.random.default_rng(3)
    n = 5000
    q = np.zeros(n, N.TOI_INPUT_DTYPE)
    r = rng.uniform(0.1, 0.8, (2, n)).astype(np.float32)
    c = rng.uniform(-3, 3, (2, 2, n, 3)).astype(np.float32)  # shape, start / end
    for k, side in enumerate("ab"):
        q["params_" + side][:, 3] = r[k]
        sw = q["sweep_" + side]
        sw[:, 6] = sw[:, 14] = 1.0
        sw[:, 7:10], sw[:, 15:18] = c[k, 0], c[k, 1]
    q["t_max"] = 1.0
    out = pipe.time_of_impact(q)
    t = out[:, 1].copy().view(np.float32).astype(np.float64)
    c = c.astype(np.float64)
    gap = lambda s: np.linalg.norm((1 - s)[:, None] * (c[1, 0] - c[0, 0]) + s[:, None] * (c[1, 1] - c[0, 1]), axis=1)
    target = np.maximum(SLOP, r[0].astype(np.float64) + r[1] - 3 * SLOP)
    # The tolerance of the root, plus the rounding of coordinates below 8 m.
    tol = 0.25 * SLOP + 8 * 2.0 ** -20
    touch = out[:, 0] == TOUCHING
    assert touch.sum() > 300
    assert np.all(np.abs(gap(t) - target)[touch & (t > 0)] <= tol)
    # Separated: the closest approach (a parabola's vertex) stays above it.
    d0, d1 = c[1, 0] - c[0, 0], c[1, 1] - c[0, 1]
    e = d1 - d0
    s = np.clip(-(d0 * e).sum(1) / (e * e).sum(1), 0, 1)
    apart = out[:, 0] == SEPARATED
    assert np.all(gap(s)[apart] >= (target - tol)[apart])
    pipe.close()
