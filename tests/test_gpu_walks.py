"""GPU: the pairs of a world that is wide on one axis only against all pairs
of its fat AABBs."""
import numpy as np
import pytest

from bounce_b200 import _native as N
from bounce_b200 import scene as S
from bounce_b200.pipeline import CollisionPipeline

pytestmark = pytest.mark.gpu


def stepped(scene, passes=3, **kw):
    pipe = CollisionPipeline(scene, **kw)
    drv = S.KinematicDriver(scene)
    for k in range(passes):
        if k:
            drv.advance()
        pipe.collide(drv.state17())
    return pipe


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
