"""The tree's global levels where test_gpu_tree_levels does not reach: the tree over the developed crystals
of an uneven set."""
import numpy as np
import pytest

import fgrain_gb300 as fg
from oracle import oracle as orc
from tests.test_gpu_tree_levels import levels_needed

pytestmark = pytest.mark.gpu


def check(em, cr, developed_only=False):
    order, leaves, boxes = fg.reference_tree(em, developed_only)
    ro, rl, rb = orc.bvh_export(cr, developed_only)
    np.testing.assert_array_equal(order, ro)
    k = np.argsort(rl[:, 0], kind="stable")
    np.testing.assert_array_equal(leaves, rl[k])
    np.testing.assert_array_equal(boxes, rb[k])


def attributes(rng, n):
    quat = rng.normal(size=(n, 4))
    quat /= np.linalg.norm(quat, axis=1, keepdims=True)
    return rng.uniform(0.1, 0.6, (n, 3)), quat, np.ones(n)


def test_developed_crystals_more_uneven_than_their_set(engine):
    """A bunch of 1,500 developed crystals and one at every halving of the way to it, and 28,000 others far
    off: both trees need the halvings, but the developed ones' holds a twentieth of the crystals."""
    rng = np.random.default_rng(2)
    box = np.array([60.0, 50.0, 12.0])
    ladder = box * 2.0 ** -np.arange(11)[:, None]
    bunch = rng.random((1500, 3)) * box * 2.0 ** -12
    pos = np.concatenate([ladder, bunch, box * (0.6, 0, 0) + rng.random((28000, 3)) * box * (0.4, 1, 1)])
    n, dev = len(pos), np.arange(len(pos)) < 1511

    def allowed(k):
        return int(np.ceil(np.log2(k / 1024))) + 8

    assert levels_needed(pos) <= allowed(n) and levels_needed(pos[dev]) > allowed(dev.sum())
    dims, quat, sens = attributes(rng, n)
    em = fg.VirtualEmulsionLayer.from_crystals(fg.EmulsionConfig((100.0, 60.0, 20.0), 1.0), pos, dims, quat, sens,
                                               engine=engine)
    cr = orc.Crystals(pos, dims, quat, sens, np.zeros(n, np.int32))
    cr.developed[:], cr.expansion[:] = dev, np.where(dev, 1.2, 0.0)
    em.set_development(cr.developed, cr.expansion)
    check(em, cr, developed_only=True)
    em.close()
