"""The tree's global levels where test_gpu_tree_levels does not reach: the tree over the developed crystals
of an uneven set, a leaf of more crystals than a block builds, and builds on either side of the size from
which a warp takes eight words of positions and not two (64-bit keys: uploaded, 32-bit: synthesized).
Order, leaves and boxes are exactly those of BVH::build (bvh.rs:157-295)."""
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


@pytest.mark.parametrize("equal", [1025, 1500, 5000])
def test_a_leaf_of_many_equal_centroids(engine, equal):
    """More equal centroids than one block takes are a leaf of the global levels (bvh.rs:222-226)."""
    rng = np.random.default_rng(equal)
    box = np.array([60.0, 50.0, 12.0])
    pos = np.concatenate([np.tile(box * 0.01, (equal, 1)), box * (0.6, 0, 0) + rng.random((9000, 3)) * box * (0.4, 1, 1)])
    pos = pos[rng.permutation(len(pos))]
    n = len(pos)
    dims, quat, sens = attributes(rng, n)
    em = fg.VirtualEmulsionLayer.from_crystals(fg.EmulsionConfig((100.0, 60.0, 20.0), 1.0), pos, dims, quat, sens,
                                               engine=engine)
    cr = orc.Crystals(pos, dims, quat, sens, np.zeros(n, np.int32))
    check(em, cr)
    _, leaves, _ = fg.reference_tree(em)
    assert leaves[:, 1].max() == equal
    em.close()


@pytest.mark.parametrize("n", [519_999, 520_000, 640_000])
def test_uploaded_sets_about_the_longer_chunks(engine, n):
    rng = np.random.default_rng(n)
    pos = rng.random((n, 3)) * [300.0, 260.0, 12.0]
    dims, quat, sens = attributes(rng, n)
    em = fg.VirtualEmulsionLayer.from_crystals(fg.EmulsionConfig((300.0, 260.0, 12.0), 1.0), pos, dims, quat, sens,
                                               engine=engine)
    check(em, orc.Crystals(pos, dims, quat, sens, np.zeros(n, np.int32)))
    em.close()


@pytest.mark.parametrize("w,h", [(240.0, 310.0), (300.0, 340.0)])
def test_synthesized_sets_about_the_longer_chunks(engine, w, h):
    em = fg.VirtualEmulsionLayer.synthesize(fg.EmulsionConfig.preset("t-max", w, h), 9, engine)
    assert (len(em) > 520_000) == (w * h > 90_000.0)
    c = em.crystals()
    check(em, orc.Crystals(c["pos"], c["dims"], c["quat"], c["sensitivity"], c["morphology"]))
    em.close()
