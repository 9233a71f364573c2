"""The reference tree's global levels (sets above the 1,024 elements one block finishes) at the edges
of their chunks and words, on even, uneven and degenerate sets, with 64-bit keys (uploaded sets) and
32-bit keys (synthesized sets, whose crystals the oracle then rebuilds): element order, leaves and
FP64 leaf boxes exactly as BVH::build (bvh.rs:157-295).  A set so uneven that its halving leaves more
than 1,024 crystals in a node after the levels allowed (log2(n / 1024) rounded up, plus 8) is refused."""
import numpy as np
import pytest

import fgrain_gb300 as fg
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def check(em, cr):
    order, leaves, boxes = fg.reference_tree(em)
    ro, rl, rb = orc.bvh_export(cr)
    np.testing.assert_array_equal(order, ro)
    k = np.argsort(rl[:, 0], kind="stable")
    np.testing.assert_array_equal(leaves, rl[k])
    np.testing.assert_array_equal(boxes, rb[k])


def levels_needed(pos):
    """Spatial-median levels with a node of more than 1,024 points (a node of equal points takes one
    too, which finds that it does not split)."""
    nodes, level = [pos], 0
    while nodes:
        level += 1
        nxt = []
        for p in nodes:
            lo, hi = p.min(0), p.max(0)
            e = hi - lo
            axis = 0 if e[0] >= e[1] and e[0] >= e[2] else (1 if e[1] >= e[2] else 2)
            if e[axis] <= 1e-7:
                continue
            big = p[:, axis] >= 0.5 * (lo[axis] + hi[axis])
            nxt += [p[~big], p[big]]
        nodes = [p for p in nxt if len(p) > 1024]
    return level


@pytest.mark.parametrize("kind", ["even", "clustered", "one axis", "many equal"])
@pytest.mark.parametrize("n", [1025, 1056, 2047, 2048, 2049, 4097, 16384, 30011])
def test_uploaded_sets(engine, kind, n):
    rng = np.random.default_rng(n)
    if kind == "even":
        pos = rng.random((n, 3)) * [60.0, 50.0, 12.0]
    elif kind == "clustered":
        pos = np.exp(rng.normal(size=(n, 3)) * 0.8)
    elif kind == "one axis":
        pos = np.stack([rng.random(n) * 100.0, np.full(n, 2.0), np.full(n, 3.0)], 1)
    else:
        pos = rng.random((n, 3)) * 20.0
        pos[rng.random(n) < 0.4] = [4.0, 5.0, 6.0]  # more than a block's worth in one leaf, for larger n
    dims = rng.uniform(0.1, 0.6, (n, 3))
    quat = rng.normal(size=(n, 4))
    quat /= np.linalg.norm(quat, axis=1, keepdims=True)
    sens = np.ones(n)
    cfg = fg.EmulsionConfig((100.0, 60.0, 20.0), 1.0)
    allowed = int(np.ceil(np.log2(n / 1024))) + 8
    if levels_needed(pos) > allowed:
        with pytest.raises(fg.GpuError) as refused:
            fg.VirtualEmulsionLayer.from_crystals(cfg, pos, dims, quat, sens, engine=engine)
        assert refused.value.status == 19  # FG_ERR_DEVICE_OVERFLOW
        return
    em = fg.VirtualEmulsionLayer.from_crystals(cfg, pos, dims, quat, sens, engine=engine)
    check(em, orc.Crystals(pos, dims, quat, sens, np.zeros(n, np.int32)))
    em.close()


@pytest.mark.parametrize("stock,w,h", [("tri-x", 24.0, 20.0), ("t-max", 33.0, 41.0), ("hp5", 150.0, 90.0),
                                       ("t-max", 240.0, 300.0)])
def test_synthesized_sets(engine, stock, w, h):
    em = fg.VirtualEmulsionLayer.synthesize(fg.EmulsionConfig.preset(stock, w, h), 9, engine)
    c = em.crystals()
    check(em, orc.Crystals(c["pos"], c["dims"], c["quat"], c["sensitivity"], c["morphology"]))
    em.close()


# One block's subtree with 64-bit keys: nodes that start, end and straddle the words of 32 positions.
@pytest.mark.parametrize("kind", ["even", "clustered", "one axis", "pairs"])
@pytest.mark.parametrize("n", [1, 4, 5, 31, 32, 33, 64, 65, 200, 1023, 1024])
def test_uploaded_sets_of_one_block(engine, kind, n):
    rng = np.random.default_rng(100 + n)
    if kind == "even":
        pos = rng.random((n, 3)) * [60.0, 50.0, 12.0]
    elif kind == "clustered":
        pos = np.exp(rng.normal(size=(n, 3)))
    elif kind == "one axis":
        pos = np.stack([np.full(n, 1.0), rng.random(n) * 50.0, np.full(n, 3.0)], 1)
    else:
        pos = np.repeat(rng.random((n // 2 + 1, 3)) * 30.0, 2, axis=0)[:n]
    dims = rng.uniform(0.1, 0.6, (n, 3))
    quat = rng.normal(size=(n, 4))
    quat /= np.linalg.norm(quat, axis=1, keepdims=True)
    sens = np.ones(n)
    em = fg.VirtualEmulsionLayer.from_crystals(fg.EmulsionConfig((100.0, 60.0, 20.0), 1.0), pos, dims, quat, sens,
                                               engine=engine)
    check(em, orc.Crystals(pos, dims, quat, sens, np.zeros(n, np.int32)))
    em.close()
