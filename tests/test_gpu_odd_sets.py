"""Sets and settings at the limits of what the calls accept: emulsions for whose cells there is no memory
left, and crystals with negative half-sizes (whose geometry is that of their magnitudes:
crystal.rs:140-217 pairs or squares them)."""
import numpy as np
import pytest

import fgrain_gb300 as fg
from fgrain_gb300 import _abi
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

SIZE = (30.0, 28.0, 12.0)


def lattice(radius=0.5, morph=0):
    """A jittered lattice of about 4,300 crystals: positions, half-sizes, quaternions and the film's
    configuration."""
    rng = np.random.default_rng(3)
    k = [int(v / 1.3) for v in SIZE]
    g = np.stack(np.meshgrid(*[np.arange(q) for q in k], indexing="ij"), -1).reshape(-1, 3)
    pos = (g + 0.5 + rng.uniform(-0.12, 0.12, g.shape)) * (np.array(SIZE) / k)
    quat = rng.normal(size=(len(pos), 4))
    quat /= np.linalg.norm(quat, axis=1, keepdims=True)
    cfg = fg.EmulsionConfig(SIZE, 1.0, 0.5, 0.2, fg.Morphology(morph), 1.0, fg.GelatinOptics(), 1.0)
    return cfg, pos, np.full((len(pos), 3), radius), quat


def smallest_budget(make):
    """The least device budget (to 4 KB) under which make() gives an emulsion, and that emulsion: it has
    no cells, since what they need comes on top of everything else."""
    lib = _abi.load()
    lo, hi = 0, 1 << 28
    try:
        while hi - lo > 4096:
            mid = (lo + hi) // 2
            lib.fg_set_device_budget(mid)
            try:
                make().close()
                hi = mid
            except fg.GpuError as x:
                assert x.status == _abi.FG_ERR_OOM
                lo = mid
        lib.fg_set_device_budget(hi)
        return hi, make()
    finally:
        lib.fg_set_device_budget(0)


def counts(em):
    tile = np.random.default_rng(4).random((32, 32)).astype(np.float32)
    em.set_latent_counts(np.zeros(len(em), np.uint32))
    fg.expose_emulsion(em, tile, fg.ExposureConfig(20.0, 0.12, 1.3, 48), 7)
    return em.latent_counts()


# Bytes a crystal without cells: records (also in FP64, and as they came, when uploaded), state and the
# tree with its walk records; cells take about 110 more.
@pytest.mark.parametrize("kind,bytes_per_crystal", [("uploaded", 600), ("synthesized", 470)])
def test_an_emulsion_without_room_for_cells_keeps_the_walk(engine, kind, bytes_per_crystal):
    cfg, pos, dims, quat = lattice()

    def make():
        if kind == "uploaded":
            return fg.VirtualEmulsionLayer.from_crystals(cfg, pos, dims, quat, np.ones(len(pos)), engine=engine)
        return fg.VirtualEmulsionLayer.synthesize(fg.EmulsionConfig.preset("tri-x", 40.0, 40.0), 3, engine)

    budget, tight = smallest_budget(make)
    roomy = make()
    assert budget <= bytes_per_crystal * len(roomy) + (1 << 16)
    a, b = counts(tight), counts(roomy)
    assert b.sum() > 1000
    np.testing.assert_array_equal(a, b)
    dcfg = fg.DevelopmentConfig(4, 1.2, 1.25, 0.85)
    fg.develop_emulsion(tight, dcfg)
    fg.develop_emulsion(roomy, dcfg)
    for x, y in zip(tight.development(), roomy.development()):
        np.testing.assert_array_equal(x, y)
    tight.close()
    roomy.close()


@pytest.mark.parametrize("signs", [(-1, -1, -1), (-1, 1, 1)])
@pytest.mark.parametrize("morph", [0, 2])
@pytest.mark.parametrize("every", [1, 5])
def test_negative_half_sizes_keep_the_walk(engine, signs, morph, every):
    """A negative half-size has no part in the set's largest one, by which the cells search; counts and
    development are those of the walk, which the set takes for certain without room for cells."""
    cfg, pos, dims, quat = lattice(morph=morph)
    dims[::every] *= np.array(signs) * (1.0, 1.2, 0.9)

    def make():
        return fg.VirtualEmulsionLayer.from_crystals(cfg, pos, dims, quat, np.ones(len(pos)), engine=engine)

    _, walk = smallest_budget(make)
    em = make()
    a = counts(walk)
    assert a.sum() > 100
    np.testing.assert_array_equal(counts(em), a)
    for prox in (1.25, 0.7):
        dcfg = fg.DevelopmentConfig(2, 1.2, prox, 0.85)
        fg.develop_emulsion(walk, dcfg)
        fg.develop_emulsion(em, dcfg)
        for x, y in zip(em.development(), walk.development()):
            np.testing.assert_array_equal(x, y)
    walk.close()
    em.close()


@pytest.mark.parametrize("signs", [(-1, 1, 1), (1, -1, 1), (1, 1, -1)])
def test_cubes_with_a_negative_half_size_scan_as_in_the_oracle(engine, signs):
    cfg, pos, dims, quat = lattice()
    dims = dims * (1.0, 1.2, 0.8) * np.array(signs)
    n = len(pos)
    developed = (np.random.default_rng(1).random(n) < 0.3).astype(np.uint8)
    expansion = np.full(n, 1.2)
    em = fg.VirtualEmulsionLayer.from_crystals(cfg, pos, dims, quat, np.ones(n), engine=engine)
    em.set_development(developed, expansion)
    cr = orc.Crystals(pos, dims, quat, np.ones(n), np.zeros(n, np.int32))
    cr.developed[:], cr.expansion[:] = developed, expansion
    scfg = fg.ScanConfig(40, 36, 4, 0, 0.3)
    hits = np.asarray(fg.scan_ray_hits(em, scfg, 5)).ravel()
    em.close()
    ref = orc.scan(cr, cfg, scfg, 5, want_hits=True)["ray_hits"]
    assert ref.sum() > 10_000
    np.testing.assert_array_equal(hits, ref)


@pytest.mark.parametrize("prox,expansion", [(-0.3, 1.2), (0.3, -1.2), (-0.3, -1.2), (0.0, 1.2)])
def test_a_negative_touch_distance_develops_as_by_the_walk(engine, prox, expansion):
    """The reference's query box is then inside out and meets the leaves that hold it (bvh.rs:350-402)."""
    cfg, pos, dims, quat = lattice()
    pos[1::2] = pos[::2][:len(pos[1::2])] + [0.25, 0.1, -0.1]  # pairs that touch

    def make():
        return fg.VirtualEmulsionLayer.from_crystals(cfg, pos, dims, quat, np.ones(len(pos)), engine=engine)

    _, walk = smallest_budget(make)
    em = make()
    dcfg = fg.DevelopmentConfig(2, expansion, prox, 0.85)
    n = np.random.default_rng(5).integers(0, 5, len(pos)).astype(np.uint32)
    got = []
    for x in (em, walk):
        x.set_latent_counts(n)
        fg.develop_emulsion(x, dcfg)
        got.append(x.development())
        x.close()
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)
