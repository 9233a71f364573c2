"""Production transport on uploaded crystal sets chosen for the edges of its cells: segments of more
hits than one visit keeps, sets of one crystal, crystals whose reach or place sends the set to the
tree walk.  Counts against the oracle's exposure with the reference's hit rule (transport.rs:48-188).

Tolerance: the device traces in FP32, so a hit may flip when a photon passes within about 1e-6
relative of a crystal's surface and a latent photon when a draw lies as close to a fraction; both
are rarer than 1e-3 of a crystal's hits, so counts agree within 2 + 1e-3 of the count (a flip also
moves the energy of the packet's later hits, within the same share).
"""
import numpy as np
import pytest

import fgrain_gb300 as fg
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def lattice(w, h, d, step, radius, rng, jitter=0.1):
    n = [max(int(v / step), 1) for v in (w, h, d)]
    g = np.stack(np.meshgrid(*[np.arange(k) for k in n], indexing="ij"), -1).reshape(-1, 3)
    pos = (g + 0.5 + rng.uniform(-jitter, jitter, g.shape)) * (np.array([w, h, d]) / n)
    q = rng.normal(size=(len(pos), 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    return pos, np.full((len(pos), 3), radius), q


def case(name):
    """(film w, h, d; positions, half-sizes, quaternions; morphology; scattering per um)."""
    rng = np.random.default_rng(11)
    if name == "many hits":  # about 25 crystals along every ray: several visits per segment
        return (12.0, 12.0, 40.0), *lattice(12.0, 12.0, 40.0, 1.1, 0.95, rng), 2, 0.005
    if name == "cubes with many hits":
        return (10.0, 10.0, 30.0), *lattice(10.0, 10.0, 30.0, 1.2, 0.62, rng), 0, 0.005
    if name == "one crystal":
        return (6.0, 5.0, 8.0), np.array([[3.0, 2.5, 4.0]]), np.full((1, 3), 0.8), np.array([[0.1, 0.2, 0.3, 0.9]]), 0, 0.03
    if name == "one long row":  # one row of cells, many crystals along x
        return (60.0, 1.5, 1.5), *lattice(60.0, 1.5, 1.5, 1.3, 0.5, rng), 2, 0.05
    pos, dims, q = lattice(15.0, 14.0, 9.0, 1.3, 0.45, rng)
    if name == "one giant":  # reach far above the spacing
        dims[len(dims) // 2] = 4.0
    elif name == "outside the box":
        pos[::7] += np.array([0.0, 15.0, -3.0])
    elif name == "bunched":  # every crystal in a corner of its film
        pos *= 0.25
    else:
        assert name == "even"
    return (15.0, 14.0, 9.0), pos, dims, q, 1 if name == "bunched" else 0, 0.05


@pytest.mark.parametrize("name", ["even", "many hits", "cubes with many hits", "one crystal", "one long row",
                                  "one giant", "outside the box", "bunched"])
def test_counts_match_the_oracle(engine, name):
    (w, h, d), pos, dims, quat, morph, scatter = case(name)
    quat = quat / np.linalg.norm(quat, axis=1, keepdims=True)
    n = len(pos)
    sens = np.random.default_rng(12).uniform(0.6, 1.4, n)
    cfg = fg.EmulsionConfig((w, h, d), 1.0, 0.5, 0.2, fg.Morphology(morph), 1.0,
                            fg.GelatinOptics(scattering_coeff=scatter), 1.0)
    tile = np.random.default_rng(13).uniform(0.2, 1.0, (9, 11)).astype(np.float32)
    ecfg = fg.ExposureConfig(20.0, 0.12, 1.3, 48)
    cr = orc.Crystals(pos, dims, quat, sens, np.full(n, morph))
    _, _, hits = orc.expose(cr, cfg, tile, ecfg, 77)
    em = fg.VirtualEmulsionLayer.from_crystals(cfg, pos, dims, quat, sens, engine=engine)
    fg.expose_emulsion(em, tile, ecfg, 77)
    got = em.latent_counts().astype(np.int64)
    ref = cr.latent.astype(np.int64)
    assert ref.sum() > 0
    np.testing.assert_array_less(np.abs(got - ref), 2.0 + 1e-3 * ref + 1e-9)
    assert abs(engine.timings()["hits"] - hits) <= 2 + 1e-3 * hits
    em.close()


@pytest.mark.parametrize("name", ["even", "many hits", "one crystal", "one long row", "one giant", "outside the box"])
def test_clumps_match_the_oracle(engine, name):
    """Development (development.rs:59-188) over the cells, or over the tree where the set has none:
    mask, clump ids and expansions exactly."""
    (w, h, d), pos, dims, quat, morph, _ = case(name)
    quat = quat / np.linalg.norm(quat, axis=1, keepdims=True)
    n = len(pos)
    cfg = fg.EmulsionConfig((w, h, d), 1.0, 0.5, 0.2, fg.Morphology(morph))
    counts = np.random.default_rng(14).integers(0, 8, n).astype(np.uint32)
    em = fg.VirtualEmulsionLayer.from_crystals(cfg, pos, dims, quat, np.ones(n), engine=engine)
    em.set_latent_counts(counts)
    dcfg = fg.DevelopmentConfig(4, 1.2, 1.25, 0.85)
    rep = fg.develop_emulsion(em, dcfg)
    cr = orc.Crystals(pos, dims, quat, np.ones(n), np.full(n, morph))
    cr.latent[:] = counts
    ref = orc.develop(cr, dcfg)
    dv, cl, ex = em.development()
    np.testing.assert_array_equal(dv, cr.developed)
    np.testing.assert_array_equal(cl, cr.clump)
    np.testing.assert_array_equal(ex, np.where(cr.developed, cr.expansion, 0.0))
    assert rep.total_clumps == ref["total_clumps"]
    em.close()


@pytest.mark.parametrize("stock,grain,side", [("t-max", 1.1, 120), ("tri-x", 2.4, 150)])
def test_counts_do_not_depend_on_the_photons_in_flight(engine, stock, grain, side):
    """A tile's latent photons are the same alone (a few photons a lane) and beside others (many)."""
    params = [fg.tile_params(stock, 1 / grain, side, side + i, 1.0, 0.0, 70 + i) for i in range(16)]
    rng = np.random.default_rng(6)
    tiles = [rng.random((p.height_px, p.width_px)).astype(np.float32) for p in params]
    both, photons = [], []
    for k in (1, 16):
        b = fg.Batch(params[:k], engine, use_graph=False)
        b.set_exposure(tiles[:k])
        b.run()
        photons.append(b.wait()["photons"])
        both.append(b.tile_crystals(0)["counts"])
        b.close()
    assert photons[1] > 10 * photons[0]
    np.testing.assert_array_equal(both[0], both[1])
    assert both[0].sum() > 1000
