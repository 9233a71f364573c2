"""Films so deep, or crystals so large, that a segment absorbs many hits: transport by the tree walk, in
batches and emulsions, against the oracle's exposure of the same crystals (transport.rs:48-188), beside
tiles of ordinary depth, and where the crystals lie unevenly.

Tolerance: FP32 decides few hits and draws differently from the oracle: 99 % of the crystals have its count
exactly, as the batch's pipeline test asks, and the photons in all agree to 1e-3."""
import numpy as np
import pytest

import fgrain_gb300 as fg
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def tile(stock, w, h, seed, depth=None, aspect=None, scatter=None):
    p = fg.tile_params(stock, 1 / 2.4, w, h, 1.0, 0.0, seed)
    if depth:
        p.film_d = depth
    if aspect:
        p.tabular_aspect_ratio = aspect
    if scatter is not None:
        p.optics.scattering_coeff = scatter
    return p


def exposures(params):
    rng = np.random.default_rng(3)
    return [rng.uniform(0.2, 1.0, (p.height_px, p.width_px)).astype(np.float32) for p in params]


def run(engine, params, use_graph=False):
    b = fg.Batch(params, engine, use_graph=use_graph)
    b.set_exposure(exposures(params))
    for _ in range(2):
        b.run()
        b.wait()
    out = [b.tile_crystals(i) for i in range(len(params))], b.density()
    b.close()
    return out


# Scattering 0 and 45 um: about 30 hits a segment, in tiles of 54 x 50 um (a narrower one's photons leave by its
# sides).  Aspect 0.1: crystals ten times as long as wide.
CASES = [("tri-x", 45.0, None, 0.0), ("tri-x", 60.0, None, 0.02), ("t-max", None, 0.1, None)]


@pytest.mark.parametrize("stock,depth,aspect,scatter", CASES)
def test_batch_counts_match_the_oracle(engine, stock, depth, aspect, scatter):
    p = tile(stock, 130, 120, 5, depth, aspect, scatter)
    crystals, density = run(engine, [p])
    c = crystals[0]
    cr = orc.Crystals(c["pos"], c["dims"], c["quat"], c["sensitivity"], c["morphology"])
    cfg = fg.EmulsionConfig((p.film_w, p.film_h, p.film_d), p.r_min, p.mean_crystal_radius, p.size_variance,
                            fg.Morphology(p.morphology), p.tabular_aspect_ratio,
                            fg.GelatinOptics(p.optics.refractive_index, p.optics.absorption_coeff,
                                             p.optics.scattering_coeff, p.optics.anisotropy_g,
                                             p.optics.antihalation_reflectance, p.optics.antihalation_density),
                            p.base_sensitivity)
    ecfg = fg.ExposureConfig(p.photons_per_sq_um, p.illumination_angle_rad, p.crystal_absorption_coeff, p.max_bounces)
    orc.expose(cr, cfg, exposures([p])[0], ecfg, 6)
    got, ref = c["counts"].astype(np.int64), cr.latent.astype(np.int64)
    assert ref.sum() > 1000
    assert (got == ref).mean() > 0.99
    assert abs(got.sum() - ref.sum()) <= 1e-3 * ref.sum()


@pytest.mark.parametrize("stock,depth,aspect,scatter", CASES)
def test_a_deep_tile_changes_no_other(engine, stock, depth, aspect, scatter):
    """One deep tile takes its whole batch to the walk; an ordinary tile's crystals, counts and density are those
    it has alone, through the cells; plain launches and the captured graph agree."""
    small, deep = tile("tri-x", 64, 48, 9), tile(stock, 130, 120, 5, depth, aspect, scatter)
    (c0,), (d0,) = run(engine, [small])
    for graph in (False, True):
        crystals, density = run(engine, [small, deep], graph)
        for k in c0:
            np.testing.assert_array_equal(crystals[0][k], c0[k])
        np.testing.assert_array_equal(density[0], d0)


def test_emulsions_of_many_hits_expose_as_batches(engine):
    """An uploaded set of the crystals of a deep tile gets the tile's counts."""
    p = tile("tri-x", 130, 120, 5, 45.0, None, 0.0)
    c = run(engine, [p])[0][0]
    cfg = fg.EmulsionConfig((p.film_w, p.film_h, p.film_d), p.r_min, p.mean_crystal_radius, p.size_variance,
                            fg.Morphology(p.morphology), p.tabular_aspect_ratio,
                            fg.GelatinOptics(p.optics.refractive_index, p.optics.absorption_coeff,
                                             p.optics.scattering_coeff, p.optics.anisotropy_g,
                                             p.optics.antihalation_reflectance, p.optics.antihalation_density),
                            p.base_sensitivity)
    em = fg.VirtualEmulsionLayer.from_crystals(cfg, c["pos"], c["dims"], c["quat"], c["sensitivity"], c["morphology"],
                                               engine)
    ecfg = fg.ExposureConfig(p.photons_per_sq_um, p.illumination_angle_rad, p.crystal_absorption_coeff, p.max_bounces)
    fg.expose_emulsion(em, exposures([p])[0], ecfg, 6)
    np.testing.assert_array_equal(em.latent_counts(), c["counts"])
    em.close()


@pytest.mark.parametrize("share,area", [(0.0, 1.0), (0.5, 0.2), (0.5, 0.1), (0.8, 0.15)])
def test_uneven_sets_match_the_oracle(engine, share, area):
    """A share of the crystals in a corner of the film: cells while the corner is not too dense, then the walk."""
    rng = np.random.default_rng(3)
    size, n = np.array([30.0, 28.0, 12.0]), 5000
    pos = rng.random((n, 3)) * size
    pos[:int(n * share), :2] *= np.sqrt(area)
    quat = rng.normal(size=(n, 4))
    quat /= np.linalg.norm(quat, axis=1, keepdims=True)
    dims = np.full((n, 3), 0.4)
    cfg = fg.EmulsionConfig(tuple(size), 1.0, 0.5, 0.2, fg.Morphology(0), 1.0, fg.GelatinOptics(), 1.0)
    tile = rng.uniform(0.2, 1.0, (24, 26)).astype(np.float32)
    ecfg = fg.ExposureConfig(20.0, 0.12, 1.3, 48)
    cr = orc.Crystals(pos, dims, quat, np.ones(n), np.zeros(n, np.int32))
    orc.expose(cr, cfg, tile, ecfg, 7)
    em = fg.VirtualEmulsionLayer.from_crystals(cfg, pos, dims, quat, np.ones(n), engine=engine)
    fg.expose_emulsion(em, tile, ecfg, 7)
    got, ref = em.latent_counts().astype(np.int64), cr.latent.astype(np.int64)
    em.close()
    assert ref.sum() > 1000 and (got == ref).mean() > 0.99
    assert abs(got.sum() - ref.sum()) <= 1e-3 * ref.sum()
