"""The scan's rays in every bin layout (bins of 1 to 16 pixels, Morton-ordered and row-ordered), at
image sizes that cut bins off, on pixels smaller and larger than the crystals: per-ray hit counts
exactly and transmittance to 1e-5 of the FP64 oracle (transmittance.rs:65-171), and the adjoint's
per-crystal gradients to 1e-4 of the oracle's."""
import numpy as np
import pytest

import fgrain_gb300 as fg
from oracle import oracle as orc
from tests.helpers import reference_cfg

pytestmark = pytest.mark.gpu


def developed_set(stock, w, h, seed):
    cfg = reference_cfg(stock, w, h)
    cr = orc.synthesize(cfg, seed)
    rng = np.random.default_rng(seed)
    cr.developed[:] = rng.random(len(cr)) < 0.6
    cr.expansion[:] = np.where(cr.developed, 1.2 * rng.choice([1.0, 1.33, 1.8], len(cr)), 0.0)
    return cfg, cr


@pytest.mark.parametrize("stock", ["tri-x", "t-max"])
@pytest.mark.parametrize("size", [(37, 29), (5, 61)])
@pytest.mark.parametrize("spp", [1, 4, 9, 25, 64, 256])
def test_ray_hits_and_transmittance(engine, stock, size, spp):
    w, h = size
    cfg, cr = developed_set(stock, 16.0, 13.0, 3 + spp)
    em = fg.VirtualEmulsionLayer.from_crystals(cfg, cr.pos, cr.dims, cr.quat, cr.sens, cr.morph, engine)
    em.set_development(cr.developed, cr.expansion)
    sc = fg.ScanConfig(w, h, spp, fg.ScanMode.NegativeTransmittance, 0.25)
    buf, _ = fg.scan_emulsion(em, sc, 19)
    ref = orc.scan(cr, cfg, sc, 19, want_hits=True)
    assert (np.abs(buf - ref["T64"]) / ref["T64"]).max() <= 1e-5
    np.testing.assert_array_equal(fg.scan_ray_hits(em, sc, 19), ref["ray_hits"])
    em.close()


@pytest.mark.parametrize("spp,size", [(1, (33, 20)), (4, (19, 45)), (9, (21, 17))])
def test_adjoint(engine, spp, size):
    w, h = size
    cfg, cr = developed_set("hp5", 14.0, 12.0, 40 + spp)
    em = fg.VirtualEmulsionLayer.from_crystals(cfg, cr.pos, cr.dims, cr.quat, cr.sens, cr.morph, engine)
    em.set_development(cr.developed, cr.expansion)
    sc = fg.ScanConfig(w, h, spp, fg.ScanMode.NegativeTransmittance, 0.25)
    rng = np.random.default_rng(spp)
    sig = rng.uniform(0.2, 0.3, len(cr)).astype(np.float32)
    G = rng.normal(size=(h, w)).astype(np.float32)
    gs, ge, go = fg.scan_backward(em, sc, 7, G, sig, 0.9, 0.45)
    rs, re, ro = orc.scan_backward(cr, cfg, sc, 7, G.astype(np.float64), sig.astype(np.float64), 0.9, 0.45)
    assert np.abs(gs - rs).max() <= 1e-4 * np.abs(rs).max()
    assert (gs[cr.developed == 0] == 0).all()
    scale = np.abs(G).sum()  # of the two reductions' terms
    assert abs(ge - re) <= 1e-6 * scale and abs(go - ro) <= 1e-6 * scale
    # Without the per-crystal part the other two gradients are the same.
    lib, e = engine._lib, engine
    import ctypes as C
    a, b = C.c_double(), C.c_double()
    cfgc = sc.to_c()
    f = lambda x: x.ctypes.data_as(C.POINTER(C.c_float))
    assert lib.fg_scan_backward(e._h, em._h, C.byref(cfgc), 7, f(sig), 0.9, 0.45, f(G), None, C.byref(a), C.byref(b)) == 0
    assert (a.value, b.value) == (ge, go)
    em.close()
