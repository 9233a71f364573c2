"""Calls that are refused before any device work, with the status the header gives for them."""
import ctypes as C

import numpy as np
import pytest

import fgrain_gb300 as fg
from fgrain_gb300 import _abi

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def emulsion(engine):
    em = fg.VirtualEmulsionLayer.synthesize(fg.EmulsionConfig((8.0, 8.0, 6.0), 1.0, 0.4, 0.2), 3, engine)
    em.set_latent_counts(np.full(len(em), 9, np.uint32))
    fg.develop_emulsion(em, fg.DevelopmentConfig(4, 1.2, 1.25, 0.85))
    yield em
    em.close()


@pytest.mark.parametrize("w,h,spp", [(0, 5, 4), (5, 0, 4), (0, 0, 1), (6, 5, 300)])
@pytest.mark.parametrize("call", ["signal", "backward"])
def test_scan_sizes(emulsion, call, w, h, spp):
    e, cfg = emulsion.engine, fg.ScanConfig(w, h, spp, 0, 0.3).to_c()
    px = np.ones(max(w * h, 1), np.float32)
    out = np.zeros_like(px)
    sigma, ge, go = np.zeros(len(emulsion), np.float32), C.c_double(), C.c_double()

    def ptr(a):
        return a.ctypes.data_as(C.POINTER(C.c_float))

    if call == "signal":
        st = e._lib.fg_scan_signal(e._h, emulsion._h, C.byref(cfg), 1, None, 1.0, fg.OTF_SIGMA_REFERENCE, ptr(px), ptr(out))
    else:
        st = e._lib.fg_scan_backward(e._h, emulsion._h, C.byref(cfg), 1, None, 1.0, fg.OTF_SIGMA_REFERENCE, ptr(px),
                                     ptr(sigma), C.byref(ge), C.byref(go))
    assert st == _abi.FG_ERR_INVALID_ARG
    said = e._lib.fg_last_error(e._h).decode()
    assert ("scan size must be positive" if w * h == 0 else "samples_per_pixel too large") in said, said
    S, _ = fg.scan_signal(emulsion, fg.ScanConfig(6, 5, 4, 0, 0.3), 1)  # the engine goes on
    assert np.isfinite(S).all()
