"""Calls that are refused before any device work, with the status the header gives for them."""
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
    cfg = fg.ScanConfig(w, h, spp, 0, 0.3)
    with pytest.raises(fg.GpuError) as refused:
        if call == "signal":
            fg.scan_signal(emulsion, cfg, 1)
        else:
            fg.scan_backward(emulsion, cfg, 1, np.ones((h, w), np.float32))
    assert refused.value.status == _abi.FG_ERR_INVALID_ARG
    S, _ = fg.scan_signal(emulsion, fg.ScanConfig(6, 5, 4, 0, 0.3), 1)  # the engine goes on
    assert np.isfinite(S).all()
