"""Transport's launch shape as a batch's options set it: the counts do not depend on it, and few blocks are
as busy with few photons as with many."""
import numpy as np
import pytest

import fgrain_gb300 as fg

pytestmark = pytest.mark.gpu


def run(engine, tiles, blocks, threads=0):
    ps = [fg.tile_params("tri-x", 1 / 2.4, 64, 64, 1.0, 0.0, 5 + i) for i in range(tiles)]
    b = fg.Batch(ps, engine, use_graph=False, transport_blocks=blocks, transport_threads=threads)
    b.set_exposure([np.full((64, 64), 0.5, np.float32)] * tiles)
    ms = []
    for _ in range(4):
        b.run()
        w = b.wait()
        ms.append(w["transport_ms"])
    counts = b.tile_crystals(0)["counts"]
    b.close()
    return min(ms) / w["photons"], counts


@pytest.mark.parametrize("blocks,threads", [(1, 0), (4, 64), (32, 128)])
def test_few_blocks(engine, blocks, threads):
    """Each block works through its photons with its warps full: one tile's photons (4,267) cost a few blocks at
    most three times as much each as those of sixteen tiles (the last photons leave lanes idle)."""
    per_photon, counts = run(engine, 1, blocks, threads)
    per_photon16, counts16 = run(engine, 16, blocks, threads)
    _, default = run(engine, 1, 0)
    np.testing.assert_array_equal(counts, default)
    np.testing.assert_array_equal(counts16, default)
    if blocks <= 4:
        assert per_photon <= 3.0 * per_photon16, (per_photon, per_photon16)
