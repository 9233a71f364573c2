"""The sampler's columns where their shared memory sets how many run at once: at the deepest films that
eight columns of an SM take, one cell deeper, and at the deepest accepted (100 cells)."""
import numpy as np
import pytest

import fgrain_gb300 as fg

pytestmark = pytest.mark.gpu

CELL = 3 ** -0.5  # cells per r_min


@pytest.mark.parametrize("depth", [23.5, 24.0, 25.0, 99.5])
def test_points_are_hard_core_and_dense(engine, depth):
    from scipy.spatial import cKDTree

    size = (60.0 * CELL, 52.3 * CELL, depth * CELL)
    em = fg.VirtualEmulsionLayer.synthesize(fg.EmulsionConfig(size, 1.0, 0.4, 0.2), 5, engine)
    pos = em.crystals()["pos"]
    em.close()
    ulp = 2.0 ** -23 * max(size)  # positions are rounded to float: half an ulp on either side
    d, _ = cKDTree(pos).query(pos, k=2)
    assert d[:, 1].min() >= 1.0 - 1e-6 - ulp
    vol = np.prod(size)
    target = (0.57793168 + 0.11306788 * sum(2 / s for s in size)) * vol
    assert abs(len(pos) - target) <= 0.02 * target + 4
