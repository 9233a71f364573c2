"""The sampler's columns where their shared memory sets how many run at once: at the deepest films that
eight columns of an SM take, one cell deeper, and at the deepest accepted (100 cells); and the points of a
tile by the kernel for few columns and by the one for many."""
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


@pytest.mark.parametrize("stock,grain,tiles", [("t-max", 1.1, 8), ("tri-x", 2.4, 32), ("hp5", 2.0, 24)])
def test_points_are_the_same_by_either_kernel(engine, stock, grain, tiles):
    """A tile alone has few columns (at most 20 an SM: the kernel that draws ahead), beside the others many."""
    import torch

    params = [fg.tile_params(stock, 1 / grain, 190 + i, 170, 1.0, 0.0, 40 + i) for i in range(tiles)]

    def columns(ps):
        return sum(int(np.ceil(np.ceil(p.film_w / (p.r_min * CELL)) / 8)) * int(np.ceil(np.ceil(p.film_h / (p.r_min * CELL)) / 8))
                   for p in ps)

    line = 20 * torch.cuda.get_device_properties(0).multi_processor_count
    assert columns(params[:1]) <= line < columns(params)
    both = []
    for ps in (params[:1], params):
        b = fg.Batch(ps, engine, use_graph=False)
        b.set_exposure([np.full((p.height_px, p.width_px), 0.5, np.float32) for p in ps])
        b.run()
        b.wait()
        both.append(b.tile_crystals(0))
        b.close()
    for k in both[0]:
        np.testing.assert_array_equal(both[0][k], both[1][k])
