"""The sampler's points at the edges of its columns: films of a fraction of a column, of one column
and a cell, of one cell of depth, and of the deepest that eight columns per SM still take.  Points
are exactly hard-core (the grid test is exact integer arithmetic) and as dense as Bridson leaves
them (poisson.rs:14-132)."""
import numpy as np
import pytest

import fgrain_gb300 as fg

pytestmark = pytest.mark.gpu

CELL = 3 ** -0.5  # cells per r_min


# Film size in cells of r_min / sqrt(3) (columns are 8 x 8 cells over the full depth).
@pytest.mark.parametrize("cells", [(3.0, 2.5, 4.0), (8.0, 8.0, 5.2), (9.0, 8.5, 1.0), (17.3, 31.9, 2.4),
                                   (40.0, 25.1, 23.0), (33.0, 64.0, 30.5)])
@pytest.mark.parametrize("r_min", [0.9, 1.2])
def test_points_are_hard_core_and_dense(engine, cells, r_min):
    from scipy.spatial import cKDTree

    size = tuple(c * CELL * r_min for c in cells)
    cfg = fg.EmulsionConfig(size, r_min, 0.4, 0.2)
    em = fg.VirtualEmulsionLayer.synthesize(cfg, 5, engine)
    pos = em.crystals()["pos"]
    em.close()
    n = len(pos)
    assert n >= 1
    # Positions are rounded to float: half an ulp of the largest coordinate on either side.
    ulp = 2.0 ** -23 * max(size)
    assert (pos >= 0).all() and (pos <= np.array(size) + ulp).all()
    if n > 1:
        d, _ = cKDTree(pos).query(pos, k=2)
        assert d[:, 1].min() >= r_min * (1 - 1e-6) - ulp
    # Bridson's density in the bulk plus its surface term (the model the thinning targets); the
    # points left are at most the target plus what thinning's draws spare.
    vol = np.prod(size)
    target = (0.57793168 + 0.11306788 * r_min * sum(2 / s for s in size)) / r_min ** 3 * vol
    assert n <= target + 4 * np.sqrt(target) + 2
    if min(size) > 5 * r_min:
        assert abs(n - target) <= 0.02 * target + 4


@pytest.mark.parametrize("stock,grain", [("t-max", 1.1), ("tri-x", 2.4)])
def test_points_do_not_depend_on_the_columns_in_flight(engine, stock, grain):
    """A tile's crystals are the same alone (few columns: the kernel that draws ahead) and beside others
    (many columns)."""
    params = [fg.tile_params(stock, 1 / grain, 190 + i, 170, 1.0, 0.0, 40 + i) for i in range(8)]
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


# Depths of 1 .. 33 cells: bricks of 1 to 64 cells an edge, whose slots the compaction takes 512 at a time.
@pytest.mark.parametrize("cells", [(70.0, 45.3, 1.0), (41.0, 77.2, 1.9), (50.0, 33.3, 3.5), (9.0, 70.0, 7.6),
                                   (61.0, 40.0, 14.0), (35.5, 66.0, 19.0), (40.0, 30.0, 33.0)])
def test_crystals_come_in_slot_order(engine, cells):
    cfg = fg.EmulsionConfig(tuple(c * CELL for c in cells), 1.0, 0.4, 0.2)
    # The density model's count against the capacity of a film: the thinnest exceeds it and is refused.
    vol = np.prod([c * CELL for c in cells])
    target = (0.57793168 + 0.11306788 * sum(2 / (c * CELL) for c in cells)) * vol
    if target > 0.8 * vol + 64 + 4 * np.sqrt(0.01 * target):
        with pytest.raises(fg.GpuError, match="overflow"):
            fg.VirtualEmulsionLayer.synthesize(cfg, 9, engine)
        return
    em = fg.VirtualEmulsionLayer.synthesize(cfg, 9, engine)
    pos = em.crystals()["pos"].astype(np.float64)
    em.close()
    # Points are whole 1/1024ths of a cell, rounded to float.
    c = np.rint(pos * 1024 / CELL).astype(np.int64) >> 10
    grid = [int(np.ceil(x)) for x in cells]
    assert len(c) > 20 and (c < grid).all()
    depth_bits = max(grid[2] - 1, 0).bit_length()

    def spread(v, step):
        return sum(((v >> b) & 1) << (step * b) for b in range(12))

    lo, hi = c & ((1 << depth_bits) - 1), c >> depth_bits
    slot = ((spread(hi[:, 0], 2) | spread(hi[:, 1], 2) << 1) << (3 * depth_bits)
            | spread(lo[:, 0], 3) | spread(lo[:, 1], 3) << 1 | spread(lo[:, 2], 3) << 2)
    assert (np.diff(slot) > 0).all()
