"""The fast mode's scan at the edges of its pixel lists, bit for bit with the oracle: pixels narrower
and wider than the columns their rays look at, one ray to many a pixel, lists tested in several
parts, and shapes whose hits depend on rounding (thin plates far below the ray's start,
crystals with no extent)."""
import numpy as np
import pytest

from fgrain_gb300 import fast
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


# preset, pixel (um), width, height, then fields of the tile: rays a pixel, depth, expansion, aspect
@pytest.mark.parametrize("preset,px,w,h,fields", [
    ("tri-x", 0.05, 70, 33, {}),
    ("hp5", 1.1, 37, 45, dict(samples_per_pixel=1)),
    ("tri-x", 2.9, 40, 31, dict(samples_per_pixel=9)),
    ("t-max", 6.5, 33, 20, dict(samples_per_pixel=25)),
    ("hp5", 40.0, 24, 17, {}),
    ("tri-x", 0.8, 50, 40, dict(filament_expansion=6.0)),
    ("t-max", 0.6, 60, 50, dict(film_d=250.0, tabular_aspect_ratio=150.0)),
    ("tri-x", 0.6, 48, 40, dict(filament_expansion=0.0)),
    ("hp5", 0.7, 41, 43, dict(film_d=90.0, samples_per_pixel=2)),
    # Enough pixels for a thread each (the others: a lane for each ray).
    ("t-max", 0.2, 230, 301, {}),
    ("hp5", 0.15, 301, 203, dict(samples_per_pixel=9, filament_expansion=4.0)),
    ("tri-x", 0.3, 257, 243, dict(samples_per_pixel=1, film_d=40.0)),
])
def test_scan_bit_exact_with_oracle(engine, preset, px, w, h, fields):
    p = fast.tile_params_fast(preset, px, w, h, 6.0, 0.5, 21)
    for k, v in fields.items():
        setattr(p, k, v)
    tile = np.random.default_rng(4).random((h, w)).astype(np.float32)
    d, cells = fast.render_tile_fast(tile, p, engine, cells=True)
    do, co = orc.fast_tile(p, tile)
    for f in ("pos", "dims_exp", "rot", "flags"):
        np.testing.assert_array_equal(cells[f], co[f], err_msg=f)
    np.testing.assert_array_equal(d, do)
    np.testing.assert_array_equal(fast.render_tile_fast(tile, p, engine), do)
