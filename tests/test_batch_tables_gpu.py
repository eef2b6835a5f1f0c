"""The batch's source where a tile's lattice positions are no numbers: such octaves are not looked
up in a table and the tile's heights are NaN; the tiles beside it are as they are alone."""

import numpy as np
import pytest

from terraingen_b200.batch import TILE, Batch, TileSet
from terraingen_b200.layouts import CRATER_RECORD, CRATER_SHAPE_KERNEL, fractal

pytestmark = pytest.mark.gpu


def _tiles(sizes):
    tiles = np.zeros(len(sizes), TILE)
    offset = 0
    for t, (w, h, pixel) in zip(tiles, sizes):
        t["width"], t["height"], t["pitch"], t["height_offset"] = w, h, w, offset
        t["pixel_width"], t["pixel_height"] = pixel, -pixel
        offset += w * h
    return TileSet(tiles=tiles, fractals=np.array([fractal(seed=3, wavelength=512.0, amplitude=5.0,
                                                           octaves=8)]),
                   elevation=0.0, crater_kernel=np.zeros((), CRATER_SHAPE_KERNEL),
                   crater_records=np.zeros(0, CRATER_RECORD), crater_data=np.zeros(0, np.float32),
                   crater_footprints=np.zeros(0), boulders=np.zeros((0, 5)))


def _run(device, sizes):
    ts = _tiles(sizes)
    out = np.zeros(ts.output_floats, np.float32)
    with Batch(device) as b:
        b.run(ts, out)
    return [ts.tile_view(out, i) for i in range(len(sizes))]


@pytest.mark.parametrize("size", [(1, 1), (40, 3)])
def test_a_pixel_past_the_floats_gives_nan(device, size):
    bad, good = _run(device, [(*size, 1e300), (65, 33, 0.5)])
    assert np.isnan(bad).all()
    np.testing.assert_array_equal(good, _run(device, [(65, 33, 0.5)])[0])
