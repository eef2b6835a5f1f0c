"""The single-fractal fBm kernel against the general stack kernel, which evaluates the same
octaves cell by cell: the same heights at the edges of its tiles and rows, for octaves that fit a
block's lattice table and octaves that do not, far positions and no-data cells."""

import ctypes as C

import numpy as np
import pytest

from terraingen_b200 import _native as N
from terraingen_b200.layouts import fractal, noise_layer_kernel

pytestmark = pytest.mark.gpu

# width, height, pixel, x0, y0
GRIDS = [
    (1, 1, 0.5, 0.0, 0.0),
    (31, 15, 0.5, -7.0, 3.0),
    (33, 17, 0.5, 100.0, -50.0),
    (65, 129, 5.0, 1e4, -2e4),      # fine octaves exceed the tables
    (257, 63, 0.5, 1.7e6, -1.2e6),  # fine octaves lie past the tables' range
    (1601, 1537, 0.7, -300.0, 500.0),  # eight rows a thread, ragged
]


@pytest.mark.parametrize("case", GRIDS, ids=lambda c: f"{c[0]}x{c[1]}@{c[3]:g}")
@pytest.mark.parametrize("octaves", [1, 8, 13])
def test_matches_the_stack_kernel(device, case, octaves):
    w, h, pixel, x0, y0 = case
    grid = N.Grid(w, h, x0, pixel, 0.0, y0, 0.0, -pixel)
    one = fractal(seed=9, wavelength=300.0, amplitude=7.0, octaves=octaves, lacunarity=2.1,
                  gain=0.55)
    silent = fractal(seed=4, wavelength=50.0, amplitude=0.0, octaves=1)
    got, want = np.zeros((h, w), np.float32), np.zeros((h, w), np.float32)
    for fractals, out in (([one], got), ([one, silent], want)):
        f = np.array(fractals)
        N.check(device._lib.tg_noise_source(device._handle, f.ctypes.data, len(f), 1.25,
                                            C.byref(grid), out.ctypes.data, N.TG_MEMORY_HOST,
                                            None))
    np.testing.assert_array_equal(got, want)


def test_layer_skips_nodata(device):
    rng = np.random.default_rng(3)
    grid = N.Grid(77, 39, 5.0, 0.5, 0.0, -3.0, 0.0, -0.5)
    base = rng.normal(size=(39, 77)).astype(np.float32)
    base[rng.random(base.shape) < 0.3] = -9999.0
    one = fractal(seed=2, wavelength=64.0, amplitude=3.0, octaves=7)
    silent = fractal(seed=4, wavelength=50.0, amplitude=0.0, octaves=1)
    outs = []
    for fractals in ([one], [one, silent]):
        k = noise_layer_kernel(fractals)
        out = base.copy()
        N.check(device._lib.tg_noise_layer(device._handle, k.ctypes.data, k.nbytes,
                                           C.byref(grid), 1.0, 2.0, out.ctypes.data,
                                           N.NoData(2, -9999.0), N.TG_MEMORY_HOST, None))
        outs.append(out)
    np.testing.assert_array_equal(outs[0], outs[1])
    assert (outs[0][base == -9999.0] == -9999.0).all()


@pytest.mark.parametrize("origin", [(np.nan, 0.0), (0.0, np.nan), (np.inf, np.nan), (-np.inf, 0.0),
                                    (1e39, 0.0)])
def test_origins_that_are_no_floats_give_nan(device, origin):
    """Such positions are not looked up in a table; every octave is NaN, as the fractal's sum."""
    grid = N.Grid(65, 33, 5.0, 0.5, 0.0, -3.0, 0.0, -0.5)
    k = noise_layer_kernel([fractal(seed=2, wavelength=64.0, amplitude=3.0, octaves=7)])
    out = np.zeros((33, 65), np.float32)
    N.check(device._lib.tg_noise_layer(device._handle, k.ctypes.data, k.nbytes, C.byref(grid),
                                       *origin, out.ctypes.data, N.NoData(0, 0.0),
                                       N.TG_MEMORY_HOST, None))
    assert np.isnan(out).all()


@pytest.mark.parametrize("side", [833, 865])
def test_a_grid_is_its_windows_on_both_sides_of_the_rows_rule(device, side):
    """Two rows a thread on the window, and on the smaller grid; eight on the larger."""
    f = np.array([fractal(seed=9, wavelength=300.0, amplitude=7.0, octaves=9)])

    def source(x0, y0, n):
        out = np.zeros((n, n), np.float32)
        N.check(device._lib.tg_noise_source(device._handle, f.ctypes.data, 1, 0.0,
                                            C.byref(N.Grid(n, n, x0, 0.5, 0.0, y0, 0.0, -0.5)),
                                            out.ctypes.data, N.TG_MEMORY_HOST, None))
        return out

    whole = source(-100.0, 50.0, side)
    for row, col in ((0, 0), (333, 417), (side - 61, side - 61)):
        np.testing.assert_array_equal(source(-100.0 + 0.5 * col, 50.0 - 0.5 * row, 61),
                                      whole[row:row + 61, col:col + 61])
