"""Worley noise against the definition's 5 x 5 cells in numpy's single precision, the same bits:
points whose nearest feature, or second nearest, lies beyond the 3 x 3 cells searched first."""

import ctypes as C

import numpy as np
import pytest

from terraingen_b200 import _native as N
from terraingen_b200.layouts import fractal

pytestmark = pytest.mark.gpu

F = np.float32


def _pcg3d(x, y, z):
    with np.errstate(over="ignore"):
        x, y, z = (np.asarray(v, np.uint32) * np.uint32(1664525) + np.uint32(1013904223)
                   for v in (x, y, z))
        x = x + y * z
        y = y + z * x
        z = z + x * y
        x, y, z = (v ^ (v >> np.uint32(16)) for v in (x, y, z))
        x = x + y * z
        y = y + z * x
        z = z + x * y
    return x, y, z


def _unit(h):
    return (h >> np.uint32(8)).astype(F) * F(2.0 ** -24)


def _squares(x, y, seed):
    """The 5 x 5 cells' squared distances, row by row, and their points' values."""
    cx, cy = np.floor(x), np.floor(y)
    fx, fy = x - cx, y - cy
    squares, values = [], []
    for dy in range(-2, 3):
        for dx in range(-2, 3):
            with np.errstate(over="ignore"):
                h = _pcg3d((cx.astype(np.int64) + dx).astype(np.uint32),
                           (cy.astype(np.int64) + dy).astype(np.uint32), np.uint32(seed))
            px, py = F(dx) + _unit(h[1]) - fx, F(dy) + _unit(h[2]) - fy
            squares.append(px * px + py * py)
            values.append(F(2.0) * _unit(h[0]) - F(1.0))
    return np.array(squares), np.array(values)


@pytest.mark.parametrize("basis", [3, 4, 5, 6], ids=["F1", "F2", "F2-F1", "Voronoi"])
def test_matches_all_cells(device, basis):
    n, pixel, seed = 512, 0.37, 21
    key = _pcg3d(*(np.array([v], np.uint32) for v in (seed, 0, 0)))
    f = np.array([fractal(seed=seed, wavelength=1.0, amplitude=1.0, octaves=1, basis=basis)])
    got = np.zeros((n, n), np.float32)
    N.check(device._lib.tg_noise_source(device._handle, f.ctypes.data, 1, 0.0,
                                        C.byref(N.Grid(n, n, -3.0, pixel, 0.0, 5.0, 0.0, -pixel)),
                                        got.ctypes.data, N.TG_MEMORY_HOST, None))
    x = (-3.0 + (np.arange(n) + 0.5) * pixel).astype(F)[None, :] + np.zeros((n, 1), F)
    y = (5.0 - (np.arange(n) + 0.5) * pixel).astype(F)[:, None] + np.zeros((1, n), F)
    squares, values = _squares(x + _unit(key[1]), y + _unit(key[2]), key[0][0])
    order = np.sort(squares, axis=0)
    f1, f2 = np.sqrt(order[0]), np.sqrt(order[1])
    assert (f1 >= 1.0).sum() > 20 and ((f1 < 1.0) & (f2 >= 1.0)).sum() > 1000
    if basis == 6:
        want = np.take_along_axis(values, squares.argmin(axis=0)[None], axis=0)[0]
    else:
        d = {3: f1 * F(0.707106781186547524), 4: f2 * F(0.447213595499957939),
             5: (f2 - f1) * F(0.447213595499957939)}[basis]
        want = F(2.0) * np.minimum(d, F(1.0)) - F(1.0)
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("basis", [0, 1, 2, 3, 6])
def test_a_stack_that_reads_second_nearest_points_changes_no_other_basis(device, basis):
    """The kernel with that search and the one without."""
    grid = N.Grid(97, 45, 10.0, 0.7, 0.0, 5.0, 0.0, -0.7)
    one = fractal(seed=9, wavelength=20.0, amplitude=7.0, octaves=4, basis=basis, type=1)
    outs = []
    for other in (1, 4, 5):
        f = np.array([one, fractal(seed=4, wavelength=50.0, amplitude=0.0, octaves=1,
                                   basis=other)])
        out = np.zeros((45, 97), np.float32)
        N.check(device._lib.tg_noise_source(device._handle, f.ctypes.data, 2, 0.0, C.byref(grid),
                                            out.ctypes.data, N.TG_MEMORY_HOST, None))
        outs.append(out)
    assert np.ptp(outs[0]) > 0.0
    np.testing.assert_array_equal(outs[1], outs[0])
    np.testing.assert_array_equal(outs[2], outs[0])
