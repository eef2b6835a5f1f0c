"""Fractal stacks over a grid against the same cells evaluated a row at a time: the stack kernel
takes four cells of a column together and keeps a lattice cell's hashes between them, which must
not show, for every basis, type and blend, warped or not."""

import numpy as np
import pytest

from terraingen_b200 import centered
from terraingen_b200.layouts import fractal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("basis", range(7))
@pytest.mark.parametrize("kind", range(4))
@pytest.mark.parametrize("height", [1, 3, 4, 37])
def test_rows_alone_and_together(device, basis, kind, height):
    grid = centered(45, height, 0.5, 64.0, -32.0)
    fractals = np.array([
        fractal(seed=3, wavelength=20.0, amplitude=3.0, octaves=3, basis=basis, type=kind,
                warp_amplitude=4.0 if basis % 2 else 0.0, warp_wavelength=16.0),
        fractal(seed=5, wavelength=9.0, amplitude=2.0, octaves=2, basis=(basis + 2) % 7,
                type=(kind + 1) % 4, blend=kind),
    ])
    got = np.zeros((height, 45), np.float32)
    device.noise_source(fractals, grid, got, elevation=0.5)
    for row in range(height):
        strip = centered(45, 1, 0.5, 64.0, grid.y0 - 0.5 * row - 0.25)
        want = np.zeros((1, 45), np.float32)
        device.noise_source(fractals, strip, want, elevation=0.5)
        np.testing.assert_array_equal(got[row], want[0])
