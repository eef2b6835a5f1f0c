"""The boulder bake, whose block numbers its boulders' cells in one sequence, against the domes in
numpy: grids that end inside a bin, bins of more boulders than a staged chunk, boulders over bins'
edges and off the grid, heights of either sign, cells without data."""

import numpy as np
import pytest

from terraingen_b200.device import centered

pytestmark = pytest.mark.gpu


def baked(stones, grid, heights, width, nodata):
    """DomeHeight averaged over `width`, max-composited on the heights before the layer."""
    best = heights.astype(np.float64)
    x = grid.x0 + (np.arange(grid.width) + 0.5) * grid.pixel
    y = grid.y0 - (np.arange(grid.height) + 0.5) * grid.pixel

    def area(u):
        u = np.clip(u, -1.0, 1.0)
        return 0.5 * (u * np.sqrt(1.0 - u * u) + np.arcsin(u))

    for bx, by, diameter, exposed, weight in stones:
        d, r = np.hypot(x[None, :] - bx, y[:, None] - by), 0.5 * diameter
        lift = exposed * (area((d + 0.5 * width) / r) - area((d - 0.5 * width) / r)) * r / width
        drawn = (lift > 0.0) & (weight > 0.0)
        best = np.maximum(best, np.where(drawn, heights.astype(np.float64) + weight * lift, best))
    out = best.astype(np.float32)
    out[heights == nodata] = nodata
    return out


@pytest.mark.parametrize("size", [(1, 1), (31, 33), (65, 40), (96, 32)])
@pytest.mark.parametrize("count", [1, 40, 700])
def test_matches_the_domes(device, size, count):
    rng = np.random.default_rng(count + size[0])
    grid = centered(*size, 0.5, 30.0, -12.0)
    span = np.array([grid.width, grid.height]) * grid.pixel
    stones = np.zeros((count, 5))
    stones[:, 0] = grid.x0 + rng.uniform(-0.2, 1.2, count) * span[0]
    stones[:, 1] = grid.y0 - rng.uniform(-0.2, 1.2, count) * span[1]
    stones[:, 2] = rng.uniform(0.6, 6.0, count)
    stones[:, 3] = 0.5 * stones[:, 2]
    stones[:, 4] = rng.choice([0.0, 0.4, 1.0], count)
    heights = rng.normal(scale=3.0, size=(grid.height, grid.width)).astype(np.float32)
    heights[rng.random(heights.shape) < 0.1] = -9999.0
    got = heights.copy()
    device.boulders_bake(stones, grid, got, grid.pixel, nodata=(2, -9999.0))
    want = baked(stones, grid, heights, grid.pixel, np.float32(-9999.0))
    # The same doubles rounded once to float: at most a rounding apart.
    np.testing.assert_allclose(got, want, rtol=2.0 ** -23, atol=2e-7)
