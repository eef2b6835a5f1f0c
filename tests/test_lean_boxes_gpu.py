"""The plain binned crater kernel, which numbers the cells of each staged crater's box, against the
general binned kernel (the same records under a mantling that nothing without a datum reads): grids
that end inside a bin, bins with more craters than a staged chunk, grids flipped along an axis,
cells without data."""

import ctypes as C

import numpy as np
import pytest

from terraingen_b200 import _native as N
from terraingen_b200 import workloads as W
from terraingen_b200.device import centered

pytestmark = pytest.mark.gpu

# width, height, pixel, crater density against the synthetic terrain's
GRIDS = [(1, 1, 0.5, 1.0), (31, 33, 0.5, 1.0), (65, 64, 1.0, 6.0), (100, 37, 0.25, 2.0),
         (33, 129, 2.0, 3.0)]


def apply(device, batch, grid, base, nodata):
    kernel, records, data, footprints = batch
    out = base.copy()
    N.check(device._lib.tg_craters_apply(
        device._handle, kernel.ctypes.data, kernel.nbytes, records.ctypes.data, len(records),
        data.ctypes.data, len(data), footprints.ctypes.data, C.byref(grid), out.ctypes.data,
        N.NoData(*nodata), N.TG_MEMORY_HOST, None))
    return out


@pytest.mark.parametrize("case", GRIDS, ids=lambda c: f"{c[0]}x{c[1]}@{c[2]:g}")
@pytest.mark.parametrize("profile", [0, 1, 2])
@pytest.mark.parametrize("flip", [False, True])
def test_matches_the_general_kernel(device, case, profile, flip):
    w, h, pixel, density = case
    spec = centered(w, h, pixel, 120.0, -75.0)
    c = density * 200000.0 / ((4097 * 0.5) ** 2 * (1.0 - 500.0 ** -2.0))
    shaping = W.config2_shaping()
    shaping.profile = profile
    batch = W.crater_batch(W.crater_population(5, c, 1.0, 500.0), spec, shaping=shaping)
    grid = spec.native()
    if flip:  # rows run south to north
        grid.origin_y -= h * pixel
        grid.pixel_height = pixel
    rng = np.random.default_rng(w)
    base = rng.normal(size=(h, w)).astype(np.float32)
    base[rng.random(base.shape) < 0.1] = -9999.0
    general = batch[0].copy()
    general["mantling"] = 1e-30
    got = apply(device, batch, grid, base, (2, -9999.0))
    want = apply(device, (general,) + batch[1:], grid, base, (2, -9999.0))
    assert (got[base == -9999.0] == -9999.0).all()
    # The crater tests' bound on the reference's heights.
    assert np.abs(got.astype(np.float64) - want).max() <= 1e-3
