"""Seams over gaps without a whole coarse post: the sweeps of the only level all but solve them, to
the direct solve's field."""

import numpy as np
import pytest

from oracle import seams as S

pytestmark = pytest.mark.gpu


def _data(kind, w, h):
    y, x = np.mgrid[0:h, 0:w]
    return {"columns": x % 9 > 0, "rows": y % 7 > 0, "diagonals": (x + y) % 23 > 1,
            "grid": (x % 2 == 0) & (y % 2 == 0)}[kind].astype(np.uint8)


@pytest.mark.parametrize("kind", ["columns", "rows", "diagonals", "grid"])
@pytest.mark.parametrize("mode, most", [("height", 3), ("slope", 6)])
def test_thin_gaps_take_few_iterations(device, kind, mode, most):
    w, h = 83, 61
    rng = np.random.default_rng(7)
    data = _data(kind, w, h)
    y, x = np.mgrid[0:h, 0:w]
    diff = (2.0 + np.sin(x / 9.0) + 0.5 * np.cos(y / 5.0) +
            0.05 * rng.normal(size=(h, w))).astype(np.float32)
    diff[data == 0] = np.nan
    got, stats = device.seam_solve(data, diff, 1.0, 1.0, mode, decay_length=30.0)
    assert stats["unknowns"] > 0 and stats["levels"] == 1
    assert 1 <= stats["iterations"] <= most
    want = S.solve(data, diff, 1.0, 1.0, mode, 30.0)
    # Float fields of a few meters from a residual of 1e-10; the seam tests' bound.
    assert np.abs(got.astype(np.float64) - want).max() <= 1e-4
