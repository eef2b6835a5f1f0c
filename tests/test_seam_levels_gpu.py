"""The seam solve over gaps whose coarser levels are ragged or vanish (a coarse post is an unknown
only where all four finer posts are): thin and odd gaps, lattices whose rows end inside a word of
the unknown masks, against the direct solve of the same system."""

import numpy as np
import pytest

from oracle import seams as S

pytestmark = pytest.mark.gpu

# lattice width, height, gap (col0, row0, col1, row1)
GAPS = [
    (33, 17, (9, 6, 10, 11)),     # one column: no coarse post at all
    (65, 31, (20, 5, 22, 26)),    # two columns off the pairs
    (97, 40, (31, 8, 34, 33)),
    (64, 64, (10, 10, 50, 51)),   # a hole whose levels end at a few posts
    (129, 67, (60, 0, 129, 67)),  # a gap over the lattice's edges
]


@pytest.mark.parametrize("gap", GAPS, ids=lambda g: f"{g[0]}x{g[1]}")
@pytest.mark.parametrize("mode", ["height", "slope"])
@pytest.mark.parametrize("sweeps", [1, 2, 3])
def test_matches_the_direct_solve(device, gap, mode, sweeps):
    w, h, (c0, r0, c1, r1) = gap
    rng = np.random.default_rng(w + h)
    data = np.ones((h, w), np.uint8)
    data[r0:r1, c0:c1] = 0
    y, x = np.mgrid[0:h, 0:w]
    diff = (2.0 + np.sin(x / 9.0) + 0.5 * np.cos(y / 5.0) +
            0.05 * rng.normal(size=(h, w))).astype(np.float32)
    diff[data == 0] = np.nan
    got, stats = device.seam_solve(data, diff, 1.0, 1.0, mode, decay_length=7.0, sweeps=sweeps)
    want = S.solve(data, diff, 1.0, 1.0, mode, 7.0)
    assert stats["unknowns"] > 0 and stats["iterations"] < 200
    # Float fields of a few meters from a residual of 1e-10; the seam tests' bound.
    assert np.abs(got.astype(np.float64) - want).max() <= 1e-4
