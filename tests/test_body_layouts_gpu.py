"""The sphere's kernel with the arguments of a stack of few octaves and with those of any stack: a
fractal that adds nothing but octaves changes no bit."""

import ctypes as C

import numpy as np
import pytest

from terraingen_b200 import _native as N
from terraingen_b200.layouts import fractal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("octaves", [1, 15, 16])
@pytest.mark.parametrize("warp", [0.0, 25.0])
def test_more_octaves_than_the_small_arguments_hold(device, octaves, warp):
    one = fractal(seed=9, wavelength=900.0, amplitude=7.0, octaves=octaves, warp_amplitude=warp,
                  warp_wavelength=300.0)
    grid = N.Grid(75, 41, 10.0, 1e-3, 0.0, 5.0, 0.0, -1e-3)
    outs = []
    # 16 octaves with a warp's 12 more, twice and a third time; 17 octaves.
    for more in ([], [(16, 0.0)], [(16, 25.0), (16, 25.0)], [(17, 0.0)], [(32, 0.0)]):
        f = np.array([one] + [fractal(seed=4, wavelength=50.0, amplitude=0.0, octaves=o,
                                      warp_amplitude=w, warp_wavelength=80.0) for o, w in more])
        out = np.zeros((41, 75), np.float32)
        N.check(device._lib.tg_noise_source_body(device._handle, f.ctypes.data, len(f), 1.25,
                                                 C.byref(grid), 1737400.0, out.ctypes.data,
                                                 N.TG_MEMORY_HOST, None))
        outs.append(out)
    assert np.ptp(outs[0]) > 0.0
    for out in outs[1:]:
        np.testing.assert_array_equal(out, outs[0])
