"""The bounds under which the source kernels look lattice cells up in a table without checking the
place: only positions that are numbers inside the table's box."""

from __future__ import annotations

import ctypes as C
import math

import pytest

from host_math import compiled

NAN, INF = math.nan, math.inf


@pytest.fixture(scope="module")
def box(tmp_path_factory):
    lib = compiled(tmp_path_factory.mktemp("lattice"), """
#include "lattice_box.h"
using namespace tgb;
extern "C" int fbm_tabled(double x0, double y0, double pixel, double ox, double oy, float f) {
    const Grid g{64, 48, x0, pixel, 0.0, y0, 0.0, -pixel};
    return lattice_tabled(lattice_reach(g, Positions{ox, oy, nullptr, nullptr}), f);
}
""")
    lib.fbm_tabled.argtypes = [C.c_double] * 5 + [C.c_float]
    return lib


@pytest.mark.parametrize("origin", [(NAN, 0.0), (0.0, NAN), (NAN, NAN), (INF, 0.0), (0.0, -INF),
                                    (INF, NAN), (-INF, INF), (1e39, 0.0), (0.0, -1e39)])
@pytest.mark.parametrize("frequency", [1.0 / 512.0, 1e-38, 1e-45])
def test_positions_that_are_no_floats_are_not_tabled(box, origin, frequency):
    assert not box.fbm_tabled(100.0, -50.0, 0.5, *origin, frequency)


@pytest.mark.parametrize("frequency", [NAN, INF, 1e30])
@pytest.mark.parametrize("x0", [0.0, 100.0])
def test_frequencies_without_a_place_are_not_tabled(box, frequency, x0):
    assert not box.fbm_tabled(x0, 0.0, 0.5, 0.0, 0.0, frequency)


def test_ordinary_positions_are_tabled_up_to_their_range(box):
    assert box.fbm_tabled(0.0, 0.0, 0.5, 0.0, 0.0, 1.0 / 512.0)
    assert box.fbm_tabled(1.0e6, -1.0e6, 0.5, 0.0, 0.0, 0.125)
    assert not box.fbm_tabled(1.1e6, -1.1e6, 0.5, 0.0, 0.0, 0.125)
