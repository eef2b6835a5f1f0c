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
extern "C" int batch_tabled(float fx, float fy, float ax, float ay, float bx, float by,
                            uint32_t c0, uint32_t c1, uint32_t r0, uint32_t r1) {
    return lattice_boxed(lattice_box(OctaveAnchor{0, 0, fx, fy, ax, ay, bx, by}, c0, c1, r0, r1));
}
""")
    lib.batch_tabled.argtypes = [C.c_float] * 6 + [C.c_uint32] * 4
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


# Bins of a tile: the only cell, a first bin, a later one.
BINS = [(0, 0, 0, 0), (0, 31, 0, 31), (32, 63, 64, 95)]


@pytest.mark.parametrize("bin", BINS)
@pytest.mark.parametrize("field", range(6))
@pytest.mark.parametrize("value", [NAN, INF, -INF, 3e38])
def test_a_bin_is_tabled_only_where_all_its_cells_are_in_range(box, bin, field, value):
    anchor = [0.25, 0.75, 1e-3, -2e-4, 2e-4, 1e-3]  # fx, fy, ax, ay, bx, by
    assert box.batch_tabled(*anchor, *bin)
    anchor[field] = value
    fx, fy, ax, ay, bx, by = anchor
    c0, c1, r0, r1 = bin
    cells = [q for c in {c0, c1} for r in {r0, r1}
             for q in (fx + r * ay + c * ax, fy + r * by + c * bx)]
    in_range = all(abs(q) < 2e6 for q in cells)  # False for NaN
    assert box.batch_tabled(*anchor, *bin) == in_range


@pytest.mark.parametrize("bin", BINS)
def test_a_bin_of_an_overflowing_pixel_is_not_tabled(box, bin):
    assert not box.batch_tabled(0.0, 0.0, INF, 0.0, 0.0, INF, *bin)
    assert not box.batch_tabled(0.0, 0.0, INF, -INF, INF, INF, *bin)
