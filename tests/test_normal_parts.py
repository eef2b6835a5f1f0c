"""The arguments a diamond-square node's normal is made of, against their exact values: each is an
integer expression of the whole 53-bit draw, rounded once to float."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from host_math import compiled


@pytest.fixture(scope="module")
def parts(tmp_path_factory):
    lib = compiled(tmp_path_factory.mktemp("normal"), """
#include "normal_parts.h"
extern "C" void turns(const uint32_t* z, const uint32_t* w, int n, float* out) {
    for (int i = 0; i < n; ++i) out[i] = tgb::normal_turn(z[i], w[i]);
}
""")
    return lib


def _draws():
    """Words of a draw (the low 5 and 6 bits are not part of it) and its 53 bits."""
    rng = np.random.default_rng(11)
    edge = [0, 1, 2, 3, 1 << 25, (1 << 26) - 1, 1 << 26, (1 << 51) - 1, 1 << 51, (1 << 51) + 1,
            (1 << 52) - 1, 1 << 52, (1 << 52) + 1, 3 << 51, (1 << 53) - 2, (1 << 53) - 1]
    near = [int(c) + int(d) for c in (0, 1 << 51, 1 << 52, 3 << 51, 1 << 53)
            for d in rng.integers(-(1 << 30), 1 << 30, 500)]
    low = [int(v) >> int(s) for v, s in zip(rng.integers(0, 1 << 53, 2000),
                                            rng.integers(0, 53, 2000))]
    m = np.array([v % (1 << 53) for v in edge + near + low +
                  [int(v) for v in rng.integers(0, 1 << 53, 20000)]], np.int64)
    high = ((m >> 26) << 5).astype(np.uint32) | rng.integers(0, 32, len(m)).astype(np.uint32)
    rest = ((m & ((1 << 26) - 1)) << 6).astype(np.uint32) | \
        rng.integers(0, 64, len(m)).astype(np.uint32)
    return m, high, rest


def test_a_turn_takes_all_bits_of_its_draw(parts):
    m, z, w = _draws()
    got = np.zeros(len(m), np.float32)
    parts.turns(z.ctypes.data_as(C.c_void_p), w.ctypes.data_as(C.c_void_p), len(m),
                got.ctypes.data_as(C.c_void_p))
    # 53-bit integers are exact in double, so this rounds once.
    want = np.where(m >= 1 << 52, m - (1 << 53), m).astype(np.float64).astype(np.float32)
    np.testing.assert_array_equal(got, want)
