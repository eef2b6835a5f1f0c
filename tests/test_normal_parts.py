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
extern "C" void ratios(const uint32_t* x, const uint32_t* y, int n, float* f, int* k) {
    for (int i = 0; i < n; ++i) {
        const tgb::NormalRatio r = tgb::normal_ratio(x[i], y[i]);
        f[i] = r.f;
        k[i] = r.k;
    }
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


def test_a_logarithm_takes_its_argument_rounded_once(parts):
    m, x, y = _draws()
    f, k = np.zeros(len(m), np.float32), np.zeros(len(m), np.int32)
    parts.ratios(*(a.ctypes.data_as(C.c_void_p) for a in (x, y)), len(m),
                 f.ctypes.data_as(C.c_void_p), k.ctypes.data_as(C.c_void_p))
    n = (1 << 53) - m
    # n = 2^e (1 + f): e the exponent of n / 0.75, exactly.
    bits = np.array([int(v).bit_length() for v in n], np.int64)
    e = np.where((bits >= 2) & (n >= 3 * (1 << np.maximum(bits - 2, 0))), bits, bits - 1)
    np.testing.assert_array_equal(k, e - 53)
    want = (n - (1 << e)).astype(np.float64) * 2.0 ** -e.astype(np.float64)
    np.testing.assert_array_equal(f, want.astype(np.float32))
