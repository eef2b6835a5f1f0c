"""The lean crater kernel's profile against the general one, both compiled for the host: where the
radius is a power of two their radii are the same floats, and each quotient is rounded as the
general profile's, so the heights have its bits."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from host_math import compiled

SOURCE = """
#include <cuda_runtime.h>
#include <algorithm>
#include <cmath>
#include <cstring>
using std::min; using std::max;
#define __noinline__ __attribute__((noinline))
template <typename T> T __ldg(const T* p) { return *p; }
static float __uint_as_float(unsigned v) { float f; std::memcpy(&f, &v, 4); return f; }
static unsigned __float_as_uint(float f) { unsigned v; std::memcpy(&v, &f, 4); return v; }
static float __int_as_float(int v) { return __uint_as_float(unsigned(v)); }
static int __float_as_int(float f) { return int(__float_as_uint(f)); }
static unsigned __byte_perm(unsigned, unsigned, unsigned) { return 0; }
static float __frcp_rn(float x) { return 1.0f / x; }
static float __fdividef(float x, float y) { return x / y; }
#include "crater_math.cuh"
using namespace tgb;
static CraterShapeKernel kernel(int complex, uint32_t rim) {
    CraterShapeKernel k{};
    k.profile.rim = rim;
    k.profile.complex = complex;
    k.profile.transitionDiameter = 4.0f;
    k.profile.floorCoefficient = 0.19f;
    k.profile.floorExponent = 1.25f;
    k.profile.peakHeightCoefficient = 0.032f;
    k.profile.peakHeightExponent = 0.9f;
    k.profile.peakWidthCoefficient = 0.23f;
    k.profile.peakWidthExponent = 1.1f;
    k.profile.peakFitMaxDiameter = 100.0f;
    k.profile.complexReachRadii = 3.0f;
    k.profile.ejectaExponent = 3.0f;
    k.reachRadii = 3.0f;
    return k;
}
static CraterRecord record(float diameter) {
    CraterRecord c{};
    c.diameter = diameter;
    c.resolution = 1.0f;
    c.ellipticity = 1.0f;
    c.freshDepth = 0.196f;
    c.freshRim = 0.036f;
    c.currentDepth = 0.131f;
    c.currentRim = 0.027f;
    return c;
}
// The lean and the general profile at n distances; the constants the ejecta's fall is made of.
extern "C" void profiles(int complex, uint32_t rim, float diameter, const float* distance, int n,
                         float* lean, float* general, float* constants) {
    const CraterShapeKernel k = kernel(complex, rim);
    const CraterRecord c = record(diameter);
    const crater::LeanCrater l =
        crater::lean_crater(k, c, nullptr, 0, int4{0, 0, 0, 0}, 0.0f);
    const crater::LeanKernel lk =
        complex ? crater::lean_kernel(k) : crater::LeanKernel{0.0f, 0.0f};
    const crater::State s{c.freshDepth, c.freshRim, c.currentDepth, c.currentRim};
    for (int i = 0; i < n; ++i) {
        lean[i] = crater::lean_height(k, lk, l, distance[i]);
        general[i] = crater::fresh_height(k.profile, distance[i], diameter, s);
    }
    constants[0] = c.currentRim * diameter;
    constants[1] = lk.edge;
    constants[2] = lk.fallScale;
    constants[3] = l.floorShare;
    constants[4] = l.peakBase;
}
"""


@pytest.fixture(scope="module")
def profiles(tmp_path_factory):
    lib = compiled(tmp_path_factory.mktemp("lean"), SOURCE)

    def run(complex, rim, diameter, distance):
        lean, general = np.zeros_like(distance), np.zeros_like(distance)
        constants = np.zeros(5, np.float32)
        lib.profiles(C.c_int(complex), C.c_uint32(rim), C.c_float(diameter),
                     distance.ctypes.data_as(C.c_void_p), len(distance),
                     lean.ctypes.data_as(C.c_void_p), general.ctypes.data_as(C.c_void_p),
                     constants.ctypes.data_as(C.c_void_p))
        return lean, general, constants

    return run


def _radii(low, high):
    rng = np.random.default_rng(4)
    return np.concatenate([np.linspace(low, high, 20001), rng.uniform(low, high, 20000)])


def test_the_ejecta_falls_by_a_rounded_reciprocal(profiles):
    distance = (16.0 * _radii(1.0, 3.2)).astype(np.float32)
    lean, _, (rim, edge, scale, _, _) = profiles(1, 0, 32.0, distance)
    x = distance * np.float32(1.0 / 16.0)
    fall = np.float32(1.0) / (x * x * x)
    want = np.where(x >= np.float32(3.0), np.float32(0.0), rim * (fall - edge) * scale)
    assert want.dtype == np.float32
    np.testing.assert_array_equal(lean, want)


def test_a_complex_wall_rises_by_a_rounded_quotient(profiles):
    # Outside the peak, where the dome adds nothing.
    distance = (16.0 * _radii(0.2, 1.0)).astype(np.float32)
    lean, general, (_, _, _, floor_share, peak_base) = profiles(1, 0, 32.0, distance)
    wall = (distance >= peak_base) & (distance < 16.0)
    assert floor_share < 0.2 and wall.sum() > 20000
    np.testing.assert_array_equal(lean[wall], general[wall])


def test_a_peaks_dome_falls_by_a_rounded_quotient(profiles):
    _, _, (_, _, _, floor_share, peak_base) = profiles(1, 0, 32.0, np.zeros(1, np.float32))
    distance = (peak_base * _radii(0.0, 1.1)).astype(np.float32)
    lean, general, _ = profiles(1, 0, 32.0, distance)
    assert 0.0 < peak_base < 16.0
    np.testing.assert_array_equal(lean, general)


@pytest.mark.parametrize("rim", [0, 1, 2])
def test_a_simple_crater_is_the_general_profile(profiles, rim):
    # The edges of its pieces, the floats beside them, and all between.
    edges = np.float32([0.2, 0.98, 1.0, 1.02, 1.5])
    x = np.concatenate([_radii(0.0, 1.6).astype(np.float32), edges,
                        np.nextafter(edges, np.float32(0.0)), np.nextafter(edges, np.float32(2.0))])
    lean, general, _ = profiles(0, rim, 4.0, np.float32(2.0) * x)
    np.testing.assert_array_equal(lean, general)
