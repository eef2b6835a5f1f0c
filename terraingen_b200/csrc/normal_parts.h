// The integer part of a node's normal (ds_tile.cuh): the arguments its logarithm and its cosine
// take, formed exactly from a draw's words and rounded once.
#pragma once

#include <stdint.h>

#include "layouts.h"

namespace tgb {

// A draw u2 = m 2^-53, m the 53 bits (z >> 5) 2^26 + (w >> 6) (RandomStream's NextDouble): twice
// its share of a turn, 2 u2, taken modulo 2 into [-1, 1), in units of 2^-52. Reading the top word
// as a signed number is the modulus, so one widening multiply-add forms all 53 bits.
TG_HD inline float normal_turn(uint32_t z, uint32_t w) {
    return float(int64_t(int32_t(z) >> 5) * (int64_t(1) << 26) + int64_t(w >> 6));
}

// The bit of a word's highest one.
TG_HD inline int top_bit(uint32_t v) {
#ifdef __CUDA_ARCH__
    return 31 - __clz(int(v));
#else
    return 31 - __builtin_clz(v);
#endif
}

// 1 - u1 for a draw u1 = m 2^-53, m the 53 bits of (x, y) as above: n 2^-53 with n = 2^53 - m, as
// 2^k (1 + f) with 1 + f in [0.75, 1.5). f is an integer difference, exact before its one rounding,
// so it is relatively accurate where it is small (u1 near 0 above all, where the logarithm goes to
// 0). n is H 2^26 + L; its top two bits lie in H, but for n below 2^27, which is shifted there.
struct NormalRatio {
    float f;
    int k;
};
TG_HD inline NormalRatio normal_ratio(uint32_t x, uint32_t y) {
    const uint32_t high = x >> 5, low = y >> 6;
    uint32_t h = (1u << 27) - high - (low != 0u ? 1u : 0u);
    uint32_t l = (0u - low) & 0x3ffffffu;
    const bool few = h < 2u;
    h = few ? (h << 26) | l : h;
    l = few ? 0u : l;
    // n's exponent, one more from 1.5 times its power of two on.
    const int t = top_bit(h);
    const int e = t + int(((h << 1) >> t) & 1u);
    const int64_t rest = int64_t(int32_t(h - (1u << e))) * (int64_t(1) << 26) + int64_t(l);
    const int k = e - 27 - (few ? 26 : 0);
    const uint32_t scale = uint32_t(127 - 26 - e) << 23;  // 2^-(26 + e)
#ifdef __CUDA_ARCH__
    return NormalRatio{float(rest) * __uint_as_float(scale), k};
#else
    float s;
    __builtin_memcpy(&s, &scale, 4);
    return NormalRatio{float(rest) * s, k};
#endif
}

}  // namespace tgb
