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

}  // namespace tgb
