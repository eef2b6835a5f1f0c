// Pairs of floats in a register pair, one instruction an operation on both, and Perlin noise on them
// with the corners' gradients read from a shared lattice table (noise.cu, batch.cu).
#pragma once

#include <stdint.h>

#include "noise_math.cuh"

namespace tgb {
namespace {

// Two floats (two cells) in a register pair, each operation one instruction on both
// with the same rounding as the scalar one.
struct Pair {
    unsigned long long v;
};
__device__ __forceinline__ Pair pair_of(float a, float b) {
    Pair p;
    asm("mov.b64 %0, {%1, %2};" : "=l"(p.v) : "f"(a), "f"(b));
    return p;
}
__device__ __forceinline__ void halves(Pair p, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p.v));
}
__device__ __forceinline__ Pair both(float a) {
    return pair_of(a, a);
}
__device__ __forceinline__ Pair mul2(Pair a, Pair b) {
    Pair p;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(p.v) : "l"(a.v), "l"(b.v));
    return p;
}
__device__ __forceinline__ Pair fma2(Pair a, Pair b, Pair c) {
    Pair p;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(p.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return p;
}
// Sums and differences as a 1 + b and b (-1) + a, which round as a + b and a - b do: the
// assembler fuses a packed product into a packed add (it leaves scalar ones alone under
// -fmad=false), but not into a multiply-add. `one` is a kernel argument, so it stays a factor.
struct Arithmetic {
    Pair one, minusOne;
    __device__ __forceinline__ explicit Arithmetic(float o) : one(both(o)), minusOne(both(-o)) {}
    __device__ __forceinline__ Pair add(Pair a, Pair b) const { return fma2(a, one, b); }
    __device__ __forceinline__ Pair sub(Pair a, Pair b) const { return fma2(b, minusOne, a); }
    __device__ __forceinline__ Pair add_down(Pair a, Pair b) const {
        Pair p;
        asm("fma.rm.f32x2 %0, %1, %2, %3;" : "=l"(p.v) : "l"(a.v), "l"(one.v), "l"(b.v));
        return p;
    }
    __device__ __forceinline__ Pair fade(Pair t) const {  // noise::fade
        const Pair inner =
            add(mul2(t, sub(mul2(t, both(6.0f)), both(15.0f))), both(10.0f));
        return mul2(mul2(mul2(t, t), t), inner);
    }
    __device__ __forceinline__ Pair lerp(Pair t, Pair a, Pair b) const {  // noise::lerp
        return add(mul2(t, sub(b, a)), a);
    }
};

// Adding 1.5 * 2^23 rounding down leaves floor(q) in the low bits of a float's significand, exact
// for |q| < 2^22: the lattice cell as an integer and, subtracting it again, as a float, without
// the conversion unit.
constexpr float kFloorShift = 12582912.0f;
constexpr uint32_t kFloorBits = 0x4b400000u;

// The gradients of one lattice corner of two cells.
struct GradientPair {
    Pair x, y, s;
};
__device__ __forceinline__ Pair gradient_dot2(const GradientPair& g, Pair x, Pair y) {
    return mul2(fma2(g.x, x, mul2(g.y, y)), g.s);  // noise::gradient_dot
}
// A table holds its points' x, then y, then s coefficients, kPoints of each.
template <uint32_t kPoints>
__device__ __forceinline__ GradientPair gradient_pair(const float* table, uint32_t a, uint32_t b) {
    return GradientPair{pair_of(table[a], table[b]), pair_of(table[kPoints + a], table[kPoints + b]),
                        pair_of(table[2 * kPoints + a], table[2 * kPoints + b])};
}
// The gradients of the corners of two lattice cells, in a table of `across` points a row.
struct CellPair {
    GradientPair g00, g10, g01, g11;
};
template <uint32_t kPoints>
__device__ __forceinline__ CellPair cell_pair(const float* table, uint32_t a, uint32_t b,
                                              uint32_t across) {
    return CellPair{gradient_pair<kPoints>(table, a, b),
                    gradient_pair<kPoints>(table, a + 1u, b + 1u),
                    gradient_pair<kPoints>(table, a + across, b + across),
                    gradient_pair<kPoints>(table, a + across + 1u, b + across + 1u)};
}

}  // namespace
}  // namespace tgb
