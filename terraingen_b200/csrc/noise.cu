// fBm noise sources and noise layers over a grid (SyntheticSource::FillSamples,
// src/sources/synthetic_source.cpp:87; NoiseLayer::ApplySamples, src/layers/noise_layer.cpp:95).
//
// Compiled with -fmad=false: positions (double) and the lattice math (float) round exactly as the
// reference's -ffp-contract=off build does, so heights carry the reference CPU path's bits.
//
// The kernels are ALU-bound (4 bytes written per cell against some 60 float operations an octave).
// Each thread evaluates several cells of one column, so a warp covers 32 consecutive columns and
// every store is a full 128-byte line.
#include <algorithm>
#include <cmath>

#include "kernels.h"
#include "lattice_box.h"
#include "noise_math.cuh"
#include "packed.cuh"

namespace tgb {
namespace {

constexpr int kBlockX = 32;
constexpr int kBlockY = 8;

__device__ __forceinline__ bool is_nodata(NoData nd, float h) {
    if (nd.mode == 1u) {
        return isnan(h);
    }
    return nd.mode != 0u && h == nd.value;
}

// The float x of a column's cell centers measured from the origin (src/gpu/kernel.cpp:56-62):
// computed in double as Raster::CellCenter does, then narrowed.
__device__ __forceinline__ float column_x(const Grid& g, const Positions& at, uint32_t col,
                                          uint32_t row) {
    if (at.xs != nullptr) {
        return at.xs[col];
    }
    const double x = g.originX + (double(col) + 0.5) * g.pixelWidth +
                     (double(row) + 0.5) * g.rowRotation;
    return float(x - at.originX);
}

__device__ __forceinline__ float row_y(const Grid& g, const Positions& at, uint32_t col,
                                       uint32_t row) {
    if (at.ys != nullptr) {
        return at.ys[row];
    }
    const double y = g.originY + (double(col) + 0.5) * g.colRotation +
                     (double(row) + 0.5) * g.pixelHeight;
    return float(y - at.originY);
}

// One enabled Perlin fBm fractal without a warp, the configurations' source: its per-octave
// constants are computed once on the host, with the same float recurrences Fractal2 runs per
// cell (fractal.h:219-240), so each cell performs exactly the reference's operations on them.
constexpr int kMaxOctaves = 32;
// Lattice points a block's tables hold in all (3 floats each): 15 KB, so shared memory does not
// limit a block's occupancy below what its registers do.
constexpr uint32_t kTablePoints = 1280;
constexpr uint32_t kTableSteps = kTablePoints / 32;
struct Octaves {
    int count;
    float amplitude;
    float total;                       // sum of the weights
    float one;                         // 1
    uint32_t tabled;                   // bit o: octave o reads its block's lattice table
    uint32_t seedTerm[kMaxOctaves];    // octave seed, through pcg3d's first LCG step
    float ox[kMaxOctaves], oy[kMaxOctaves];
    float frequency[kMaxOctaves], weight[kMaxOctaves];
    float tc[kMaxOctaves], ts[kMaxOctaves];
    // A tabled octave's points: its columns and their reciprocal, how many there are, and its
    // first point in the table, a multiple of 32: the points are hashed 32 to a warp's step, and
    // step k of a block's `steps` belongs to octave stepOctave[k].
    uint16_t across[kMaxOctaves], points[kMaxOctaves], first[kMaxOctaves];
    float acrossInverse[kMaxOctaves];
    uint32_t steps;
    uint8_t stepOctave[kTableSteps];
};

constexpr uint32_t kLcgA = 1664525u, kLcgC = 1013904223u;

// pcg3d's x word for a corner whose first-step terms are already applied (hash.h:40-57).
__device__ __forceinline__ uint32_t corner_from_terms(uint32_t x, uint32_t y, uint32_t z) {
    x += y * z;
    y += z * x;
    z += x * y;
    x ^= x >> 16u;
    y ^= y >> 16u;
    z ^= z >> 16u;
    return x + y * z;
}

// The gradient of the lattice corner (ix, iy) of an octave.
__device__ __forceinline__ noise::Gradient corner_gradient(uint32_t ix, uint32_t iy,
                                                           uint32_t seedTerm) {
    return noise::gradient_of(
        corner_from_terms(ix * kLcgA + kLcgC, iy * kLcgA + kLcgC, seedTerm));
}

// PerlinNoise2 (perlin.h:72-98) at fraction (fx, fy) of a cell, its corners' gradients given.
__device__ __forceinline__ float perlin_in(const noise::Gradient (&g)[4], float fx, float fy) {
    const float n00 = noise::gradient_dot(g[0], fx, fy);
    const float n10 = noise::gradient_dot(g[1], fx - 1.0f, fy);
    const float n01 = noise::gradient_dot(g[2], fx, fy - 1.0f);
    const float n11 = noise::gradient_dot(g[3], fx - 1.0f, fy - 1.0f);
    const float u = noise::fade(fx);
    const float v = noise::fade(fy);
    return 1.41421356237309505f *
           noise::lerp(v, noise::lerp(u, n00, n10), noise::lerp(u, n01, n11));
}

// The fBm source: octave-outer over kRows cells of a column. It is bound by issuing instructions
// and by the float pipe, so:
//   - each octave of a block whose lattice points are few (its tile spans a few lattice cells)
//     reads their gradients from a table the block hashes once;
//   - the rows of such an octave run two to an instruction (Pair), 54 for two cells, and with no
//     branch between the pairs: an octave whose rows share a cell in every lane loads its
//     gradients once, any other loads them for every pair (cheaper than asking which changed:
//     293 against 303 us).
// 4097^2 cells of 8 octaves: 626 us when each thread hashed and selected its corners' gradients
// (159 instructions a cell and octave), 338 with the tables and one row to an instruction, 293
// now; the float operations alone take 200 us at the pipe's rate. Octaves too fine for the table
// hash their corners per cell. Grids are not rotated (the entry points refuse others), so a
// cell's x depends on its column alone and its y on its row alone.
template <int kRows>
__global__ void __launch_bounds__(kBlockX* kBlockY, 3)
    fbm_kernel(const Octaves oct, const Grid grid, const Positions at, const bool fill,
               const float elevation, const NoData nodata, float* __restrict__ heights) {
    static_assert(kRows % 2 == 0, "rows run in pairs");
    __shared__ float table[3 * kTablePoints];
    __shared__ uint32_t bases[kMaxOctaves];
    const uint32_t tile0 = blockIdx.y * kBlockY * kRows;
    if (oct.tabled != 0u) {
        // The tile's corner cells bound its lattice positions: every other cell's lies between
        // them but for rounding (below 1/8 of a lattice cell where octaves are tabled), which the
        // margin of one point on each side covers.
        const uint32_t c0 = blockIdx.x * kBlockX, c1 = min(c0 + kBlockX, grid.width) - 1u;
        const uint32_t r0 = tile0, r1 = min(r0 + kBlockY * kRows, grid.height) - 1u;
        float cx[4], cy[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t c = k & 1 ? c1 : c0, r = k & 2 ? r1 : r0;
            cx[k] = k > 1 ? cx[k & 1] : column_x(grid, at, c, r);
            cy[k] = k & 1 ? cy[k & 2] : row_y(grid, at, c, r);
        }
        for (uint32_t step = threadIdx.y; step < oct.steps; step += kBlockY) {
            const uint32_t o = oct.stepOctave[step];
            const uint32_t across = oct.across[o], first = oct.first[o];
            const uint32_t p = step * 32u - first + threadIdx.x;
            const float tc = oct.tc[o], ts = oct.ts[o], f = oct.frequency[o];
            float qx = INFINITY, qy = INFINITY;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                qx = fminf(qx, (cx[k] * tc - cy[k] * ts) * f + oct.ox[o]);
                qy = fminf(qy, (cx[k] * ts + cy[k] * tc) * f + oct.oy[o]);
            }
            const uint32_t ix0 = uint32_t(__float2int_rd(qx) - 1);
            const uint32_t iy0 = uint32_t(__float2int_rd(qy) - 1);
            if (p == 0u) {
                bases[o] = first - (iy0 + kFloorBits) * across - (ix0 + kFloorBits);
            }
            if (p < oct.points[o]) {
                // p / across: both below 2^11, so the half keeps the float quotient off integers.
                const uint32_t j = uint32_t((float(p) + 0.5f) * oct.acrossInverse[o]);
                const noise::Gradient g =
                    corner_gradient(ix0 + p - j * across, iy0 + j, oct.seedTerm[o]);
                float* entry = table + step * 32u + threadIdx.x;
                entry[0] = g.x;
                entry[kTablePoints] = g.y;
                entry[2 * kTablePoints] = g.s;
            }
        }
        __syncthreads();
    }
    const uint32_t row0 = tile0 + threadIdx.y * kRows;
    if (row0 >= grid.height) {
        return;
    }
    // Lanes past the last column evaluate it with the others and write nothing.
    const bool inside = blockIdx.x * kBlockX + threadIdx.x < grid.width;
    const uint32_t col = inside ? blockIdx.x * kBlockX + threadIdx.x : grid.width - 1u;
    const int rows = min(kRows, int(grid.height - row0));
    constexpr int kPairs = kRows / 2;
    const float x0 = column_x(grid, at, col, row0);
    const Pair x = both(x0);
    Pair ys[kPairs], sum[kPairs];
#pragma unroll
    for (int k = 0; k < kPairs; ++k) {
        const uint32_t a = row0 + min(2 * k, rows - 1), b = row0 + min(2 * k + 1, rows - 1);
        ys[k] = pair_of(row_y(grid, at, col, a), row_y(grid, at, col, b));
        sum[k] = both(0.0f);
    }
    const Arithmetic on(oct.one);
    for (int o = 0; o < oct.count; ++o) {
        const float tc = oct.tc[o], ts = oct.ts[o], f = oct.frequency[o];
        const float ox = oct.ox[o], oy = oct.oy[o], w = oct.weight[o];
        if ((oct.tabled >> o) & 1u) {
            const uint32_t base = bases[o], across = oct.across[o];
            Pair fx[kPairs], fy[kPairs];
            uint32_t cells[kPairs][2];  // each row's cell's place in the table
            bool same = true;
#pragma unroll
            for (int k = 0; k < kPairs; ++k) {
                // Fractal2's rotation and lattice position, split as split2 does.
                const Pair y = ys[k];
                const Pair qx = on.add(
                    mul2(on.sub(mul2(x, both(tc)), mul2(y, both(ts))), both(f)), both(ox));
                const Pair qy = on.add(
                    mul2(on.add(mul2(x, both(ts)), mul2(y, both(tc))), both(f)), both(oy));
                const Pair lx = on.add_down(qx, both(kFloorShift));
                const Pair ly = on.add_down(qy, both(kFloorShift));
                fx[k] = on.sub(qx, on.sub(lx, both(kFloorShift)));
                fy[k] = on.sub(qy, on.sub(ly, both(kFloorShift)));
                float ax, bx, ay, by;
                halves(lx, ax, bx);
                halves(ly, ay, by);
                cells[k][0] = base + __float_as_uint(ay) * across + __float_as_uint(ax);
                cells[k][1] = base + __float_as_uint(by) * across + __float_as_uint(bx);
                same = same && cells[k][0] == cells[0][0] && cells[k][1] == cells[0][0];
            }
            CellPair g = cell_pair<kTablePoints>(table, cells[0][0], cells[0][1], across);
            auto add = [&](int k) {
                const Pair gx = on.sub(fx[k], both(1.0f)), gy = on.sub(fy[k], both(1.0f));
                const Pair n00 = gradient_dot2(g.g00, fx[k], fy[k]);
                const Pair n10 = gradient_dot2(g.g10, gx, fy[k]);
                const Pair n01 = gradient_dot2(g.g01, fx[k], gy);
                const Pair n11 = gradient_dot2(g.g11, gx, gy);
                const Pair u = on.fade(fx[k]), v = on.fade(fy[k]);
                const Pair n = mul2(both(1.41421356237309505f),
                                    on.lerp(v, on.lerp(u, n00, n10), on.lerp(u, n01, n11)));
                sum[k] = on.add(mul2(both(w), n), sum[k]);
            };
            if (__all_sync(0xffffffffu, same)) {
                // Every lane's rows in one cell (broad octaves): no branch between the pairs.
#pragma unroll
                for (int k = 0; k < kPairs; ++k) {
                    add(k);
                }
                continue;
            }
#pragma unroll
            for (int k = 0; k < kPairs; ++k) {
                if (k > 0) {
                    g = cell_pair<kTablePoints>(table, cells[k][0], cells[k][1], across);
                }
                add(k);
            }
            continue;
        }
        const uint32_t sz = oct.seedTerm[o];
        noise::Gradient g[4];
        int32_t cx = 0, cy = 0;
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            float ya, yb, sa, sb;
            halves(ys[r / 2], ya, yb);
            halves(sum[r / 2], sa, sb);
            const float y = r & 1 ? yb : ya;
            const float rx = x0 * tc - y * ts;
            const float ry = x0 * ts + y * tc;
            const noise::Cell2 c = noise::split2(rx * f + ox, ry * f + oy);
            if (r == 0 || c.ix != cx || c.iy != cy) {
                cx = c.ix;
                cy = c.iy;
                const uint32_t x0 = uint32_t(c.ix), y0 = uint32_t(c.iy);
                g[0] = corner_gradient(x0, y0, sz);
                g[1] = corner_gradient(x0 + 1u, y0, sz);
                g[2] = corner_gradient(x0, y0 + 1u, sz);
                g[3] = corner_gradient(x0 + 1u, y0 + 1u, sz);
            }
            const float add = w * perlin_in(g, c.fx, c.fy);
            sum[r / 2] = r & 1 ? pair_of(sa, sb + add) : pair_of(sa + add, sb);
        }
    }
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
        if (r >= rows || !inside) {
            break;
        }
        const size_t i = size_t(row0 + r) * grid.width + col;
        float base = elevation;
        if (!fill) {
            base = heights[i];
            if (is_nodata(nodata, base)) {
                continue;
            }
        }
        // EvaluateFractals of one enabled fractal: amplitude * (1 * sum / total).
        float sa, sb;
        halves(sum[r / 2], sa, sb);
        heights[i] = base + oct.amplitude * (1.0f * (r & 1 ? sb : sa) / oct.total);
    }
}

// Which octaves a block of kBlockX columns by `tileRows` rows reads from its table, and where:
// those whose lattice box over the tile fits what is left of the table, coarsest first, with
// every lattice position of the grid below 2^18 (so that the float positions are good to 1/8 and
// kFloorShift is exact). Positions from arrays are not bounded by a tile's corners: none.
void place_tables(Octaves& oct, const Grid& g, const Positions& at, uint32_t tileRows) {
    oct.tabled = 0u;
    oct.steps = 0u;
    if (at.xs != nullptr || at.ys != nullptr) {
        return;
    }
    const double reach = lattice_reach(g, at);
    const double spanC = double(kBlockX - 1), spanR = double(tileRows - 1);
    const double wide = spanC * std::fabs(g.pixelWidth) + spanR * std::fabs(g.rowRotation);
    const double high = spanC * std::fabs(g.colRotation) + spanR * std::fabs(g.pixelHeight);
    for (int o = 0; o < oct.count; ++o) {
        const double f = std::fabs(double(oct.frequency[o]));
        const double tc = std::fabs(double(oct.tc[o])), ts = std::fabs(double(oct.ts[o]));
        if (!lattice_tabled(reach, oct.frequency[o])) {
            continue;
        }
        // The box's cells, their far corners, the margin on each side and one for rounding.
        const double across = std::floor((wide * tc + high * ts) * f) + 5.0;
        const double down = std::floor((wide * ts + high * tc) * f) + 5.0;
        if (!(across * down <= double((kTableSteps - oct.steps) * 32u))) {
            continue;
        }
        oct.tabled |= 1u << o;
        oct.first[o] = uint16_t(oct.steps * 32u);
        oct.across[o] = uint16_t(across);
        oct.acrossInverse[o] = 1.0f / float(across);
        oct.points[o] = uint16_t(across * down);
        for (uint32_t p = 0; p < oct.points[o]; p += 32u) {
            oct.stepOctave[oct.steps++] = uint8_t(o);
        }
    }
}

template <int kRows>
void launch_fbm(Octaves& oct, const Grid& grid, const Positions& at, bool fill, float elevation,
                NoData nodata, float* heights, cudaStream_t stream) {
    const uint32_t rowsPerBlock = kBlockY * kRows;
    place_tables(oct, grid, at, rowsPerBlock);
    const dim3 block(kBlockX, kBlockY);
    const dim3 blocks((grid.width + kBlockX - 1) / kBlockX,
                      (grid.height + rowsPerBlock - 1) / rowsPerBlock);
    fbm_kernel<kRows><<<blocks, block, 0, stream>>>(oct, grid, at, fill, elevation, nodata,
                                                    heights);
}

// Any stack of fractals (bases, types, blends, warps). Every octave's key, frequency and turn are
// made once on the host by the float recurrences the reference runs per cell, so a cell's
// operations are the reference's; each thread takes kStackRows cells of a column, octave-outer,
// so the choice of basis and type is made once for them and a lattice cell's hashes serve the
// rows that stay in it. It is bound by issuing instructions (82 % of cycles): 1025^2 cells of four
// fractals (warped ridges, simplex, value, Worley) took 255 us cell by cell, with each cell
// remaking the octaves' keys and hashing 25 Worley cells, and take 171.
constexpr int kStackRows = 4;
constexpr int kWarpOctaves = 4;   // DomainWarp (fractals.h:151)
constexpr int kStackOctaves = kMaxFractals * (kMaxOctaves + 2 * kWarpOctaves);
struct StackOctave {
    uint32_t seed;
    float ox, oy, frequency, tc, ts;
};
struct StackLayout {
    uint32_t count;  // enabled fractals, in order
    struct {
        uint32_t basis, type, blend;
        int octaves;
        uint16_t first, warp;  // its octaves; its warp's 2 kWarpOctaves
        float amplitude, gain, offset, warpAmplitude;
    } fractals[kMaxFractals];
    StackOctave octaves[kStackOctaves];
};

// The corners' gradients or values of the lattice cell the last row was in.
struct LatticeCell {
    int32_t ix, iy;
    bool held;
    float a[4], b[4], c[4];  // gradients (x, y, s), or values in a
};

__device__ __forceinline__ float perlin_held(LatticeCell& m, float x, float y, uint32_t seed) {
    const noise::Cell2 c = noise::split2(x, y);
    if (!m.held || c.ix != m.ix || c.iy != m.iy) {
        m.held = true;
        m.ix = c.ix;
        m.iy = c.iy;
        const uint32_t sz = seed * kLcgA + kLcgC;
#pragma unroll
        for (uint32_t k = 0; k < 4u; ++k) {
            const noise::Gradient g = corner_gradient(uint32_t(c.ix) + (k & 1u),
                                                      uint32_t(c.iy) + (k >> 1u), sz);
            m.a[k] = g.x;
            m.b[k] = g.y;
            m.c[k] = g.s;
        }
    }
    const noise::Gradient g[4] = {{m.a[0], m.b[0], m.c[0]},
                                  {m.a[1], m.b[1], m.c[1]},
                                  {m.a[2], m.b[2], m.c[2]},
                                  {m.a[3], m.b[3], m.c[3]}};
    return perlin_in(g, c.fx, c.fy);
}

__device__ __forceinline__ float value_held(LatticeCell& m, float x, float y, uint32_t seed) {
    const noise::Cell2 c = noise::split2(x, y);
    if (!m.held || c.ix != m.ix || c.iy != m.iy) {
        m.held = true;
        m.ix = c.ix;
        m.iy = c.iy;
#pragma unroll
        for (uint32_t k = 0; k < 4u; ++k) {
            m.a[k] = noise::lattice_value(uint32_t(c.ix) + (k & 1u), uint32_t(c.iy) + (k >> 1u),
                                          seed);
        }
    }
    const float u = noise::fade(c.fx), v = noise::fade(c.fy);
    return noise::lerp(v, noise::lerp(u, m.a[0], m.a[1]), noise::lerp(u, m.a[2], m.a[3]));
}

// Worley distances mapped to [-1, 1], or the nearest point's value (basis2's cases; without kSecond
// none that reads the second nearest).
template <bool kSecond>
__device__ __forceinline__ float worley_basis(uint32_t basis, float x, float y, uint32_t seed) {
    const float kInvSqrt2 = 0.707106781186547524f;
    const float kInvSqrt5 = 0.447213595499957939f;
    const bool second =
        kSecond && (basis == kBasisWorleyF2 || basis == kBasisWorleyF2MinusF1);
    const noise::WorleyD w = noise::worley2(x, y, seed, second);
    if (basis == kBasisVoronoi) {
        return w.value;
    }
    const float d = !second                   ? w.f1 * kInvSqrt2
                    : basis == kBasisWorleyF2 ? w.f2 * kInvSqrt5
                                              : (w.f2 - w.f1) * kInvSqrt5;
    return 2.0f * noise::smin(d, 1.0f) - 1.0f;
}

// One octave of a basis at the rows' positions (Fractal2's turn and lattice position).
template <bool kSecond>
__device__ __forceinline__ void basis_rows(const StackOctave& o, uint32_t basis,
                                           const float (&x)[kStackRows],
                                           const float (&y)[kStackRows], float (&n)[kStackRows]) {
    float px[kStackRows], py[kStackRows];
#pragma unroll
    for (int r = 0; r < kStackRows; ++r) {
        const float rx = x[r] * o.tc - y[r] * o.ts;
        const float ry = x[r] * o.ts + y[r] * o.tc;
        px[r] = rx * o.frequency + o.ox;
        py[r] = ry * o.frequency + o.oy;
    }
    LatticeCell held;
    held.held = false;
    if (basis == kBasisPerlin) {
#pragma unroll
        for (int r = 0; r < kStackRows; ++r) {
            n[r] = perlin_held(held, px[r], py[r], o.seed);
        }
    } else if (basis == kBasisValue) {
#pragma unroll
        for (int r = 0; r < kStackRows; ++r) {
            n[r] = value_held(held, px[r], py[r], o.seed);
        }
    } else {
        // The rows turn through the first place, so they are indexed without a local array and
        // the longer bases stand in the code once (the kernel waits for instructions otherwise).
#pragma unroll 1
        for (int r = 0; r < kStackRows; ++r) {
            const float v = basis == kBasisSimplex ? noise::simplex2(px[0], py[0], o.seed)
                                                   : worley_basis<kSecond>(basis, px[0], py[0],
                                                                         o.seed);
#pragma unroll
            for (int k = 0; k < kStackRows - 1; ++k) {
                px[k] = px[k + 1];
                py[k] = py[k + 1];
                n[k] = n[k + 1];
            }
            n[kStackRows - 1] = v;
        }
    }
}

template <bool kSecond>
__global__ void __launch_bounds__(kBlockX* kBlockY, 3)
    noise_kernel(const __grid_constant__ StackLayout stack, const Grid grid, const Positions at,
                 const bool fill, const float elevation, const NoData nodata,
                 float* __restrict__ heights) {
    const uint32_t col = blockIdx.x * kBlockX + threadIdx.x;
    const uint32_t row0 = (blockIdx.y * kBlockY + threadIdx.y) * kStackRows;
    if (col >= grid.width || row0 >= grid.height) {
        return;
    }
    const int rows = min(kStackRows, int(grid.height - row0));
    float x[kStackRows], y[kStackRows], height[kStackRows];
#pragma unroll
    for (int r = 0; r < kStackRows; ++r) {
        const uint32_t row = row0 + min(r, rows - 1);
        x[r] = column_x(grid, at, col, row);
        y[r] = row_y(grid, at, col, row);
        height[r] = 0.0f;
    }
#pragma unroll 1
    for (uint32_t i = 0; i < stack.count; ++i) {
        const auto& f = stack.fractals[i];
        float px[kStackRows], py[kStackRows];
#pragma unroll
        for (int r = 0; r < kStackRows; ++r) {
            px[r] = x[r];
            py[r] = y[r];
        }
        // The warp's displacements along x and y (DomainWarp, fractals.h:151: Perlin fBm of four
        // octaves at the unwarped positions), then the fractal at the warped ones.
#pragma unroll 1
        for (int pass = f.warpAmplitude > 0.0f ? 0 : 2; pass < 3; ++pass) {
            const bool warps = pass < 2;
            const uint32_t first = warps ? f.warp + uint32_t(pass * kWarpOctaves) : f.first;
            const int octaves = warps ? kWarpOctaves : f.octaves;
            const uint32_t basis = warps ? uint32_t(kBasisPerlin) : f.basis;
            const uint32_t type = warps ? uint32_t(kTypeFbm) : f.type;
            const float gain = warps ? 0.5f : f.gain, offset = warps ? 1.0f : f.offset;
            noise::Sums s[kStackRows];
            float qx[kStackRows], qy[kStackRows];
#pragma unroll
            for (int r = 0; r < kStackRows; ++r) {
                s[r] = noise::sums_start();
                qx[r] = warps ? x[r] : px[r];
                qy[r] = warps ? y[r] : py[r];
            }
#pragma unroll 1
            for (int o = 0; o < octaves; ++o) {
                float n[kStackRows];
                basis_rows<kSecond>(stack.octaves[first + o], basis, qx, qy, n);
#pragma unroll
                for (int r = 0; r < kStackRows; ++r) {
                    s[r] = noise::add_octave(s[r], type, gain, offset, o, n[r]);
                }
            }
#pragma unroll
            for (int r = 0; r < kStackRows; ++r) {
                const float value =
                    noise::finish(s[r], type, warps ? f.warpAmplitude : 1.0f, offset);
                px[r] = pass == 0 ? x[r] + value : px[r];
                py[r] = pass == 1 ? y[r] + value : py[r];
                if (!warps) {
                    height[r] = i == 0u ? f.amplitude * value
                                        : noise::blend_stack(height[r], value, f.amplitude,
                                                             f.blend);
                }
            }
        }
    }
#pragma unroll
    for (int r = 0; r < kStackRows; ++r) {
        if (r >= rows) {
            break;
        }
        const size_t i = size_t(row0 + r) * grid.width + col;
        float base = elevation;
        if (!fill) {
            base = heights[i];
            if (is_nodata(nodata, base)) {
                continue;
            }
        }
        heights[i] = base + height[r];
    }
}

// pcg3d on the host (hash.h:40).
void host_pcg3d(uint32_t (&v)[3]) {
    for (uint32_t& w : v) {
        w = w * kLcgA + kLcgC;
    }
    v[0] += v[1] * v[2];
    v[1] += v[2] * v[0];
    v[2] += v[0] * v[1];
    for (uint32_t& w : v) {
        w ^= w >> 16u;
    }
    v[0] += v[1] * v[2];
    v[1] += v[2] * v[0];
    v[2] += v[0] * v[1];
}

float host_unit(uint32_t h) {
    return float(h >> 8u) * 0x1p-24f;
}

uint32_t host_pcg(uint32_t v) {  // hash.h:33
    const uint32_t state = v * 747796405u + 2891336453u;
    const uint32_t word = ((state >> ((state >> 28u) + 4u)) ^ state) * 277803737u;
    return (word >> 22u) ^ word;
}

// The octaves of a fractal, in Fractal2's order of float operations (fractal.h:219-240); this unit
// is built without contraction, so they round as on the reference's CPU.
void host_octaves(StackOctave* out, uint32_t seed, float wavelength, float lacunarity,
                  int octaves) {
    float frequency = 1.0f / wavelength;
    float tc = 1.0f, ts = 0.0f;
    for (int o = 0; o < octaves; ++o) {
        uint32_t v[3] = {seed, uint32_t(o), 0u};
        host_pcg3d(v);
        out[o] = StackOctave{v[0], host_unit(v[1]), host_unit(v[2]), frequency, tc, ts};
        frequency *= lacunarity;
        const float nc = tc * TGB_TURN_COS - ts * TGB_TURN_SIN;
        ts = ts * TGB_TURN_COS + tc * TGB_TURN_SIN;
        tc = nc;
    }
}

bool stack_layout(const FractalStack& stack, StackLayout& out) {
    out.count = 0;
    int used = 0;
    for (uint32_t i = 0; i < stack.count && i < kMaxFractals; ++i) {
        const Fractal& f = stack.fractals[i];
        if (!f.enabled) {
            continue;
        }
        if (f.octaves > kMaxOctaves) {
            return false;  // the entry points refuse it
        }
        auto& l = out.fractals[out.count++];
        l.basis = f.basis;
        l.type = f.type;
        l.blend = f.blend;
        l.octaves = std::max(f.octaves, 0);
        l.amplitude = f.amplitude;
        l.gain = f.gain;
        l.offset = f.offset;
        l.warpAmplitude = f.warpAmplitude;
        l.first = uint16_t(used);
        host_octaves(out.octaves + used, f.seed, f.wavelength, f.lacunarity, l.octaves);
        used += l.octaves;
        l.warp = uint16_t(used);
        if (f.warpAmplitude > 0.0f) {
            const uint32_t seed = host_pcg(f.seed ^ TGB_WARP_SALT);
            host_octaves(out.octaves + used, seed, f.warpWavelength, 2.0f, kWarpOctaves);
            host_octaves(out.octaves + used + kWarpOctaves, host_pcg(seed), f.warpWavelength,
                         2.0f, kWarpOctaves);
            used += 2 * kWarpOctaves;
        }
    }
    return true;
}

// Per point: PcgHash(i), Pcg3dHash((x bits, y bits, seed)), then Perlin, simplex, value, Worley
// F1/F2/value, and Perlin fBm / ridged / billow / hybrid (seed `seed`) at (x, y).
__global__ void noise_probe_kernel(const float* __restrict__ xy, uint32_t n, uint32_t seed,
                                   uint32_t* __restrict__ hashes, float* __restrict__ values) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) {
        return;
    }
    const float x = xy[2 * i], y = xy[2 * i + 1];
    hashes[4 * i] = noise::pcg(i);
    const noise::U3 h = noise::pcg3d(noise::U3{__float_as_uint(x), __float_as_uint(y), seed});
    hashes[4 * i + 1] = h.x;
    hashes[4 * i + 2] = h.y;
    hashes[4 * i + 3] = h.z;
    float* v = values + 12 * i;
    v[0] = noise::perlin2(x, y, seed);
    v[1] = noise::simplex2(x, y, seed);
    v[2] = noise::value2(x, y, seed);
    const noise::WorleyD w = noise::worley2(x, y, seed, true);
    v[3] = w.f1;
    v[4] = w.f2;
    v[5] = w.value;
    FractalParams p{seed, 1000.0f, 100.0f, 8, 2.0f, 0.5f, kBasisPerlin, kTypeFbm, 1.0f};
    v[6] = noise::fractal2(x, y, p);
    p.type = kTypeRidged;
    v[7] = noise::fractal2(x, y, p);
    p.type = kTypeBillow;
    v[8] = noise::fractal2(x, y, p);
    p.type = kTypeHybrid;
    v[9] = noise::fractal2(x, y, p);
    v[10] = noise::perlin3(x, y, 0.5f * (x - y), seed);
    v[11] = noise::perlin_fbm3_float(x, y, 0.25f * x, seed, 3, 0.5f);
}

}  // namespace

namespace {

// Golden-angle turn about (1, 2, 3) / sqrt(14) between 3D octave lattices, in double (Fractal3,
// fractal.h:286-289).
constexpr double kTurn3d[3][3] = {
    {-0.6132711010727254, -0.293401570821183, 0.7333580809050306},
    {0.7897926788435601, -0.24097777005594262, 0.5640542870894418},
    {0.011228581128535142, 0.9251190369776896, 0.37951111497202883}};

struct BodyOctave {
    double frequency;
    uint32_t seed, key;  // pcg(seed)
    float ox, oy, oz;
};
template <int kTurns, int kBodyOctaves>
struct BodyLayout {
    uint32_t count;  // enabled fractals, in order
    struct {
        uint32_t basis, type, blend;
        int octaves;
        uint16_t first, warp;  // its octaves; its warp's 3 kWarpOctaves
        float amplitude, gain, offset, warpAmplitude;
    } fractals[kMaxFractals];
    double turn[kTurns][9];  // an octave's turn, the same for every fractal
    BodyOctave octaves[kBodyOctaves];
};
// Any stack, and one of few octaves: a launch's arguments are copied with it, and 14 KB of them and
// 32 turns made on the host took 1.5 us of a call of 17.5 (129^2 cells); with 3 KB and 16 turns they take 0.1.
using FullBody = BodyLayout<kMaxOctaves, kMaxFractals * (kMaxOctaves + 3 * kWarpOctaves)>;
using SmallBody = BodyLayout<16, 48>;

// gradient3's sixteen directions as coefficients: two of x, y, z with signs, so their sum with
// multiply-adds rounds once, as gradient3's u + v.
__device__ __forceinline__ float4 gradient3_of(uint32_t h) {
    const float su = (h & 1u) != 0u ? -1.0f : 1.0f, sv = (h & 2u) != 0u ? -1.0f : 1.0f;
    float4 g = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    (h < 8u ? g.x : g.y) = su;
    (h < 4u ? g.y : (h == 12u || h == 14u ? g.x : g.z)) = sv;
    return g;
}

// PerlinNoise3 at a cell (perlin.h:113-128; corner keys x, y, z + pcg(seed), the last term `key`)
// with its corners' directions read from a shared table: selecting them per corner kept the integer
// pipe 77 % busy.
__device__ __forceinline__ float perlin3_table(const noise::Cell3& c, uint32_t key,
                                               const float4* directions) {
    uint32_t ax[2], ay[2], az[2];
#pragma unroll
    for (uint32_t d = 0; d < 2u; ++d) {
        ax[d] = (uint32_t(c.ix) + d) * kLcgA + kLcgC;
        ay[d] = (uint32_t(c.iy) + d) * kLcgA + kLcgC;
        az[d] = (uint32_t(c.iz) + d + key) * kLcgA + kLcgC;
    }
    const float x[2] = {c.fx, c.fx - 1.0f}, y[2] = {c.fy, c.fy - 1.0f}, z[2] = {c.fz, c.fz - 1.0f};
    float k[8];
#pragma unroll
    for (uint32_t n = 0; n < 8u; ++n) {
        const uint32_t i = n & 1u, j = (n >> 1u) & 1u, m = n >> 2u;
        const float4 g = directions[corner_from_terms(ax[i], ay[j], az[m]) & 15u];
        k[n] = fmaf(g.x, x[i], fmaf(g.y, y[j], g.z * z[m]));
    }
    const float u = noise::fade(c.fx), v = noise::fade(c.fy), w = noise::fade(c.fz);
    const float near = noise::lerp(v, noise::lerp(u, k[0], k[1]), noise::lerp(u, k[2], k[3]));
    const float far = noise::lerp(v, noise::lerp(u, k[4], k[5]), noise::lerp(u, k[6], k[7]));
    return noise::sclamp(noise::lerp(w, near, far), -1.0f, 1.0f);
}

// Fractal3's octaves (fractal.h:284-316) at a point: world coordinates in double, each octave's
// lattice point split in double before narrowing.
template <typename Layout>
__device__ __forceinline__ noise::Sums body_octaves(const Layout& stack, uint32_t first,
                                                    int octaves, uint32_t basis, uint32_t type,
                                                    float gain, float offset, double x, double y,
                                                    double z, const float4* directions) {
    noise::Sums s = noise::sums_start();
#pragma unroll 1
    for (int o = 0; o < octaves; ++o) {
        const BodyOctave& k = stack.octaves[first + o];
        const double(&t)[9] = stack.turn[o];
        const double rx = t[0] * x + t[1] * y + t[2] * z;
        const double ry = t[3] * x + t[4] * y + t[5] * z;
        const double rz = t[6] * x + t[7] * y + t[8] * z;
        const noise::Cell3 c = noise::split3_precise(rx * k.frequency + double(k.ox),
                                                     ry * k.frequency + double(k.oy),
                                                     rz * k.frequency + double(k.oz));
        const float n = basis == kBasisPerlin ? perlin3_table(c, k.key, directions)
                                              : noise::basis3(basis, c, k.seed);
        s = noise::add_octave(s, type, gain, offset, o, n);
    }
    return s;
}

// A SyntheticSource on a sphere (SyntheticSource::NoiseAt with FractalStackAt on a body,
// surface_noise.cpp:14-17): each cell center's position R (cos lat cos lon, cos lat sin lon,
// sin lat) (UnitVector, surface.cpp:45), from the host's cosines and sines of each column's
// longitude and each row's latitude, then the stack in 3D. The octaves' turns, frequencies and
// keys are made once on the host, by the recurrences in double that Fractal3 runs per cell. It is
// bound by issuing instructions (84 % of cycles). 1025^2 cells, 8 octaves: 146 us when each cell
// multiplied its own matrices, 120 with the host's, 82 with the corners' directions from a table
// (calls of 81.3 us with room for seven blocks an SM, 82.5 without that bound, 83 to 85 with eight
// to ten).
template <typename Layout>
__global__ void __launch_bounds__(128, 7)
    noise_body_kernel(const __grid_constant__ Layout stack, float elevation, uint32_t width,
                      uint32_t height, const double* __restrict__ lons,
                      const double* __restrict__ lats, double radius,
                      float* __restrict__ heights) {
    __shared__ float4 directions[16];
    if (threadIdx.y == 0 && threadIdx.x < 16u) {
        directions[threadIdx.x] = gradient3_of(threadIdx.x);
    }
    __syncthreads();
    const uint32_t col = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t row = blockIdx.y * blockDim.y + threadIdx.y;
    if (col >= width || row >= height) {
        return;
    }
    const double cosLon = lons[2 * col], sinLon = lons[2 * col + 1];
    const double cosLat = lats[2 * row], sinLat = lats[2 * row + 1];
    const double x = cosLat * cosLon * radius;
    const double y = cosLat * sinLon * radius;
    const double z = sinLat * radius;
    float sum = 0.0f;
#pragma unroll 1
    for (uint32_t i = 0; i < stack.count; ++i) {
        const auto& f = stack.fractals[i];
        double px = x, py = y, pz = z;
        if (f.warpAmplitude > 0.0f) {  // DomainWarp3 (fractals.h:218-243)
            float d[3];
#pragma unroll 1
            for (int a = 0; a < 3; ++a) {
                const float v = noise::finish(
                    body_octaves(stack, f.warp + uint32_t(a * kWarpOctaves), kWarpOctaves,
                                 kBasisPerlin, kTypeFbm, 0.5f, 1.0f, x, y, z, directions),
                    kTypeFbm, f.warpAmplitude, 1.0f);
                d[0] = a == 0 ? v : d[0];
                d[1] = a == 1 ? v : d[1];
                d[2] = a == 2 ? v : d[2];
            }
            px = x + double(d[0]);
            py = y + double(d[1]);
            pz = z + double(d[2]);
        }
        const float value = noise::finish(body_octaves(stack, f.first, f.octaves, f.basis, f.type,
                                                       f.gain, f.offset, px, py, pz, directions),
                                          f.type, 1.0f, f.offset);
        sum = i == 0u ? f.amplitude * value : noise::blend_stack(sum, value, f.amplitude, f.blend);
    }
    heights[size_t(row) * width + col] = elevation + sum;
}

void host_body_octaves(BodyOctave* out, uint32_t seed, float wavelength, float lacunarity,
                       int octaves) {
    double frequency = 1.0 / double(wavelength);
    for (int o = 0; o < octaves; ++o) {
        uint32_t h[3] = {seed, uint32_t(o), 0u}, g[3] = {seed, uint32_t(o), 1u};
        host_pcg3d(h);
        host_pcg3d(g);
        out[o] = BodyOctave{frequency, h[0], host_pcg(h[0]), host_unit(h[1]), host_unit(h[2]), host_unit(g[0])};
        frequency *= double(lacunarity);
    }
}

template <int kTurns, int kBodyOctaves>
bool body_layout(const FractalStack& stack, BodyLayout<kTurns, kBodyOctaves>& out) {
    double t[9] = {1.0, 0.0, 0.0, 0.0, 1.0, 0.0, 0.0, 0.0, 1.0};
    for (int o = 0; o < kTurns; ++o) {
        double next[9];
        for (int r = 0; r < 3; ++r) {
            for (int c = 0; c < 3; ++c) {
                out.turn[o][3 * r + c] = t[3 * r + c];
                next[3 * r + c] = kTurn3d[r][0] * t[c] + kTurn3d[r][1] * t[3 + c] +
                                  kTurn3d[r][2] * t[6 + c];
            }
        }
        std::copy(next, next + 9, t);
    }
    out.count = 0;
    int used = 0;
    for (uint32_t i = 0; i < stack.count && i < kMaxFractals; ++i) {
        const Fractal& f = stack.fractals[i];
        if (!f.enabled) {
            continue;
        }
        if (f.octaves > kMaxOctaves) {
            return false;  // the entry points refuse it
        }
        auto& l = out.fractals[out.count++];
        l.basis = f.basis;
        l.type = f.type;
        l.blend = f.blend;
        l.octaves = std::max(f.octaves, 0);
        l.amplitude = f.amplitude;
        l.gain = f.gain;
        l.offset = f.offset;
        l.warpAmplitude = f.warpAmplitude;
        l.first = uint16_t(used);
        host_body_octaves(out.octaves + used, f.seed, f.wavelength, f.lacunarity, l.octaves);
        used += l.octaves;
        l.warp = uint16_t(used);
        if (f.warpAmplitude > 0.0f) {
            uint32_t seed = f.seed ^ TGB_WARP_SALT;
            for (int a = 0; a < 3; ++a) {
                seed = host_pcg(seed);
                host_body_octaves(out.octaves + used, seed, f.warpWavelength, 2.0f, kWarpOctaves);
                used += kWarpOctaves;
            }
        }
    }
    return true;
}

}  // namespace

cudaError_t launch_noise_body(const FractalStack& stack, float elevation, uint32_t width,
                              uint32_t height, const double* lons, const double* lats,
                              double radius, float* heights, cudaStream_t stream) {
    if (width == 0 || height == 0) {
        return cudaSuccess;
    }
    static_assert(sizeof(FullBody) < 16384, "a kernel argument");
    const dim3 block(32, 4);
    const dim3 grid((width + 31) / 32, (height + 3) / 4);
    int deepest = kWarpOctaves, octaves = 0;
    for (uint32_t i = 0; i < stack.count && i < kMaxFractals; ++i) {
        const Fractal& f = stack.fractals[i];
        if (f.enabled) {
            deepest = std::max(deepest, int(f.octaves));
            octaves += f.octaves + (f.warpAmplitude > 0.0f ? 3 * kWarpOctaves : 0);
        }
    }
    auto launch = [&](auto layout) {
        if (!body_layout(stack, layout)) {
            return cudaErrorInvalidValue;
        }
        noise_body_kernel<<<grid, block, 0, stream>>>(layout, elevation, width, height, lons, lats,
                                                      radius, heights);
        return cudaGetLastError();
    };
    return deepest <= 16 && octaves <= 48 ? launch(SmallBody{}) : launch(FullBody{});
}

cudaError_t launch_noise(const FractalStack& stack, const Grid& grid, const Positions& at,
                         bool fill, float elevation, NoData nodata, float* heights,
                         cudaStream_t stream) {
    if (grid.width == 0 || grid.height == 0) {
        return cudaSuccess;
    }
    // The fast path: exactly one enabled fractal, Perlin fBm, no warp.
    int enabled = 0;
    const Fractal* only = nullptr;
    for (uint32_t i = 0; i < stack.count && i < kMaxFractals; ++i) {
        if (stack.fractals[i].enabled) {
            ++enabled;
            only = &stack.fractals[i];
        }
    }
    const bool single = enabled == 1 && only->basis == kBasisPerlin && only->type == kTypeFbm &&
                        !(only->warpAmplitude > 0.0f) && only->octaves <= kMaxOctaves;
    const dim3 block(kBlockX, kBlockY);
    if (single) {
        // Fractal2's per-octave values, in its order of float operations (fractal.h:219-240);
        // this unit is built without contraction, so they round as on the reference's CPU.
        Octaves oct{};
        oct.count = only->octaves;
        oct.amplitude = only->amplitude;
        float frequency = 1.0f / only->wavelength;
        float tc = 1.0f, ts = 0.0f, weight = 1.0f, total = 0.0f;
        for (int o = 0; o < only->octaves; ++o) {
            uint32_t v[3] = {only->seed, uint32_t(o), 0u};
            host_pcg3d(v);
            oct.seedTerm[o] = v[0] * kLcgA + kLcgC;  // the octave seed's first LCG step
            oct.ox[o] = host_unit(v[1]);
            oct.oy[o] = host_unit(v[2]);
            oct.frequency[o] = frequency;
            oct.tc[o] = tc;
            oct.ts[o] = ts;
            oct.weight[o] = weight;
            total += weight;
            weight *= only->gain;
            frequency *= only->lacunarity;
            const float nc = tc * TGB_TURN_COS - ts * TGB_TURN_SIN;
            ts = ts * TGB_TURN_COS + tc * TGB_TURN_SIN;
            tc = nc;
        }
        oct.total = total;
        oct.one = 1.0f;
        // Rows a thread takes: 8 amortize a block's tables best, once there are enough blocks; a
        // small grid's octaves run in parallel over its cells instead of in series over a few
        // blocks (257^2: the kernel took 17 us with 8 rows; with 2 the whole call takes 12), and
        // octaves that are hashed per cell gain nothing from more rows. So 8 rows from two and a
        // half blocks of them an SM on where at least half of the octaves are tabled, else from
        // eight. Us a call with 8 and with 2: 8 octaves, all tabled, 769^2 21.6 and 19.8, 833^2 21.6
        // and 21.8, 865^2 21.6 and 23.8, 1537^2 48.4 and 60.7; 24 octaves, most of them hashed,
        // 1281^2 170 and 163, 1537^2 229 and 227.
        const size_t columns = (grid.width + kBlockX - 1) / kBlockX;
        const size_t lines = (grid.height + kBlockY - 1) / kBlockY;
        const size_t most = columns * lines / 8;  // blocks of 8 rows a thread
        bool eight = most >= 8 * size_t(kSms);
        if (!eight && 2 * most >= 5 * size_t(kSms)) {
            place_tables(oct, grid, at, kBlockY * 8);
            int tabled = 0;
            for (uint32_t bits = oct.tabled; bits != 0u; bits &= bits - 1u) {
                ++tabled;
            }
            eight = 2 * tabled >= oct.count;
        }
        if (eight) {
            launch_fbm<8>(oct, grid, at, fill, elevation, nodata, heights, stream);
        } else {
            launch_fbm<2>(oct, grid, at, fill, elevation, nodata, heights, stream);
        }
        return cudaGetLastError();
    }
    static_assert(sizeof(StackLayout) < 16384, "a kernel argument");
    StackLayout layout;
    if (!stack_layout(stack, layout)) {
        return cudaErrorInvalidValue;
    }
    const uint32_t rowsPerBlock = kBlockY * kStackRows;
    const dim3 blocks((grid.width + kBlockX - 1) / kBlockX,
                      (grid.height + rowsPerBlock - 1) / rowsPerBlock);
    // A kernel that holds the search for a second nearest point, which no other basis reads, costs a
    // stack of other bases 2 % (1025^2 cells of warped ridges, simplex, value and Worley F1: 182 us
    // with it, 174 without).
    bool second = false;
    for (uint32_t i = 0; i < layout.count; ++i) {
        const uint32_t basis = layout.fractals[i].basis;
        second = second || basis == kBasisWorleyF2 || basis == kBasisWorleyF2MinusF1;
    }
    const auto kernel = second ? noise_kernel<true> : noise_kernel<false>;
    kernel<<<blocks, block, 0, stream>>>(layout, grid, at, fill, elevation, nodata, heights);
    return cudaGetLastError();
}

cudaError_t launch_noise_probe(const float* xy, uint32_t n, uint32_t seed, uint32_t* hashes,
                               float* values, cudaStream_t stream) {
    if (n == 0) {
        return cudaSuccess;
    }
    noise_probe_kernel<<<(n + 127) / 128, 128, 0, stream>>>(xy, n, seed, hashes, values);
    return cudaGetLastError();
}

}  // namespace tgb
