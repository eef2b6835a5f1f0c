// Boulder relief baking (BoulderLayer::ApplySamples with dome relief,
// src/layers/boulders/boulder_relief.cpp:426-439): each cell of each boulder's box gets
// max(height, base + weight * dome), base being the cell's height before the layer
// (DrawFeatures, include/terraingen/sources/sample_block.h:107-116) and the dome averaged over a
// sample width (DomeHeight, boulder_relief.cpp:44-57), in double as the reference computes it.
//
// Max-compositing is order-free: rounding to float is monotonic, so the result is
// float(max(height, max over boulders of base + weight * dome)) whatever order boulders come in,
// which lets them be binned by atomics. Launch structure as crater shaping (craters.cu): count,
// scan, scatter into kBinCells-square bins, then one CTA per bin stages its entries in shared
// memory by TMA bulk copies and each thread bakes 4 cells. A boulder touches the cells of its
// box's pixel window (ForEachFeatureCell, include/terraingen/raster/cell_loops.h:129-152).
#include "binning.cuh"
#include "kernels.h"

namespace tgb {
namespace {

constexpr int kThreads = 256;
constexpr int kCellsPerThread = 4;
constexpr uint32_t kChunk = 96;  // 64-byte entries per staged chunk (6 KB)

using namespace binning;

__global__ void boulder_count_kernel(const BoulderRecord* __restrict__ boulders, uint32_t n,
                                     const Grid grid, double width, BoulderBins bins) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) {
        return;
    }
    const BoulderRecord b = boulders[i];
    // ReliefBox on a plane (boulder_relief.cpp:24): reach 0.5 (diameter + width).
    const double reach = 0.5 * (b.diameter + width);
    int c0, c1, r0, r1;
    window_of(grid, b.x - reach, b.y - reach, b.x + reach, b.y + reach, c0, c1, r0, r1);
    const bool drawn = c0 < c1 && r0 < r1 && b.weight > 0.0;
    bins.windows[i] = drawn ? make_int4(c0, c1, r0, r1) : make_int4(1, 0, 1, 0);
    if (!drawn) {
        return;
    }
    const uint32_t bx0 = uint32_t(c0) / kBinCells, bx1 = uint32_t(c1 - 1) / kBinCells;
    const uint32_t by0 = uint32_t(r0) / kBinCells, by1 = uint32_t(r1 - 1) / kBinCells;
    for (uint32_t by = by0; by <= by1; ++by) {
        for (uint32_t bx = bx0; bx <= bx1; ++bx) {
            atomicAdd(bins.counts + by * bins.binsX + bx, 1u);
        }
    }
}

__global__ void boulder_scatter_kernel(const BoulderRecord* __restrict__ boulders, uint32_t n,
                                       BoulderBins bins) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !boulder_bins_usable(bins)) {
        return;
    }
    const int4 w = bins.windows[i];
    if (w.x >= w.y) {
        return;
    }
    const BoulderRecord b = boulders[i];
    BoulderEntry e;
    e.x = b.x;
    e.y = b.y;
    e.radius = 0.5 * b.diameter;
    e.exposed = b.exposedHeight;
    e.weight = b.weight;
    e.c0 = w.x;
    e.c1 = w.y;
    e.r0 = w.z;
    e.r1 = w.w;
    const uint32_t bx0 = uint32_t(w.x) / kBinCells, bx1 = uint32_t(w.y - 1) / kBinCells;
    const uint32_t by0 = uint32_t(w.z) / kBinCells, by1 = uint32_t(w.w - 1) / kBinCells;
    for (uint32_t by = by0; by <= by1; ++by) {
        for (uint32_t bx = bx0; bx <= bx1; ++bx) {
            const uint32_t bin = by * bins.binsX + bx;
            const uint32_t slot = bins.counts[bin] + atomicAdd(bins.cursor + bin, 1u);
            if (slot < bins.capacity) {
                bins.entries[slot] = e;
            }
        }
    }
}

// A double as a signed integer of the same order (and back), for a maximum by integer atomics.
__device__ __forceinline__ long long ordered(double v) {
    const long long b = __double_as_longlong(v);
    return b >= 0 ? b : b ^ 0x7fffffffffffffffll;
}
__device__ __forceinline__ double unordered(long long k) {
    return __longlong_as_double(k >= 0 ? k : k ^ 0x7fffffffffffffffll);
}

// A staged boulder's cells of a bin: columns [c0, c0 + wide) by rows from r0.
struct BakeBox {
    uint16_t c0, r0, wide, cells;
    float inverse;  // 1 / wide
};

constexpr uint32_t kStarts = 128;  // the power of two the search for a chunk's boulder spans

// The bake is bound by latency: a bin holds a few boulders of a few cells, and a dome's square
// root, arcsines and quotients in double take about a thousand cycles in series. The cells of all
// staged boulders' windows are therefore numbered in one sequence (a scan of the windows' sizes)
// and taken by the block's threads side by side, each drawing its dome onto the cell by an integer
// maximum in shared memory; going through the boulders in turn, four cells a thread, took 176 us on
// 4097^2 cells with 17,000 drawn boulders, and takes 97. Only cells that a boulder raised are
// written. Four CTAs per SM (64 registers a thread).
__global__ void __launch_bounds__(kThreads, 4)
    boulder_bake_kernel(const Grid grid, const double width, const NoData nodata,
                        const BoulderBins bins, float* __restrict__ heights,
                        uint32_t* __restrict__ flags, const uint32_t polls) {
    __shared__ __align__(128) BoulderEntry stage[2][kChunk];
    __shared__ __align__(8) uint64_t bars[2];
    __shared__ long long best[kBinCells * kBinCells];
    __shared__ float bases[kBinCells * kBinCells];
    __shared__ uint32_t liveRows[kBinCells];
    __shared__ BakeBox boxes[kChunk];
    __shared__ uint32_t starts[kStarts + 1];  // past the chunk: its total
    static_assert(kChunk % 32u == 0u && kChunk <= kStarts && kBinCells == 32 && kThreads == 256,
                  "the scan's shape");
    const uint32_t bin = bins.firstBin + blockIdx.x;
    if (!boulder_bins_usable(bins)) {
        // The entries were not scattered: nothing is baked, the host grows them and runs again.
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            atomicOr(flags, 4u);
        }
        return;
    }
    const uint32_t first = bins.counts[bin];
    const uint32_t count = bins.counts[bin + 1] - first;
    if (count == 0u) {
        return;
    }
    const uint32_t binX = bin % bins.binsX, binY = bin / bins.binsX;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t chunks = (count + kChunk - 1) / kChunk;
    auto issue = [&](uint32_t c) {
        const uint32_t s = c & 1u;
        const uint32_t bytes = min(kChunk, count - c * kChunk) * uint32_t(sizeof(BoulderEntry));
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_expect_tx(&bars[s], bytes);
        bulk_copy_g2s(&stage[s][0], bins.entries + first + c * kChunk, bytes, &bars[s]);
    };
    // Thread 0 starts the entry fetch before the cells' base heights are loaded, so the two
    // memory latencies overlap; the barrier after the loads publishes the mbarrier init.
    if (tid == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        issue(0);
        if (chunks > 1) {
            issue(1);
        }
    }
    const uint32_t row0 = binY * kBinCells, col0 = binX * kBinCells;
    const uint32_t myRow = warp * 4u + lane / 8u, myCol = (lane % 8u) * kCellsPerThread;
    const uint32_t cell0 = myRow * kBinCells + myCol;
    float* const mine = heights + size_t(row0 + myRow) * grid.width + col0 + myCol;
    float base[kCellsPerThread];
    uint32_t live = 0;
#pragma unroll
    for (int j = 0; j < kCellsPerThread; ++j) {
        base[j] = 0.0f;
        if (row0 + myRow < grid.height && col0 + myCol + j < grid.width) {
            base[j] = mine[j];
            live |= is_nodata(nodata, base[j]) ? 0u : 1u << j;
        }
        bases[cell0 + j] = base[j];
        best[cell0 + j] = ordered(double(base[j]));
    }
    uint32_t rowLive = live << myCol;
#pragma unroll
    for (int d = 1; d < 8; d <<= 1) {  // the row's 8 lanes
        rowLive |= __shfl_xor_sync(0xffffffffu, rowLive, d);
    }
    if (lane % 8u == 0u) {
        liveRows[myRow] = rowLive;
    }
    __syncthreads();
    uint32_t phase[2] = {0u, 0u};
    uint32_t evaluated = 0;
    for (uint32_t c = 0; c < chunks; ++c) {
        const uint32_t s = c & 1u;
        const bool arrived = mbar_wait(&bars[s], phase[s], polls);
        if (__syncthreads_or(!arrived)) {
            // A copy did not land within `polls`: record it, then wait (bounded by the default
            // limit) for the copies still in flight into this buffer and the other one (chunk
            // c + 1 is issued by now), so no bulk copy is left writing into a finished CTA.
            if (tid == 0) {
                atomicOr(flags, 2u);
                mbar_wait(&bars[s], phase[s]);
                if (c + 1 < chunks) {
                    mbar_wait(&bars[s ^ 1u], phase[s ^ 1u]);
                }
            }
            return;
        }
        phase[s] ^= 1u;
        const uint32_t n = min(kChunk, count - c * kChunk);
        // Warp 0: each window's part of the bin and the scan of their sizes.
        if (warp == 0) {
            constexpr uint32_t kEach = kChunk / 32u;
            uint32_t size[kEach], sum = 0;
#pragma unroll
            for (uint32_t i = 0; i < kEach; ++i) {
                const uint32_t e = kEach * lane + i;
                BakeBox box{0, 0, 0, 0, 0.0f};
                if (e < n) {
                    const BoulderEntry& b = stage[s][e];
                    const int c0 = max(b.c0 - int(col0), 0), c1 = min(b.c1 - int(col0), 32);
                    const int r0 = max(b.r0 - int(row0), 0), r1 = min(b.r1 - int(row0), 32);
                    if (c0 < c1 && r0 < r1) {
                        box.c0 = uint16_t(c0);
                        box.r0 = uint16_t(r0);
                        box.wide = uint16_t(c1 - c0);
                        box.cells = uint16_t((c1 - c0) * (r1 - r0));
                        box.inverse = 1.0f / float(c1 - c0);
                    }
                }
                boxes[e] = box;
                size[i] = box.cells;
                sum += box.cells;
            }
            uint32_t before = sum;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, before, d);
                before += lane >= uint32_t(d) ? v : 0u;
            }
            const uint32_t total = __shfl_sync(0xffffffffu, before, 31);
            before -= sum;
#pragma unroll
            for (uint32_t i = 0; i < kEach; ++i) {
                starts[kEach * lane + i] = before;
                before += size[i];
            }
            for (uint32_t e = kChunk + lane; e <= kStarts; e += 32u) {
                starts[e] = total;
            }
        }
        __syncthreads();
        const uint32_t total = starts[kStarts];
        for (uint32_t f = tid; f < total; f += kThreads) {
            uint32_t e = 0;
#pragma unroll
            for (uint32_t step = kStarts / 2; step > 0; step >>= 1) {
                e += starts[e + step] <= f ? step : 0u;  // the last whose first cell is at most f
            }
            const BakeBox box = boxes[e];
            const uint32_t local = f - starts[e];
            const uint32_t r = uint32_t((float(local) + 0.5f) * box.inverse);
            const uint32_t row = box.r0 + r, col = box.c0 + local - r * box.wide;
            if (!((liveRows[row] >> col) & 1u)) {
                continue;
            }
            ++evaluated;
            // The cell's center in double (Raster::CellCenter), and RockRelief without facets:
            // the dome, not below 0 (boulder.h:90-95).
            const BoulderEntry& b = stage[s][e];
            const double x = grid.originX + (double(col0 + col) + 0.5) * grid.pixelWidth;
            const double y = grid.originY + (double(row0 + row) + 0.5) * grid.pixelHeight;
            const double relief = fmax(dome(b, hypot(x - b.x, y - b.y), width), 0.0);
            if (relief > 0.0) {
                const uint32_t cell = row * kBinCells + col;
                atomicMax(best + cell, ordered(double(bases[cell]) + b.weight * relief));
            }
        }
        __syncthreads();
        if (tid == 0 && c + 2 < chunks) {
            issue(c + 2);
        }
    }
    const uint32_t warpPairs = __reduce_add_sync(0xffffffffu, evaluated);
    if (lane == 0 && warpPairs > 0) {
        atomicAdd(reinterpret_cast<unsigned long long*>(flags + 2), (unsigned long long)warpPairs);
    }
#pragma unroll
    for (int j = 0; j < kCellsPerThread; ++j) {
        const long long k = best[cell0 + j];
        if (((live >> j) & 1u) != 0u && k != ordered(double(base[j]))) {
            mine[j] = float(unordered(k));
        }
    }
}

}  // namespace

cudaError_t launch_boulder_count(const BoulderRecord* boulders, uint32_t n, const Grid& grid,
                                 double width, const BoulderBins& bins, cudaStream_t stream) {
    if (n == 0) {
        return cudaSuccess;
    }
    boulder_count_kernel<<<(n + 255) / 256, 256, 0, stream>>>(boulders, n, grid, width, bins);
    return cudaGetLastError();
}

cudaError_t launch_boulder_scatter(const BoulderRecord* boulders, uint32_t n,
                                   const BoulderBins& bins, cudaStream_t stream) {
    if (n == 0) {
        return cudaSuccess;
    }
    boulder_scatter_kernel<<<(n + 255) / 256, 256, 0, stream>>>(boulders, n, bins);
    return cudaGetLastError();
}

cudaError_t launch_boulder_bake(const Grid& grid, double width, NoData nodata,
                                const BoulderBins& bins, float* heights, uint32_t* flags,
                                cudaStream_t stream, uint32_t firstBinRow, uint32_t binRows,
                                uint32_t polls) {
    if (firstBinRow >= bins.binsY) {
        return cudaSuccess;
    }
    const uint32_t rowsRun = std::min(binRows, bins.binsY - firstBinRow);
    const uint32_t nbins = bins.binsX * rowsRun;
    if (nbins == 0) {
        return cudaSuccess;
    }
    BoulderBins strip = bins;
    strip.firstBin = firstBinRow * bins.binsX;
    boulder_bake_kernel<<<nbins, kThreads, 0, stream>>>(grid, width, nodata, strip, heights,
                                                        flags, polls);
    return cudaGetLastError();
}

}  // namespace tgb
