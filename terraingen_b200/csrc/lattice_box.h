// Which lattice positions a block may look up in a shared table. A cell's place in the table is
// formed from its position's bits without a bounds check (packed.cuh), so a grid is tabled only
// where every position is known to be a number inside the box the block hashed.
#pragma once

#include <cmath>

#include "kernels.h"

namespace tgb {

// The largest |x| + |y| of a cell's corner from the origin, and infinity unless every corner of
// the grid is a number below 2^100: the cells' positions lie between the corners', so they are
// finite as floats and stay so through an octave's turn.
inline double lattice_reach(const Grid& g, const Positions& at) {
    double reach = 0.0;
    for (int k = 0; k < 4; ++k) {
        const double c = k & 1 ? double(g.width) : 0.0, r = k & 2 ? double(g.height) : 0.0;
        const double x = g.originX + c * g.pixelWidth + r * g.rowRotation - at.originX;
        const double y = g.originY + c * g.colRotation + r * g.pixelHeight - at.originY;
        const double far = std::fabs(x) + std::fabs(y);
        if (!(far < 0x1p100)) {
            return INFINITY;  // NaN too, which a maximum would drop
        }
        reach = far > reach ? far : reach;
    }
    return reach;
}

// Whether an octave's positions over a grid of that reach are good to 1/8 of a lattice cell and
// within kFloorShift's exact range: below 2^18 lattice cells. False for a frequency that is not a
// number, and for an infinite one.
inline bool lattice_tabled(double reach, float frequency) {
    return reach * std::fabs(double(frequency)) < 262144.0;
}

// The smallest box of an octave's positions, from its anchor, over columns [c0, c1] and rows
// [r0, r1]: those at the four corners.
struct LatticeBox {
    float x0, x1, y0, y1;
};
TG_HD inline LatticeBox lattice_box(const OctaveAnchor& a, uint32_t c0, uint32_t c1, uint32_t r0,
                                    uint32_t r1) {
    LatticeBox b{INFINITY, -INFINITY, INFINITY, -INFINITY};
    for (int k = 0; k < 4; ++k) {
        const float fc = float(k & 1 ? c1 : c0), fr = float(k & 2 ? r1 : r0);
        const float qx = fmaf(fc, a.ax, fmaf(fr, a.ay, a.fx));
        const float qy = fmaf(fc, a.bx, fmaf(fr, a.by, a.fy));
        b.x0 = fminf(b.x0, qx);
        b.x1 = fmaxf(b.x1, qx);
        b.y0 = fminf(b.y0, qy);
        b.y1 = fmaxf(b.y1, qy);
    }
    return b;
}

// Whether a table may hold the box: within kFloorShift's range and small enough to count in 32
// bits. Corners that are not numbers leave no trace in a minimum or a maximum, so a box of none
// but such corners is empty, and refused here. No box has only some: a finite corner means that
// steps and anchor are finite, and then a fused multiply-add gives no NaN.
TG_HD inline bool lattice_boxed(const LatticeBox& b) {
    return b.x0 <= b.x1 && b.y0 <= b.y1 && b.x0 > -2e6f && b.x1 < 2e6f && b.y0 > -2e6f &&
           b.y1 < 2e6f && b.x1 - b.x0 < 1024.0f && b.y1 - b.y0 < 1024.0f;
}

}  // namespace tgb
