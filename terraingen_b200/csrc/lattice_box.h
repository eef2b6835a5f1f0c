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

}  // namespace tgb
