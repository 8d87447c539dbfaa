// Cost of a column-pair stage by strip height, for the rules that choose it.
#pragma once

#include <math.h>

#include "dispatch.cuh"

namespace go {

// Time (arbitrary units) of `blocks` strips of r rows: whole waves of the
// resident blocks, and of the last, partly filled one a share that grows with
// its filling; see pair_rows for the fit.
inline double pair_strip_cost(long long blocks, int r) {
    const double w = (double)blocks / (148.0 * shape_blocks_per_sm(GO_SHAPE_PAIR));
    const double whole = floor(w), f = w - whole;
    return (r + 2) * (whole + (f > 0.0 ? 0.35 + 0.65 * f : 0.0)) * (2.2 + 0.2 / ceil(w));
}

}  // namespace go
