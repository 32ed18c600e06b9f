// diagonals.h -- rows on the anti-diagonals of FastSweep 3D's wavefront.  The CPU
// tests compile it.
#pragma once

#include "common.cuh"

namespace dolk {

// pairs (jj, kk) in 1 .. H, 1 .. D with jj + kk < c
DOL_HD int rows_before_diagonal(int H, int D, int c)
{
    const long long m = H < c - 2 ? H : c - 2;
    if (m <= 0) return 0;
    long long full = c - 1 - D;   // jj up to this many have all D of theirs
    full = full < 0 ? 0 : (full > m ? m : full);
    return (int)(full * D + (m - full) * (c - 1) - (m * (m + 1) - full * (full + 1)) / 2);
}

}  // namespace dolk
