// edt_layout.h -- where the fields of the mask EDT lie in its workspace.  Plain C++,
// so that the CPU tests compile it.
#pragma once

#include <stddef.h>

namespace dolk {

// the x pass's 16-bit field, rows `pitch` cells apart; a volume's y pass field
// (32 bits) starts behind it.  `rows`: h, times d in a volume (above 2^31 for
// narrow volumes: 1 x 46341 x 46341).
inline size_t edt_x_bytes(int pitch, long long rows)
{
    return ((size_t)pitch * (size_t)rows * 2 + 255) & ~(size_t)255;
}

inline size_t edt_bytes(int dim, int pitch, int h, int d)
{
    const long long rows = (long long)h * (dim == 3 ? d : 1);
    return edt_x_bytes(pitch, rows) + (dim == 3 ? (size_t)pitch * (size_t)rows * 4 : 0);
}

}  // namespace dolk
