// Host build of csrc/diagonals.h for the CPU tests.
#include "diagonals.h"

extern "C" int host_rows_before_diagonal(int H, int D, int c) { return dolk::rows_before_diagonal(H, D, c); }
