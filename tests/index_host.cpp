// Host build of the offset arithmetic of large fields (csrc/border.cuh,
// csrc/edt_layout.h) for the CPU tests.
#include "border.cuh"
#include "edt_layout.h"

extern "C" void host_word_cells(long long wid, int w, long long* first, int* n)
{
    dolk::word_cells(wid, w, dolk::words_per_row(w), first, n);
}
extern "C" size_t host_edt_x_bytes(int pitch, int h, int d) { return dolk::edt_x_bytes(pitch, (long long)h * d); }
extern "C" size_t host_edt_bytes(int dim, int pitch, int h, int d) { return dolk::edt_bytes(dim, pitch, h, d); }
