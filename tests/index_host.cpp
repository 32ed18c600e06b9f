// Host build of the offset arithmetic of large fields (csrc/edt_layout.h) for the CPU tests.
#include "edt_layout.h"

extern "C" size_t host_edt_x_bytes(int pitch, int h, int d) { return dolk::edt_x_bytes(pitch, (long long)h * d); }
extern "C" size_t host_edt_bytes(int dim, int pitch, int h, int d) { return dolk::edt_bytes(dim, pitch, h, d); }
