// dan_serial.cuh -- Danielsson (DistanceOcclusionLib.cpp:702-778 2D, :2264-2394
// 3D) as one serial walk of a field by NW warps: rows in place, each row's x
// passes exact in parallel (row.cuh).
#pragma once

#include "row.cuh"

namespace dolk {

// Rows of a field as one warp group sees them
template <int DIM, int S>
struct Field {
    unsigned char *lo, *hi;   // the array
    int w, h, xw;             // xw: the warp's first cell

    DOL_DI unsigned char* row(int z, int y) const
    {
        return lo + (((long long)z * h + y) * w + xw) * (DIM == 3 ? 6 : 4);
    }
};

// V[s] = closer(V[s], the slice before shifted by dz)
template <int S>
DOL_DI void pull_z(Cells<3, S>& V, const uint32_t (&xy)[S], const int (&z)[S], int dz)
{
#pragma unroll
    for (int s = 0; s < S; s++) consider(V, s, xy[s], trunc16(z[s] + dz));
}

// The right and the left x pass of a row
template <int DIM, int S, int NW>
DOL_DI void x_passes(Cells<DIM, S>& V, int cw, RowShared<NW>& sh, int& par)
{
    row_pass_w<DIM, S, NW, +1, NoDiag>(V, NoDiag{}, cw, sh, par, chain_none(cw));
    row_pass_w<DIM, S, NW, -1, NoDiag>(V, NoDiag{}, cw, sh, par, chain_none(cw));
}

// rows in flight: a row and the slice before's
template <int DIM, int S>
using SerialIO = RowIO<DIM, S, DIM == 3 ? 2 : 1>;

// The whole field, or one way (0: up, 1: down) through a volume's slices; all 32 NW
// threads of the group call it together.  `strip`: this warp's RowIO strips.
template <int DIM, int S, int NW>
__device__ void dan_serial(void* cells, int w, int h, int d, int cw, unsigned char* strip, RowShared<NW>& sh,
                           int way = -1)
{
    using IO = SerialIO<DIM, S>;
    using Row = Cells<DIM, S>;
    if (h < 2 && DIM == 2) return;
    const int wi = (threadIdx.x >> 5) & (NW - 1);
    Field<DIM, S> f;
    f.lo = static_cast<unsigned char*>(cells);
    f.hi = f.lo + (long long)w * h * (DIM == 3 ? d : 1) * IO::kCell;
    f.w = w;
    f.h = h;
    f.xw = wi * 32 * S;
    const IO io{strip, min(32 * S, w - f.xw)};
    const int steps = 2 * (h - 1);
    auto row_of = [&](int i) { return i < h - 1 ? i + 1 : 2 * h - 3 - i; };
    int par = 0;
    Row P, V;
    constexpr int rc = 0, rq = 1;   // strips: the next row, the row of the slice before
    const int pass0 = DIM == 3 && way > 0 ? way : 0, pass1 = DIM == 3 && way != 0 ? 2 : 1, first = DIM == 3 ? 1 : 0, last = DIM == 3 ? d : 1;
    for (int pass = pass0; pass < pass1; pass++) {
        const int dz = pass == 0 ? -cw : cw;
        for (int k = first; k < last; k++) {
            const int z = DIM == 3 ? (pass == 0 ? k : d - 1 - k) : 0;
            const int zp = pass == 0 ? z - 1 : z + 1;
            auto zpull = [&](Row& r, int y) {   // the fetched row rq of the slice before
                if constexpr (DIM == 3) {
                    uint32_t wd[IO::kWords], xy[S];
                    int zz[S];
                    io.words(wd, rq, f.row(zp, y));
                    IO::split(wd, xy, zz);
                    pull_z<S>(r, xy, zz, dz);
                }
            };
            __syncwarp();   // the previous slice's last rows are stored
            io.fetch(rc, f.row(z, 0), f.lo, f.hi);
            if (DIM == 3) io.fetch(rq, f.row(zp, 0), f.lo, f.hi);
            io.cells_of(P, rc, f.row(z, 0), cw);
            if (DIM == 3) {   // row 0: the z pull only
                zpull(P, 0);
                if (h > 1) {
                    io.fetch(rc, f.row(z, 1), f.lo, f.hi);
                    io.fetch(rq, f.row(zp, 1), f.lo, f.hi);
                }
                io.put_cells(f.row(z, 0), P);
            } else {
                io.fetch(rc, f.row(z, 1), f.lo, f.hi);
            }
            for (int i = 0; i < steps; i++) {
                const int y = row_of(i);
                const bool down = i < h - 1;
                io.cells_of(V, rc, f.row(z, y), cw);
                if (DIM == 3 && down) zpull(V, y);
                if (i + 1 < steps) {   // the next row, while this one is scanned
                    const int yn = row_of(i + 1);
                    io.fetch(rc, f.row(z, yn), f.lo, f.hi);
                    if (DIM == 3 && i + 1 < h - 1) io.fetch(rq, f.row(zp, yn), f.lo, f.hi);
                }
                merge_y<DIM, S>(P, V, down ? -cw : cw);
                x_passes<DIM, S, NW>(P, cw, sh, par);
                io.put_cells(f.row(z, y), P);
            }
        }
    }
}

}  // namespace dolk
