// dan_slices.cuh -- Danielsson 3D (DistanceOcclusionLib.cpp:2264-2394) of one
// volume by one CTA: slices in order, the rows of a slice in parallel chunks.
//
// A slice's sweep needs the finished slice before it, so a volume is a chain of
// slices.  Inside a slice the chain of rows is cut into one chunk of rows per
// warp and solved as a fixed point, as k_dan_blocks.cu does for whole volumes:
// a chunk's down sweep takes the last down row of the chunk above, its up
// sweep the first finished row of the chunk below, both as last seen; chunks
// whose inputs changed run again.  Consecutive slices differ little, so the
// rows seen start as the slice before's, shifted by the slice step: most
// slices settle in two or three rounds, each as long as one chunk's rows,
// where the serial walk takes every row in turn.
#pragma once

#include "dan_serial.cuh"

namespace dolk {

// NW warps, rows of at most 32 S cells.
template <int S>
struct SliceIO {
    using IO = SerialIO<3, S>;
    // cells of a row in shared memory: S words and S halves per lane
    static constexpr size_t kRow = (size_t)S * 32 * 6;
    // strips of the warps, the slice's h rows, three boundary rows per chunk, a flag word per chunk
    static __host__ __device__ constexpr size_t bytes(int h, int nw)
    {
        return nw * IO::kBytes + (size_t)h * kRow + 3 * (size_t)nw * kRow;
    }
    DOL_DI static void put(unsigned char* row, const Cells<3, S>& v)
    {
        const int lane = threadIdx.x & 31;
        uint32_t* a = reinterpret_cast<uint32_t*>(row);
        int16_t* b = reinterpret_cast<int16_t*>(row + (size_t)S * 128);
#pragma unroll
        for (int s = 0; s < S; s++) {
            a[s * 32 + lane] = v.xy[s];
            b[s * 32 + lane] = (int16_t)v.z[s];
        }
    }
    DOL_DI static void get(const unsigned char* row, uint32_t (&xy)[S], int (&z)[S])
    {
        const int lane = threadIdx.x & 31;
        const uint32_t* a = reinterpret_cast<const uint32_t*>(row);
        const int16_t* b = reinterpret_cast<const int16_t*>(row + (size_t)S * 128);
#pragma unroll
        for (int s = 0; s < S; s++) {
            xy[s] = a[s * 32 + lane];
            z[s] = b[s * 32 + lane];
        }
    }
    // as cells; those past the row's end as "none"
    DOL_DI static void get(const unsigned char* row, Cells<3, S>& c, int live, int cw)
    {
        get(row, c.xy, c.z);
#pragma unroll
        for (int s = 0; s < S; s++) {
            c.W[s] = w_of<3>(c.xy[s], c.z[s]);
            c.L[s] = len_of(c.xy[s], c.W[s]);
        }
        if (live < S) {
#pragma unroll
            for (int s = 0; s < S; s++)
                if (s >= live) set_none(c, s, cw);
        }
    }
};

// The whole volume, in place, by a CTA of NW warps; smem: SliceIO<S>::bytes.
template <int S, int NW>
__device__ void dan_slices(void* cells, int w, int h, int d, int cw, unsigned char* smem)
{
    using SM = SliceIO<S>;
    using IO = typename SM::IO;
    using Row = Cells<3, S>;
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    Field<3, S> f;
    f.lo = static_cast<unsigned char*>(cells);
    f.hi = f.lo + (long long)w * h * d * IO::kCell;
    f.w = w;
    f.h = h;
    f.xw = 0;
    const IO io{smem + wi * IO::kBytes, w};
    unsigned char* rows = smem + NW * IO::kBytes;      // the slice
    unsigned char* seenD = rows + (size_t)h * SM::kRow;   // per chunk: its last down row, as the chunk below saw it
    unsigned char* seenU = seenD + NW * SM::kRow;         // its first finished row, as the chunk above saw it
    unsigned char* newD = seenU + NW * SM::kRow;
    __shared__ unsigned s_changed[2][NW];   // bit 0: the down row, bit 1: the first row
    const int R = (h + NW - 1) / NW, nc = (h + R - 1) / R;
    const int y0 = wi * R, y1 = min(y0 + R, h), L = max(0, y1 - y0);   // chunk wi; none for wi >= nc
    const bool has_d = wi > 0 && L > 0, has_u = L > 0 && y1 < h;
    const int n = io.live();
    constexpr int ra = 0, rz = 1;   // strips: the row itself, the row of the slice before
    auto absent = [&](Row& r) {   // wins against none when shifted by +-cw in y
#pragma unroll
        for (int s = 0; s < S; s++) {
            r.xy[s] = 0;
            r.z[s] = 0;
            r.W[s] = 0;
            r.L[s] = INT_MAX - cw * cw;
        }
    };
    bool fresh = true;   // no slice before gives the rows seen
    for (int pass = 0; pass < 2; pass++) {
        const int dz = pass == 0 ? -cw : cw;
        for (int k = 1; k < d; k++) {
            const int z = pass == 0 ? k : d - 1 - k;
            const int zp = pass == 0 ? z - 1 : z + 1;
            // the rows seen: the slice before's, one step on in z (a guess; any would do)
            if (L > 0 && !fresh) {
                for (unsigned char* row : {seenD + wi * SM::kRow, seenU + wi * SM::kRow}) {
                    int16_t* b = reinterpret_cast<int16_t*>(row + (size_t)S * 128);
#pragma unroll
                    for (int s = 0; s < S; s++) b[s * 32 + lane] = (int16_t)(b[s * 32 + lane] + dz);
                }
            }
            if (lane == 0) s_changed[0][wi] = 3u;
            __syncthreads();   // and: the slice before is stored
            for (int round = 0;; round++) {
                // run when an input changed in the round before (the first round: always)
                const unsigned in = (wi > 0 ? s_changed[round & 1][wi - 1] & 1u : 0u) |
                                    (wi + 1 < nc ? s_changed[round & 1][wi + 1] & 2u : 0u);
                const bool run = L > 0 && (round == 0 || in != 0);
                unsigned changed = 0;
                if (run) {
                    Row P, C;
                    io.fetch(ra, f.row(z, y0), f.lo, f.hi);
                    io.fetch(rz, f.row(zp, y0), f.lo, f.hi);
                    if (has_d && !(fresh && round == 0)) SM::get(seenD + (wi - 1) * SM::kRow, P, n, cw);
                    else absent(P);
#pragma unroll 1
                    for (int i = 0; i < 2 * L; i++) {
                        const bool down = i < L;
                        const int q = down ? i : 2 * L - 1 - i, y = y0 + q;
                        if (down) {
                            io.cells_of(C, ra, f.row(z, y), cw);
                            uint32_t wd[IO::kWords], xy[S];
                            int zz[S];
                            io.words(wd, rz, f.row(zp, y));
                            IO::split(wd, xy, zz);
                            pull_z<S>(C, xy, zz, dz);
                            if (i + 1 < L) {
                                io.fetch(ra, f.row(z, y + 1), f.lo, f.hi);
                                io.fetch(rz, f.row(zp, y + 1), f.lo, f.hi);
                            }
                        } else if (i > L) {
                            SM::get(rows + (size_t)y * SM::kRow, C, n, cw);
                        } else {   // the turn
                            C = P;
                            if (has_u && !(fresh && round == 0)) SM::get(seenU + (wi + 1) * SM::kRow, P, n, cw);
                            else absent(P);
                        }
                        // (slice row 0 has no passes going down, its last row none going up)
                        merge_y<3, S>(P, C, down ? -cw : cw);
                        if (down ? y > 0 : y < h - 1) {
                            RowShared<1> none;
                            int par = 0;
                            x_passes<3, S, 1>(P, cw, none, par);
                        }
                        SM::put(rows + (size_t)y * SM::kRow, P);
                        if (i == L - 1) SM::put(newD + wi * SM::kRow, P);
                    }
                }
                __syncthreads();   // the rows seen have been read
                if (run) {
                    auto update = [&](unsigned char* seen, const unsigned char* now) -> bool {
                        uint32_t a[S], b[S];
                        int az[S], bz[S];
                        SM::get(seen, a, az);
                        SM::get(now, b, bz);
                        bool diff = fresh && round == 0;
#pragma unroll
                        for (int s = 0; s < S; s++) diff |= s < n && (a[s] != b[s] || az[s] != bz[s]);
                        const bool any = __any_sync(0xFFFFFFFFu, diff);
                        if (any) {
                            uint32_t* pa = reinterpret_cast<uint32_t*>(seen);
                            int16_t* pb = reinterpret_cast<int16_t*>(seen + (size_t)S * 128);
#pragma unroll
                            for (int s = 0; s < S; s++) {
                                pa[s * 32 + lane] = b[s];
                                pb[s * 32 + lane] = (int16_t)bz[s];
                            }
                        }
                        return any;
                    };
                    if (wi + 1 < nc && update(seenD + wi * SM::kRow, newD + wi * SM::kRow)) changed |= 1u;
                    if (wi > 0 && update(seenU + wi * SM::kRow, rows + (size_t)y0 * SM::kRow)) changed |= 2u;
                }
                if (lane == 0) s_changed[(round & 1) ^ 1][wi] = changed;
                if (!__syncthreads_or(changed != 0)) break;
                if (round > 2 * NW + 8) break;   // (a chunk more is right after every other round)
            }
            fresh = false;
            // the slice is final: store it
            if (L > 0) {
                for (int y = y0; y < y1; y++) {
                    Row P;
                    SM::get(rows + (size_t)y * SM::kRow, P.xy, P.z);
                    io.put_cells(f.row(z, y), P);
                }
            }
        }
        fresh = true;   // the other direction starts from rows that have not been seen
    }
    __syncthreads();
}

}  // namespace dolk
