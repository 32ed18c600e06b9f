// k_scan.cu -- Danielsson and FastSweep 2D by one CTA or one warp with a row's cells
// in registers (dan_scan.cuh, scan.cuh): the fields for which that is faster than
// the walk by warps over rows in shared memory (k_sweep.cu).
//
// What bounds them: the latency of a row step.  Where each is used, by whole calls
// on value noise (lattice 20) | 30 points, time with k_sweep.cu's kernels over time
// with these:
//   Danielsson 2D, rows of less than 112 cells but for 32 and 64, which fill a
//     warp's lanes: 16 x 400 1.24 | 1.18, 48 x 400 1.39 | 1.14, 80 x 48 1.16 | 1.01,
//     but 64 x 400 0.96 | 0.94, 120 x 400 1.10 | 0.89, 200 x 400 0.81 | 0.67;
//     wide rows in images of few rows, where points leave long chains in x:
//     more than 512 cells and less than 32 rows (1000 x 16 1.04 | 1.22, 2000 x 12
//     0.75 | 1.30), more than 2048 and less than 128 (3000 x 32 0.68 | 1.43,
//     3000 x 150 0.68 | 1.08)
//   Danielsson 3D, rows of less than 1200 cells but for multiples of 256:
//     16 x 60 x 10 1.45 | 1.47, 128 x 60 x 10 1.03 | 0.95, 400 x 60 x 3 1.08 | 1.27,
//     but 256 x 60 x 10 0.70 | 0.61, 1400 x 60 x 3 0.51 | 0.46; one row per slice
//     1.7 to 3.5 up to 700 cells, 0.5 at 1400
//   FastSweep 2D, rows of up to 32 cells (8 x 500 1.41 | 1.43, 32 x 500 1.28 | 1.35,
//     40 x 500 0.54 | 0.47) and wide rows as above (1000 x 16 0.84 | 1.25, 2500 x 16
//     0.89 | 1.84, 2500 x 150 0.80 | 0.98)
#include "dan_scan.cuh"
#include "kernels.h"

namespace dolk {

template <int DIM, int S>
__global__ void __launch_bounds__(512) k_dan_scan(void* __restrict__ dl, int w, int h, int d, int cw)
{
    if constexpr (DIM == 2) {
        __shared__ ScanShared<C2> sh;
        danielsson2_cta<S>(static_cast<uint32_t*>(dl), w, h, cw, sh);
    } else {
        __shared__ ScanShared<C3> sh;
        danielsson3_cta<S>(static_cast<int16_t*>(dl), w, h, d, cw, sh);
    }
}

template <int DIM, int S>
__global__ void __launch_bounds__(32) k_dan_scan_warp(void* __restrict__ dl, int w, int h, int d, int cw)
{
    if constexpr (DIM == 2) danielsson2_warp<S>(static_cast<uint32_t*>(dl), w, h, cw);
    else danielsson3_warp<S>(static_cast<int16_t*>(dl), w, h, d, cw);
}

// ---- FastSweep 2D -------------------------------------------------------------------
// Four quadrant sweeps; the first row of each sweep is left as is; each later
// row takes the previous row's cell, then along x the previous cell of the row
// and the diagonal cell of the previous row, in that order (:655-693).  The
// diagonal candidate of a segment's first cell is its predecessor's boundary
// cell of the previous row, posted during the previous row's pass.

template <int S>
__global__ void __launch_bounds__(512) k_fastsweep2_scan(uint32_t* __restrict__ dl, int w, int h, int cw)
{
    __shared__ ScanShared<C2> sh;
    const int t = threadIdx.x;
    const int nseg = (w + S - 1) / S;
    const bool active = t < nseg;
    const int n = active ? min(S, w - t * S) : 0;
    const long long x0 = (long long)t * S;
    C2 P[S], C[S], V[S], R[S], D[S];
#pragma unroll
    for (int s = 0; s < S; s++) P[s] = C[s] = V[s] = R[s] = D[s] = C2{0, 0};
    if (h < 2) return;

    for (int sweep = 0; sweep < 4; sweep++) {
        const int dx = (sweep & 1) ? -1 : 1, dy = (sweep & 2) ? -1 : 1;
        const int ox = -cw * dx, oy = -cw * dy;
        const int y0 = dy > 0 ? 0 : h - 1;
        const int pred = t - dx;   // predecessor in this sweep's scan order
        const bool has_pred = active && pred >= 0 && pred < nseg;
        load_row<C2, S>(P, dl, (long long)y0 * w + x0, n);
        load_row<C2, S>(C, dl, (long long)(y0 + dy) * w + x0, n);
#pragma unroll
        for (int s = 0; s < S; s++) V[s] = closer(C[s], add(P[s], 0, oy));
        int g = 0;
        __syncthreads();   // the previous sweep's last pass may still read the slots
        if (active) {
            sh.guess[g][t] = dx > 0 ? seg_edge<C2, S, +1>(V, n) : seg_edge<C2, S, -1>(V, n);
            sh.edge[g][t] = dx > 0 ? seg_edge<C2, S, +1>(P, n) : seg_edge<C2, S, -1>(P, n);
        }
        __syncthreads();
        for (int j = 1; j < h; j++) {
            const int y = y0 + j * dy;
            const bool more = j + 1 < h;
            if (more) load_row<C2, S>(C, dl, (long long)(y + dy) * w + x0, n);
            // diagonal candidates from the previous row (P): own cells, then the predecessor's edge
            if (dx > 0) {
#pragma unroll
                for (int s = 1; s < S; s++) D[s] = add(P[s - 1], ox, oy);
            } else {
#pragma unroll
                for (int s = 0; s + 1 < S; s++) D[s] = add(P[s + 1], ox, oy);
            }
            if (has_pred) {
                const C2 e = add(sh.edge[g][pred], ox, oy);
                if (dx > 0) D[0] = e;
                else {
#pragma unroll
                    for (int s = 0; s < S; s++)
                        if (s == n - 1) D[s] = e;
                }
            }
            const C2 in0 = has_pred ? sh.guess[g][pred] : V[0];
            auto post = [&](const C2 (&X)[S]) {
                if (!active) return;
                if (dx > 0) {
                    sh.edge[g ^ 1][t] = seg_edge<C2, S, +1>(X, n);
                    if (more) sh.guess[g ^ 1][t] = closer(seg_edge<C2, S, +1>(C, n), add(seg_edge<C2, S, +1>(X, n), 0, oy));
                } else {
                    sh.edge[g ^ 1][t] = seg_edge<C2, S, -1>(X, n);
                    if (more) sh.guess[g ^ 1][t] = closer(seg_edge<C2, S, -1>(C, n), add(seg_edge<C2, S, -1>(X, n), 0, oy));
                }
            };
            if (dx > 0)
                row_pass<C2, S, true, +1>(R, V, t, nseg, n, cw, sh, D, in0, post);
            else
                row_pass<C2, S, true, -1>(R, V, t, nseg, n, cw, sh, D, in0, post);
            g ^= 1;
            store_row<C2, S>(dl, (long long)y * w + x0, R, n);
#pragma unroll
            for (int s = 0; s < S; s++) {
                P[s] = R[s];
                if (more) V[s] = closer(C[s], add(P[s], 0, oy));
            }
        }
    }
}

template <int S>
__global__ void __launch_bounds__(32) k_fastsweep2_scan_warp(uint32_t* __restrict__ dl, int w, int h, int cw)
{
    const int lane = threadIdx.x & 31;
    const int nseg = (w + S - 1) / S;
    const bool active = lane < nseg;
    const int n = active ? min(S, w - lane * S) : 0;
    const long long x0 = (long long)lane * S;
    C2 P[S], C[S], V[S], R[S], D[S];
#pragma unroll
    for (int s = 0; s < S; s++) P[s] = C[s] = V[s] = R[s] = D[s] = C2{0, 0};
    if (h < 2) return;
    for (int sweep = 0; sweep < 4; sweep++) {
        const int dx = (sweep & 1) ? -1 : 1, dy = (sweep & 2) ? -1 : 1;
        const int ox = -cw * dx, oy = -cw * dy;
        const int y0 = dy > 0 ? 0 : h - 1;
        const int pred = lane - dx;
        const bool has_pred = active && pred >= 0 && pred < nseg;
        const int src = pred < 0 ? 0 : (pred > 31 ? 31 : pred);
        load_row<C2, S>(P, dl, (long long)y0 * w + x0, n);
        load_row<C2, S>(C, dl, (long long)(y0 + dy) * w + x0, n);
#pragma unroll
        for (int s = 0; s < S; s++) V[s] = closer(C[s], add(P[s], 0, oy));
        for (int j = 1; j < h; j++) {
            const int y = y0 + j * dy;
            const bool more = j + 1 < h;
            if (more) load_row<C2, S>(C, dl, (long long)(y + dy) * w + x0, n);
            // diagonal candidates from the previous row: own cells, then the predecessor's edge
            C2 e;
            if (dx > 0) {
#pragma unroll
                for (int s = 1; s < S; s++) D[s] = add(P[s - 1], ox, oy);
                e = shfl_cell(0xFFFFFFFFu, seg_edge<C2, S, +1>(P, n), src);
            } else {
#pragma unroll
                for (int s = 0; s + 1 < S; s++) D[s] = add(P[s + 1], ox, oy);
                e = shfl_cell(0xFFFFFFFFu, seg_edge<C2, S, -1>(P, n), src);
            }
            if (has_pred) {
                e = add(e, ox, oy);
                if (dx > 0) D[0] = e;
                else {
#pragma unroll
                    for (int s = 0; s < S; s++)
                        if (s == n - 1) D[s] = e;
                }
            }
            if (dx > 0)
                row_pass_warp<C2, S, true, +1>(R, V, lane, nseg, n, cw, D, warp_round0_input<C2, S, +1>(V, n, lane));
            else
                row_pass_warp<C2, S, true, -1>(R, V, lane, nseg, n, cw, D, warp_round0_input<C2, S, -1>(V, n, lane));
            store_row<C2, S>(dl, (long long)y * w + x0, R, n);
#pragma unroll
            for (int s = 0; s < S; s++) {
                P[s] = R[s];
                if (more) V[s] = closer(C[s], add(P[s], 0, oy));
            }
        }
    }
}

// few wide rows (images)
static bool few_wide_rows(int w, int h) { return w > 2048 ? h < 128 : w > 512 && h < 32; }

static int threads(int w, int s) { return ((w + s - 1) / s + 31) / 32 * 32; }

// false: another kernel is faster for this field
bool launch_danielsson_scan(int dim, void* deltas, int w, int h, int d, int cw, cudaStream_t st)
{
    if (dim == 2) {
        if (few_wide_rows(w, h)) {
            if (w <= 1024) k_dan_scan<2, 4><<<1, threads(w, 4), 0, st>>>(deltas, w, h, 1, cw);
            else k_dan_scan<2, 8><<<1, threads(w, 8), 0, st>>>(deltas, w, h, 1, cw);
            return true;
        }
        if (w >= 112 || w == 32 || w == 64) return false;
        if (w < 32) k_dan_scan_warp<2, 1><<<1, 32, 0, st>>>(deltas, w, h, 1, cw);
        else if (w < 64) k_dan_scan_warp<2, 2><<<1, 32, 0, st>>>(deltas, w, h, 1, cw);
        else k_dan_scan_warp<2, 4><<<1, 32, 0, st>>>(deltas, w, h, 1, cw);
        return true;
    }
    if (w >= 1200 || (w % 256 == 0 && h > 1)) return false;
    if (w <= 32) k_dan_scan_warp<3, 1><<<1, 32, 0, st>>>(deltas, w, h, d, cw);
    else if (w <= 64) k_dan_scan_warp<3, 2><<<1, 32, 0, st>>>(deltas, w, h, d, cw);
    else if (w <= 128) k_dan_scan_warp<3, 4><<<1, 32, 0, st>>>(deltas, w, h, d, cw);
    else if (w <= 256) k_dan_scan_warp<3, 8><<<1, 32, 0, st>>>(deltas, w, h, d, cw);
    else if (w <= 512) k_dan_scan<3, 2><<<1, threads(w, 2), 0, st>>>(deltas, w, h, d, cw);
    else if (w <= 1024) k_dan_scan<3, 4><<<1, threads(w, 4), 0, st>>>(deltas, w, h, d, cw);
    else k_dan_scan<3, 8><<<1, threads(w, 8), 0, st>>>(deltas, w, h, d, cw);
    return true;
}

bool launch_fastsweep_2d_scan(void* deltas, int w, int h, int cw, cudaStream_t st)
{
    uint32_t* dl = static_cast<uint32_t*>(deltas);
    if (few_wide_rows(w, h)) {
        if (w <= 1024) k_fastsweep2_scan<4><<<1, threads(w, 4), 0, st>>>(dl, w, h, cw);
        else k_fastsweep2_scan<8><<<1, threads(w, 8), 0, st>>>(dl, w, h, cw);
        return true;
    }
    if (w > 32) return false;
    k_fastsweep2_scan_warp<1><<<1, 32, 0, st>>>(dl, w, h, cw);
    return true;
}

}  // namespace dolk
