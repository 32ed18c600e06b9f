// dan_scan.cuh -- Danielsson (DistanceOcclusionLib.cpp:702-778 2D, :2264-2394 3D) as
// one serial walk of a field whose rows stay in the registers of a CTA or a
// warp, S cells per thread, cells loaded and stored one by one (scan.cuh).
//
// The walk by warps in dan_serial.cuh moves whole 16-byte pieces through shared
// memory and tests a row before it walks it, which pays for rows that fill its
// lanes.  A step is shorter here for narrow rows and for small volumes
// (k_scan.cu has the rule and the figures).
#pragma once

#include "scan.cuh"

namespace dolk {

template <class Cell, int S, class P>
__device__ __forceinline__ void load_row(Cell (&dst)[S], const P* base, long long row_first, int n)
{
#pragma unroll
    for (int s = 0; s < S; s++)
        if (s < n) dst[s] = cell_load(base, row_first + s);
}
template <class Cell, int S, class P>
__device__ __forceinline__ void store_row(P* base, long long row_first, const Cell (&src)[S], int n)
{
#pragma unroll
    for (int s = 0; s < S; s++)
        if (s < n) cell_store(base, row_first + s, src[s]);
}

// ---- by a CTA ----------------------------------------------------------------------
// 2D: rows 1..h-1 going down, then h-2..0 going up (:709-777): one "step" per row,
// the row taking the previous step's row with a y offset of -cw (down) or
// +cw (up), then an x pass to the right and one to the left.  The next step's
// row is loaded during the current one, and each pass posts what the next
// pass needs (row_pass), so a step costs two barriers when the passes settle
// in one round.

template <int S>
__device__ __forceinline__ void danielsson2_cta(uint32_t* __restrict__ dl, int w, int h, int cw, ScanShared<C2>& sh)
{
    const int t = threadIdx.x;
    const int nseg = (w + S - 1) / S;
    const bool active = t < nseg;
    const int n = active ? min(S, w - t * S) : 0;
    const long long x0 = (long long)t * S;
    if (h < 2) return;
    const int steps = 2 * (h - 1);
    auto row_of = [&](int i) { return i < h - 1 ? i + 1 : 2 * h - 3 - i; };
    auto dy_of = [&](int i) { return i < h - 1 ? -cw : cw; };
    C2 P[S], C[S], V[S], R[S], D[S];
#pragma unroll
    for (int s = 0; s < S; s++) P[s] = C[s] = V[s] = R[s] = D[s] = C2{0, 0};

    load_row<C2, S>(P, dl, x0, n);
    load_row<C2, S>(C, dl, (long long)row_of(0) * w + x0, n);
#pragma unroll
    for (int s = 0; s < S; s++) V[s] = closer(C[s], add(P[s], 0, dy_of(0)));
    int g = 0;
    if (active) sh.guess[g][t] = seg_edge<C2, S, +1>(V, n);
    __syncthreads();
    for (int i = 0; i < steps; i++) {
        const int y = row_of(i);
        const bool more = i + 1 < steps;
        const int dyn = more ? dy_of(i + 1) : 0;
        if (more) load_row<C2, S>(C, dl, (long long)row_of(i + 1) * w + x0, n);
        const C2 in0 = (active && t > 0) ? sh.guess[g][t - 1] : V[0];
        row_pass<C2, S, false, +1>(R, V, t, nseg, n, cw, sh, D, in0, [&](const C2 (&X)[S]) {
            if (active) sh.guess[g ^ 1][t] = X[0];
        });
        g ^= 1;
        const C2 in1 = (active && t + 1 < nseg) ? sh.guess[g][t + 1] : R[0];
        row_pass<C2, S, false, -1>(P, R, t, nseg, n, cw, sh, D, in1, [&](const C2 (&X)[S]) {
            if (more && active)
                sh.guess[g ^ 1][t] = closer(seg_edge<C2, S, +1>(C, n), add(seg_edge<C2, S, +1>(X, n), 0, dyn));
        });
        g ^= 1;
        store_row<C2, S>(dl, (long long)y * w + x0, P, n);
        if (more) {
#pragma unroll
            for (int s = 0; s < S; s++) V[s] = closer(C[s], add(P[s], 0, dyn));
        }
    }
}

// 3D: slices 1..d-1 then d-2..0 (:2355-2393); each slice takes the neighbouring
// slice's cell with the z offset, then runs the 2D steps over its rows
// (:2264-2345).  The z pull is folded into the first load of each row (rows of
// the down sweep); the up sweep reads the down sweep's results.

template <int S>
__device__ __forceinline__ void danielsson3_cta(int16_t* __restrict__ dl, int w, int h, int d, int cw,
                                                ScanShared<C3>& sh)
{
    const int t = threadIdx.x;
    const int nseg = (w + S - 1) / S;
    const bool active = t < nseg;
    const int n = active ? min(S, w - t * S) : 0;
    const long long x0 = (long long)t * S;
    const long long plane = (long long)w * h;
    const int steps = 2 * (h - 1);
    auto row_of = [&](int i) { return i < h - 1 ? i + 1 : 2 * h - 3 - i; };
    auto dy_of = [&](int i) { return i < h - 1 ? -cw : cw; };
    C3 P[S], C[S], Q[S], V[S], R[S], D[S];
#pragma unroll
    for (int s = 0; s < S; s++) P[s] = C[s] = Q[s] = V[s] = R[s] = D[s] = C3{0, 0, 0};

    for (int pass = 0; pass < 2; pass++) {
        const int dz = pass == 0 ? -cw : +cw;
        for (int k = 1; k < d; k++) {
            const int z = pass == 0 ? k : d - 1 - k;
            const int zp = pass == 0 ? z - 1 : z + 1;
            const long long sb = z * plane, pb = (long long)zp * plane;
            // row 0: z pull only
            load_row<C3, S>(C, dl, sb + x0, n);
            load_row<C3, S>(Q, dl, pb + x0, n);
#pragma unroll
            for (int s = 0; s < S; s++) P[s] = closer(C[s], add(Q[s], 0, 0, dz));
            store_row<C3, S>(dl, sb + x0, P, n);
            if (h < 2) continue;
            // first step: row 1 of the down sweep (z pull, then y pull)
            load_row<C3, S>(C, dl, sb + (long long)w + x0, n);
            load_row<C3, S>(Q, dl, pb + (long long)w + x0, n);
#pragma unroll
            for (int s = 0; s < S; s++) V[s] = closer(closer(C[s], add(Q[s], 0, 0, dz)), add(P[s], 0, -cw, 0));
            int g = 0;
            __syncthreads();   // the previous slice's last pass may still read the guess slots
            if (active) sh.guess[g][t] = seg_edge<C3, S, +1>(V, n);
            __syncthreads();
            for (int i = 0; i < steps; i++) {
                const int y = row_of(i);
                const bool more = i + 1 < steps;
                const bool next_down = more && i + 1 < h - 1;
                const int dyn = more ? dy_of(i + 1) : 0;
                if (more) {
                    const long long off = (long long)row_of(i + 1) * w + x0;
                    load_row<C3, S>(C, dl, sb + off, n);
                    if (next_down) load_row<C3, S>(Q, dl, pb + off, n);
                }
                const C3 in0 = (active && t > 0) ? sh.guess[g][t - 1] : V[0];
                row_pass<C3, S, false, +1>(R, V, t, nseg, n, cw, sh, D, in0, [&](const C3 (&X)[S]) {
                    if (active) sh.guess[g ^ 1][t] = X[0];
                });
                g ^= 1;
                const C3 in1 = (active && t + 1 < nseg) ? sh.guess[g][t + 1] : R[0];
                row_pass<C3, S, false, -1>(P, R, t, nseg, n, cw, sh, D, in1, [&](const C3 (&X)[S]) {
                    if (more && active) {
                        C3 c = seg_edge<C3, S, +1>(C, n);
                        if (next_down) c = closer(c, add(seg_edge<C3, S, +1>(Q, n), 0, 0, dz));
                        sh.guess[g ^ 1][t] = closer(c, add(seg_edge<C3, S, +1>(X, n), 0, dyn, 0));
                    }
                });
                g ^= 1;
                store_row<C3, S>(dl, sb + (long long)y * w + x0, P, n);
                if (more) {
#pragma unroll
                    for (int s = 0; s < S; s++) {
                        C3 c = next_down ? closer(C[s], add(Q[s], 0, 0, dz)) : C[s];
                        V[s] = closer(c, add(P[s], 0, dyn, 0));
                    }
                }
            }
        }
    }
}

// ---- by a warp -----------------------------------------------------------------------
// Rows of at most 32 S cells: every exchange a shuffle, no shared memory and no
// barrier (row_pass_warp).  Same steps and candidate order.

template <int S>
__device__ __forceinline__ void danielsson2_warp(uint32_t* __restrict__ dl, int w, int h, int cw)
{
    const int lane = threadIdx.x & 31;
    const int nseg = (w + S - 1) / S;
    const bool active = lane < nseg;
    const int n = active ? min(S, w - lane * S) : 0;
    const long long x0 = (long long)lane * S;
    if (h < 2) return;
    const int steps = 2 * (h - 1);
    auto row_of = [&](int i) { return i < h - 1 ? i + 1 : 2 * h - 3 - i; };
    auto dy_of = [&](int i) { return i < h - 1 ? -cw : cw; };
    C2 P[S], C[S], V[S], R[S], D[S];
#pragma unroll
    for (int s = 0; s < S; s++) P[s] = C[s] = V[s] = R[s] = D[s] = C2{0, 0};
    load_row<C2, S>(P, dl, x0, n);
    load_row<C2, S>(C, dl, (long long)row_of(0) * w + x0, n);
#pragma unroll
    for (int s = 0; s < S; s++) V[s] = closer(C[s], add(P[s], 0, dy_of(0)));
    for (int i = 0; i < steps; i++) {
        const int y = row_of(i);
        const bool more = i + 1 < steps;
        if (more) load_row<C2, S>(C, dl, (long long)row_of(i + 1) * w + x0, n);
        row_pass_warp<C2, S, false, +1>(R, V, lane, nseg, n, cw, D, warp_round0_input<C2, S, +1>(V, n, lane));
        row_pass_warp<C2, S, false, -1>(P, R, lane, nseg, n, cw, D, warp_round0_input<C2, S, -1>(R, n, lane));
        store_row<C2, S>(dl, (long long)y * w + x0, P, n);
        if (more) {
            const int dyn = dy_of(i + 1);
#pragma unroll
            for (int s = 0; s < S; s++) V[s] = closer(C[s], add(P[s], 0, dyn));
        }
    }
}

template <int S>
__device__ __forceinline__ void danielsson3_warp(int16_t* __restrict__ dl, int w, int h, int d, int cw)
{
    const int lane = threadIdx.x & 31;
    const int nseg = (w + S - 1) / S;
    const bool active = lane < nseg;
    const int n = active ? min(S, w - lane * S) : 0;
    const long long x0 = (long long)lane * S;
    const long long plane = (long long)w * h;
    const int steps = 2 * (h - 1);
    auto row_of = [&](int i) { return i < h - 1 ? i + 1 : 2 * h - 3 - i; };
    auto dy_of = [&](int i) { return i < h - 1 ? -cw : cw; };
    C3 P[S], C[S], Q[S], V[S], R[S], D[S];
#pragma unroll
    for (int s = 0; s < S; s++) P[s] = C[s] = Q[s] = V[s] = R[s] = D[s] = C3{0, 0, 0};
    for (int pass = 0; pass < 2; pass++) {
        const int dz = pass == 0 ? -cw : +cw;
        for (int k = 1; k < d; k++) {
            const int z = pass == 0 ? k : d - 1 - k;
            const int zp = pass == 0 ? z - 1 : z + 1;
            const long long sb = z * plane, pb = (long long)zp * plane;
            load_row<C3, S>(C, dl, sb + x0, n);
            load_row<C3, S>(Q, dl, pb + x0, n);
#pragma unroll
            for (int s = 0; s < S; s++) P[s] = closer(C[s], add(Q[s], 0, 0, dz));
            store_row<C3, S>(dl, sb + x0, P, n);
            if (h < 2) continue;
            load_row<C3, S>(C, dl, sb + (long long)w + x0, n);
            load_row<C3, S>(Q, dl, pb + (long long)w + x0, n);
#pragma unroll
            for (int s = 0; s < S; s++) V[s] = closer(closer(C[s], add(Q[s], 0, 0, dz)), add(P[s], 0, -cw, 0));
            for (int i = 0; i < steps; i++) {
                const int y = row_of(i);
                const bool more = i + 1 < steps;
                const bool next_down = more && i + 1 < h - 1;
                if (more) {
                    const long long off = (long long)row_of(i + 1) * w + x0;
                    load_row<C3, S>(C, dl, sb + off, n);
                    if (next_down) load_row<C3, S>(Q, dl, pb + off, n);
                }
                row_pass_warp<C3, S, false, +1>(R, V, lane, nseg, n, cw, D, warp_round0_input<C3, S, +1>(V, n, lane));
                row_pass_warp<C3, S, false, -1>(P, R, lane, nseg, n, cw, D, warp_round0_input<C3, S, -1>(R, n, lane));
                store_row<C3, S>(dl, sb + (long long)y * w + x0, P, n);
                if (more) {
                    const int dyn = dy_of(i + 1);
#pragma unroll
                    for (int s = 0; s < S; s++) {
                        C3 c = next_down ? closer(C[s], add(Q[s], 0, 0, dz)) : C[s];
                        V[s] = closer(c, add(P[s], 0, dyn, 0));
                    }
                }
            }
        }
    }
}

}  // namespace dolk
