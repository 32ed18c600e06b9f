// k_sweep.cu -- Danielsson and FastSweep, exact.
//
// Danielsson (DistanceOcclusionLib.cpp:702-778 2D, :2264-2394 3D) and FastSweep
// 2D (:633-697) are serial in the sweep axis: every row needs the whole
// previous row.  One group of warps walks the rows of an image (or the slices
// and rows of a volume); a lane keeps S consecutive cells of the row in
// registers, so the vertical (and z) pulls are lane-local and only the x
// passes talk across lanes (row.cuh, exact).  The next row is loaded while the
// current one is scanned.  A row of up to 256 cells is one warp's (nothing
// crosses a barrier), wider rows take one warp per 256 cells.
//
// FastSweep 3D (:2186-2260) runs in k_fastsweep3.cu; here are the forms that need
// little scratch.  Row (y, z) of an octant sweep needs only row (y-1, z) and row
// (y, z-1) of the same sweep, so rows on an anti-diagonal y+z = c are independent.  k_fastsweep3 runs one octant per
// launch with persistent CTAs that claim rows in anti-diagonal order from an
// atomic counter and wait (bounded) on per-row ready flags.  A row is only
// claimed by a running CTA and every row it waits on was claimed earlier, so
// the earliest unfinished row can always proceed.
#include <limits.h>

#include "dan_scan.cuh"
#include "dan_serial.cuh"
#include "dan_slices.cuh"
#include "diagonals.h"
#include "kernels.h"

namespace dolk {

// ---------------------------------------------------------------- helpers ----

// L2-coherent loads for rows written by other CTAs of the same launch
__device__ __forceinline__ C3 cell_load_cg(const int16_t* p, long long i)
{
    const int16_t* c = p + 3 * i;
    return C3{__ldcg(c), __ldcg(c + 1), __ldcg(c + 2)};
}

// ------------------------------------------------------------ Danielsson ----

template <int DIM, int S, int NW>
__global__ void __launch_bounds__(32 * NW) k_dan_serial(void* __restrict__ dl, int w, int h, int d, int cw)
{
    extern __shared__ __align__(16) unsigned char strips[];
    __shared__ RowShared<NW> sh;
    if constexpr (NW > 1) {
        if (threadIdx.x == 0) sh.bar = 0;
        __syncthreads();
    }
    dan_serial<DIM, S, NW>(dl, w, h, d, cw, strips + (NW > 1 ? threadIdx.x >> 5 : 0) * SerialIO<DIM, S>::kBytes, sh);
}

// ------------------------------------------------------------- FastSweep 2D ----
// Four quadrant sweeps; the first row of each sweep is left as is; each later
// row takes the previous row's cell, then along x the previous cell of the row
// and the diagonal cell of the previous row, in that order (:655-693).  The
// diagonal candidate of a lane's first cell is its predecessor's edge cell of
// the previous row: a shuffle inside the warp, shared memory across warps.

template <int S, int NW, int DX>
__device__ __forceinline__ void fastsweep2_sweep(const Field<2, S>& f, const SerialIO<2, S>& io, int dy, int cw,
                                                 RowShared<NW>& sh, int& par, uint32_t (*edge)[NW])
{
    using Row = Cells<2, S>;
    const int lane = threadIdx.x & 31, wi = NW > 1 ? threadIdx.x >> 5 : 0;
    const int ox = -cw * DX, oy = -cw * dy;
    const int y0 = dy > 0 ? 0 : f.h - 1;
    const int x0 = f.xw + lane * S;
    Row P, V;
    Diag<S> D;
    constexpr int rc = 0;   // strip of the next row
    __syncwarp();   // the previous sweep's last rows are stored
    io.fetch(rc, f.row(0, y0), f.lo, f.hi);
    io.cells_of(P, rc, f.row(0, y0), cw);
    io.fetch(rc, f.row(0, y0 + dy), f.lo, f.hi);
    for (int j = 1; j < f.h; j++) {
        const int y = y0 + j * dy;
        io.cells_of(V, rc, f.row(0, y), cw);
        if (j + 1 < f.h) io.fetch(rc, f.row(0, y + dy), f.lo, f.hi);
        // the previous row's cell before this lane's first in scan order
        const uint32_t mine = P.xy[DX > 0 ? S - 1 : 0];
        uint32_t before = __shfl_sync(0xFFFFFFFFu, mine, DX > 0 ? (lane + 31) & 31 : (lane + 1) & 31);
        if constexpr (NW > 1) {
            if (lane == (DX > 0 ? 31 : 0)) edge[j & 1][wi] = mine;
            __syncthreads();
            const int pw = wi - DX;
            if (lane == (DX > 0 ? 0 : 31) && pw >= 0 && pw < NW) before = edge[j & 1][pw];
        }
#pragma unroll
        for (int s = 0; s < S; s++) {
            const uint32_t from = DX > 0 ? (s > 0 ? P.xy[s > 0 ? s - 1 : 0] : before)
                                         : (s + 1 < S ? P.xy[s + 1 < S ? s + 1 : s] : before);
            D.xy[s] = y_shift(from + ((uint32_t)ox << 16), oy);
            D.W[s] = w_of<2>(D.xy[s], 0);
            const bool has = DX > 0 ? x0 + s > 0 : x0 + s < f.w - 1;
            D.L[s] = has ? len_of(D.xy[s], D.W[s]) : INT_MAX;
        }
        merge_y<2, S>(P, V, oy);
        row_pass_w<2, S, NW, DX, Diag<S>>(P, D, cw, sh, par, chain_none(cw));
        io.put_cells(f.row(0, y), P);
    }
}

template <int S, int NW>
__global__ void __launch_bounds__(32 * NW) k_fastsweep2(void* __restrict__ dl, int w, int h, int cw)
{
    extern __shared__ __align__(16) unsigned char strips[];
    __shared__ RowShared<NW> sh;
    __shared__ uint32_t edge[2][NW];
    if (h < 2) return;
    if constexpr (NW > 1) {
        if (threadIdx.x == 0) sh.bar = 0;
        __syncthreads();
    }
    const int wi = NW > 1 ? threadIdx.x >> 5 : 0;
    Field<2, S> f;
    f.lo = static_cast<unsigned char*>(dl);
    f.hi = f.lo + (long long)w * h * 4;
    f.w = w;
    f.h = h;
    f.xw = wi * 32 * S;
    const SerialIO<2, S> io{strips + wi * SerialIO<2, S>::kBytes, min(32 * S, w - f.xw)};
    int par = 0;
    for (int sweep = 0; sweep < 4; sweep++) {
        const int dy = (sweep & 2) ? -1 : 1;
        if (sweep & 1)
            fastsweep2_sweep<S, NW, -1>(f, io, dy, cw, sh, par, edge);
        else
            fastsweep2_sweep<S, NW, +1>(f, io, dy, cw, sh, par, edge);
        __syncthreads();   // the edge slots are reused
    }
}

// ------------------------------------------------------------- FastSweep 3D ----

template <int S>
__global__ void __launch_bounds__(256) k_fastsweep3(int16_t* __restrict__ dl, int w, int h, int d, int cw, int sweep,
                                                    int* __restrict__ flags, int* __restrict__ counter,
                                                    const int* __restrict__ diag_start, int* __restrict__ err,
                                                    int epoch, int wait_epoch, unsigned wait_limit)
{
    __shared__ ScanShared<C3> sh;
    __shared__ long long s_item;
    __shared__ int s_c;
    const int t = threadIdx.x;
    const int nseg = (w + S - 1) / S;
    const bool active = t < nseg;
    const int n = active ? min(S, w - t * S) : 0;
    const long long x0 = (long long)t * S;
    const long long plane = (long long)w * h;
    const int dx = (sweep & 1) ? -1 : 1, dy = (sweep & 2) ? -1 : 1, dz = (sweep & 4) ? -1 : 1;
    const int oy = -cw * dy, oz = -cw * dz;
    const int yb = dy > 0 ? 0 : h - 1, zb = dz > 0 ? 0 : d - 1;
    const int H = h - 1, Dd = d - 1;
    const long long total = (long long)H * Dd;
    const int pred = t - dx;
    const bool has_pred = active && pred >= 0 && pred < nseg;
    C3 C[S], Zp[S], Yp[S], V[S], R[S], D[S];
#pragma unroll
    for (int s = 0; s < S; s++) C[s] = Zp[s] = Yp[s] = V[s] = R[s] = D[s] = C3{0, 0, 0};

    // anti-diagonal c = jj + kk (jj: rows after the first, kk: slices after
    // the first) of the item: the last c with diag_start[c] <= item.  A CTA
    // claims items in increasing order, so its c only moves forward (thread 0
    // keeps it; a few cached loads per item instead of a binary search).  A
    // row is claimed only when the CTA is free to run it: claiming the next
    // one early parks rows of the wavefront behind another row's work
    // (measured 15.2 -> 24.0 ms at 256^3).
    int c_cur = 2;
    for (;;) {
        if (t == 0) {
            const long long it = atomicAdd(counter, 1);
            if (it < total)
                while (c_cur < H + Dd && diag_start[c_cur + 1] <= it) c_cur++;
            s_item = it;
            s_c = c_cur;
        }
        __syncthreads();
        const long long item = s_item;
        const int c = s_c;
        __syncthreads();
        if (item >= total) break;
        const int jj = max(1, c - Dd) + (int)(item - diag_start[c]);
        const int kk = c - jj;
        const int y = yb + jj * dy, z = zb + kk * dz;
        const int yprev = y - dy, zprev = z - dz;

        if (t == 0) {
            // wait (bounded) until both neighbour rows of this sweep are done
            const int* fa = jj > 1 ? flags + (long long)z * h + yprev : nullptr;
            const int* fb = kk > 1 ? flags + (long long)zprev * h + y : nullptr;
            // (wait_epoch is epoch except under a test hook that makes it unreachable)
            for (unsigned it = 0;; it++) {
                bool ok = (!fa || *((volatile const int*)fa) >= wait_epoch) &&
                          (!fb || *((volatile const int*)fb) >= wait_epoch);
                if (ok) break;
                if (it >= wait_limit) { atomicExch(err, 1); break; }
                __nanosleep(128);
            }
            __threadfence();
        }
        __syncthreads();

        const long long rb = z * plane + (long long)y * w + x0;
        const long long zb_ = (long long)zprev * plane + (long long)y * w + x0;
        const long long yb_ = z * plane + (long long)yprev * w + x0;
#pragma unroll
        for (int s = 0; s < S; s++)
            if (s < n) {
                C[s] = cell_load_cg(dl, rb + s);
                Zp[s] = cell_load_cg(dl, zb_ + s);
                Yp[s] = cell_load_cg(dl, yb_ + s);
                V[s] = closer(closer(C[s], add(Zp[s], 0, 0, oz)), add(Yp[s], 0, oy, 0));
            }
        if (active) sh.guess[0][t] = dx > 0 ? seg_edge<C3, S, +1>(V, n) : seg_edge<C3, S, -1>(V, n);
        __syncthreads();
        const C3 in0 = has_pred ? sh.guess[0][pred] : V[0];
        auto nopost = [](const C3 (&)[S]) {};
        if (dx > 0)
            row_pass<C3, S, false, +1>(R, V, t, nseg, n, cw, sh, D, in0, nopost);
        else
            row_pass<C3, S, false, -1>(R, V, t, nseg, n, cw, sh, D, in0, nopost);
        store_row<C3, S>(dl, rb, R, n);
        __threadfence();
        __syncthreads();
        if (t == 0) atomicExch(flags + (long long)z * h + y, epoch);
    }
}

// diag[c]: the rows of anti-diagonals before c = jj + kk (jj in 1 .. H, kk in 1 .. D),
// that is, the sum of min(D, c - 1 - jj) over jj in 1 .. min(H, c - 2).  (On the
// device: a table copied from the host would have to outlive the copy, and a
// captured graph.)
__global__ void k_fastsweep3_diagonals(int* __restrict__ diag, int H, int D, int nd)
{
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nd) return;
    diag[c] = rows_before_diagonal(H, D, c);
}

// Slice pipeline: a CTA claims a slice kk (in sweep order,
// from an atomic counter) and walks its rows jj = 1 .. H in order, so the
// row before (y - dy, same slice) is the CTA's own previous result, kept in
// registers; only the slice before (z - dz, same row) comes from another
// CTA, through its per-row flag.  Along y a step costs one row's work, along
// z one row's work plus the hand-over (the producer's fence and flag, the
// poll, the load), where the anti-diagonal wavefront above pays the
// hand-over on every step (256^3 shapes: 11.7 against 15.2 ms).  A slice is
// claimed only by a running CTA and waits only on the slice claimed before
// it, so the earliest unfinished slice always proceeds.  A row's own cells
// are written by no other CTA of the sweep, so they are loaded before the
// wait (loading the next row's during the hand-over measured 3 % slower).
template <int S>
__global__ void __launch_bounds__(256) k_fastsweep3_slices(int16_t* __restrict__ dl, int w, int h, int d, int cw,
                                                           int sweep, int* __restrict__ flags,
                                                           int* __restrict__ counter, int* __restrict__ err,
                                                           int epoch, int wait_epoch, unsigned wait_limit)
{
    __shared__ ScanShared<C3> sh;
    __shared__ int s_slice;
    const int t = threadIdx.x;
    const int nseg = (w + S - 1) / S;
    const bool active = t < nseg;
    const int n = active ? min(S, w - t * S) : 0;
    const long long x0 = (long long)t * S;
    const long long plane = (long long)w * h;
    const int dx = (sweep & 1) ? -1 : 1, dy = (sweep & 2) ? -1 : 1, dz = (sweep & 4) ? -1 : 1;
    const int oy = -cw * dy, oz = -cw * dz;
    const int yb = dy > 0 ? 0 : h - 1, zb = dz > 0 ? 0 : d - 1;
    const int H = h - 1, Dd = d - 1;
    const int pred = t - dx;
    const bool has_pred = active && pred >= 0 && pred < nseg;
    C3 C[S], Zp[S], Yp[S], V[S], R[S], D[S];
#pragma unroll
    for (int s = 0; s < S; s++) C[s] = Zp[s] = Yp[s] = V[s] = R[s] = D[s] = C3{0, 0, 0};

    for (;;) {
        if (t == 0) s_slice = atomicAdd(counter, 1) + 1;
        __syncthreads();
        const int kk = s_slice;
        __syncthreads();
        if (kk > Dd) break;
        const int z = zb + kk * dz, zprev = z - dz;
        // the slice's first row is not updated by the sweep (:2208, :2214 start at 1)
#pragma unroll
        for (int s = 0; s < S; s++)
            if (s < n) Yp[s] = cell_load_cg(dl, z * plane + (long long)yb * w + x0 + s);
        for (int jj = 1; jj <= H; jj++) {
            const int y = yb + jj * dy;
            const long long rb = z * plane + (long long)y * w + x0;
#pragma unroll
            for (int s = 0; s < S; s++)
                if (s < n) C[s] = cell_load_cg(dl, rb + s);
            if (kk > 1 && t == 0) {
                // wait (bounded) until the slice before has done this row; the
                // poll is an acquire load, which with the barrier after it
                // orders the CTA's loads of that row after the producer's
                // stores (wait_epoch is epoch except under a test hook that
                // makes it unreachable)
                const int* fb = flags + (long long)zprev * h + y;
                for (unsigned it = 0;; it++) {
                    int f;
                    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(f) : "l"(fb) : "memory");
                    if (f >= wait_epoch) break;
                    if (it >= wait_limit) {
                        atomicExch(err, 1);
                        break;
                    }
                    __nanosleep(64);
                }
            }
            __syncthreads();
            const long long zb_ = (long long)zprev * plane + (long long)y * w + x0;
#pragma unroll
            for (int s = 0; s < S; s++)
                if (s < n) {
                    Zp[s] = cell_load_cg(dl, zb_ + s);
                    V[s] = closer(closer(C[s], add(Zp[s], 0, 0, oz)), add(Yp[s], 0, oy, 0));
                }
            if (active) sh.guess[0][t] = dx > 0 ? seg_edge<C3, S, +1>(V, n) : seg_edge<C3, S, -1>(V, n);
            __syncthreads();
            const C3 in0 = has_pred ? sh.guess[0][pred] : V[0];
            auto nopost = [](const C3 (&)[S]) {};
            if (dx > 0)
                row_pass<C3, S, false, +1>(R, V, t, nseg, n, cw, sh, D, in0, nopost);
            else
                row_pass<C3, S, false, -1>(R, V, t, nseg, n, cw, sh, D, in0, nopost);
            store_row<C3, S>(dl, rb, R, n);
#pragma unroll
            for (int s = 0; s < S; s++) Yp[s] = R[s];   // the next row's y neighbour
            // publish the row: after the barrier one thread's fence orders the
            // whole CTA's stores before the flag (the pattern of a grid
            // barrier); a thread of the second warp does it, so that thread 0
            // polls for the next row meanwhile and no other thread waits on a fence
            __syncthreads();
            if (t == (blockDim.x > 32 ? 32 : 0)) {
                __threadfence();
                atomicExch(flags + (long long)z * h + y, epoch);
            }
        }
    }
}

// --------------------------------------------------------------- launchers ----

// cells per thread: aim for at most 256 threads (fewer warps at every barrier),
// allow up to max_threads for wide rows; 0 when the row is too wide
static int pick_s(int w, int max_threads)
{
    const int options[] = {1, 2, 4, 8};
    for (int s : options)
        if ((w + s - 1) / s <= 256 && (w + s - 1) / s <= max_threads) return s;
    for (int s : options)
        if ((w + s - 1) / s <= max_threads) return s;
    return 0;
}

static int threads_for(int w, int s)
{
    int n = (w + s - 1) / s;
    return ((n + 31) / 32) * 32;
}

// Cells per lane and warps of a row: 256 cells per warp, fewer per lane for rows
// that one warp holds with fewer.  Tuning values 4 and 8 set the cells per lane
// (any other: this rule).
static void row_shape(int kind, int w, int* s, int* nw)
{
    const int tv = tune_get(kind, w);
    *s = tv == 4 || tv == 8 ? tv : (w <= 64 ? 2 : (w <= 128 ? 4 : 8));
    if (*s < 8 && w > 32 * *s * 16) *s = 8;
    if (w <= 32 && tv != 4 && tv != 8) *s = 1;
    const int need = (w + 32 * *s - 1) / (32 * *s);
    *nw = 1;
    while (*nw < need) *nw *= 2;
}

// every shape row_shape gives up to 4096 cells, f(S, NW), but for the narrow rows
// (1, 1) and (2, 1): images' alone, of 32 and 64 cells (Danielsson) and 33 to 64
// (FastSweep); k_scan.cu has the others
#define DOL_ROW_SHAPES(f) \
    f(4, 1) f(4, 2) f(4, 4) f(4, 8) f(4, 16) f(8, 1) f(8, 2) f(8, 4) f(8, 8) f(8, 16)

void launch_danielsson(int dim, void* deltas, int w, int h, int d, int cw, cudaStream_t st)
{
    int s, nw;
    row_shape(dim == 2 ? kTuneDan2 : kTuneDan3, w, &s, &nw);
    ProfScope ps("danielsson", st);
    const int tv = tune_get(dim == 2 ? kTuneDan2 : kTuneDan3, w);
    if (tv != 4 && tv != 8 && launch_danielsson_scan(dim, deltas, w, h, dim == 2 ? 1 : d, cw, st)) return;
    auto run = [&](auto kern, int warps, size_t strips) {
        if (strips > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)strips);
        kern<<<1, 32 * warps, strips, st>>>(deltas, w, h, dim == 2 ? 1 : d, cw);
    };
#define DOL_DAN_CASE(SV, NWV)                                                          \
    if (s == SV && nw == NWV) {                                                        \
        if (dim == 2)                                                                  \
            run(k_dan_serial<2, SV, NWV>, NWV, NWV * SerialIO<2, SV>::kBytes);         \
        else                                                                           \
            run(k_dan_serial<3, SV, NWV>, NWV, NWV * SerialIO<3, SV>::kBytes);         \
    }
    DOL_ROW_SHAPES(DOL_DAN_CASE)
#undef DOL_DAN_CASE
    if (s == 2) run(k_dan_serial<2, 2, 1>, 1, SerialIO<2, 2>::kBytes);
    if (s == 1) run(k_dan_serial<2, 1, 1>, 1, SerialIO<2, 1>::kBytes);
}

void launch_fastsweep_2d(void* deltas, int w, int h, int cw, cudaStream_t st)
{
    int s, nw;
    row_shape(kTuneFs2, w, &s, &nw);
    ProfScope ps("fastsweep_2d", st);
    const int tv = tune_get(kTuneFs2, w);
    if (tv != 4 && tv != 8 && launch_fastsweep_2d_scan(deltas, w, h, cw, st)) return;
#define DOL_FS_CASE(SV, NWV) \
    if (s == SV && nw == NWV)  \
        k_fastsweep2<SV, NWV><<<1, 32 * NWV, NWV * SerialIO<2, SV>::kBytes, st>>>(deltas, w, h, cw);
    DOL_ROW_SHAPES(DOL_FS_CASE)
    DOL_FS_CASE(2, 1)
#undef DOL_FS_CASE
}

size_t fastsweep3_workspace_bytes(int w, int h, int d)
{
    const size_t columns = fastsweep3_columns_bytes(w, h, d), rows = fastsweep3_workspace_bytes_min(w, h, d);
    return columns > rows ? columns : rows;
}

size_t fastsweep3_workspace_bytes_min(int w, int h, int d)
{
    (void)w;
    size_t flags = (size_t)h * d * sizeof(int);
    size_t diag = (size_t)(h + d + 2) * sizeof(int);
    return ((flags + 255) & ~(size_t)255) + ((diag + 255) & ~(size_t)255) + 256;
}

void launch_fastsweep_3d(void* deltas, int w, int h, int d, int cw, void* ws, size_t ws_bytes, int* err,
                         cudaStream_t st)
{
    if (h < 2 || d < 2) return;   // no row is ever updated (:2208, :2214 start at 1)
    if (launch_fastsweep_3d_columns(deltas, w, h, d, cw, ws, ws_bytes, err, st)) return;
    cudaGetLastError();
    char* p = static_cast<char*>(ws);
    int* flags = reinterpret_cast<int*>(p);
    p += (((size_t)h * d * sizeof(int)) + 255) & ~(size_t)255;
    int* diag = reinterpret_cast<int*>(p);
    p += (((size_t)(h + d + 2) * sizeof(int)) + 255) & ~(size_t)255;
    int* counters = reinterpret_cast<int*>(p);   // 8 ints

    const int H = h - 1, Dd = d - 1;
    cudaMemsetAsync(flags, 0, (size_t)h * d * sizeof(int), st);
    cudaMemsetAsync(counters, 0, 8 * sizeof(int), st);

    // cells per thread: tuned, else rows of at most 128 threads (more CTAs
    // per SM along the wavefront; 256^3 shapes: 15.1 ms at 128 threads, 22.0
    // at 256), else at most 256
    int s = tune_get(kTuneFs3, w);
    const bool wavefront = s < 0;   // negative tuned values: the anti-diagonal wavefront with -s cells per thread
    if (wavefront) {
        s = -s;
        const int nd = H + Dd + 2;
        k_fastsweep3_diagonals<<<(nd + 255) / 256, 256, 0, st>>>(diag, H, Dd, nd);
    }
    if (!((s == 1 || s == 2 || s == 4 || s == 8) && (w + s - 1) / s <= 256)) {
        s = pick_s(w, 128);
        if (!s) s = pick_s(w, 256);
    }
    const int T = threads_for(w, s);
    const WaitHooks hooks = wait_hooks();
    ProfScope ps("fastsweep_3d", st);
#define DOL_FS3_CASE(SV)                                                                                     \
    case SV: {                                                                                               \
        if (!wavefront) {                                                                                    \
            int per_sm = 0;                                                                                  \
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_fastsweep3_slices<SV>, T, 0);           \
            if (per_sm < 1) per_sm = 1;                                                                      \
            long long grid = (long long)per_sm * g_num_sms;                                                  \
            if (grid > Dd) grid = Dd;                                                                        \
            for (int sw = 0; sw < 8; sw++)                                                                   \
                k_fastsweep3_slices<SV><<<(int)grid, T, 0, st>>>(static_cast<int16_t*>(deltas), w, h, d, cw,  \
                                                                 sw, flags, counters + sw, err, sw + 1,       \
                                                                 sw == hooks.stall_sweep ? INT_MAX : sw + 1,  \
                                                                 hooks.limit);                                \
            break;                                                                                           \
        }                                                                                                    \
        int per_sm = 0;                                                                                      \
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_fastsweep3<SV>, T, 0);                      \
        if (per_sm < 1) per_sm = 1;                                                                          \
        long long rows = (long long)H * Dd;                                                                  \
        long long grid = (long long)per_sm * g_num_sms;                                                      \
        if (grid > rows) grid = rows;                                                                        \
        for (int sw = 0; sw < 8; sw++)                                                                       \
            k_fastsweep3<SV><<<(int)grid, T, 0, st>>>(static_cast<int16_t*>(deltas), w, h, d, cw, sw, flags,  \
                                                      counters + sw, diag, err, sw + 1,                       \
                                                      sw == hooks.stall_sweep ? INT_MAX : sw + 1,             \
                                                      hooks.limit);                                           \
    } break;
    switch (s) {
        DOL_FS3_CASE(1)
        DOL_FS3_CASE(2)
        DOL_FS3_CASE(4)
        DOL_FS3_CASE(8)
        default: break;
    }
#undef DOL_FS3_CASE
}

}  // namespace dolk

// ------------------------------------------------------------- batched SDF ----
// Thousands of independent masks and volumes in one persistent launch: each
// CTA pulls the next item (largest first) from an atomic counter and runs the
// whole signed pipeline on it -- border initialisation, Danielsson with cw = 2,
// signed distances -- with the same per-CTA code as the single-item kernels,
// so every item's output is bit-identical to a per-item call.
#include "border.cuh"

namespace dolk {

struct BatchItemDev {
    int w, h, d, pad;
    long long mask_off;    // words
    long long delta_off;   // bytes
    long long dist_off;    // floats, < 0: none
};

// Border initialisation and signed distances of an item by `nu` warps, this
// being warp u of them.  A warp takes 32 mask words at a time: lane q forms the
// bit planes of word q, then all lanes write one word's 32 cells after the
// other, so that stores run along the row.
template <int DIM>
__device__ __forceinline__ void border_warps(const uint32_t* mask, void* dl, int w, int h, int d, int u, int nu)
{
    const int lane = threadIdx.x & 31;
    const int ws = words_per_row(w);
    const long long words = (long long)ws * h * d;
    for (long long base = 32 * u; base < words; base += 32 * nu) {
        const long long wid = min(base + lane, words - 1);
        const long long row = wid / ws;
        const int k = (int)(wid - row * ws);
        long long first;
        int live;
        word_cells(wid, w, ws, &first, &live);
        uint32_t pl[7];
        if (DIM == 2) {
            const Planes2 p = border2_word(w, h, mask, (int)row, k);
            pl[0] = p.mx; pl[1] = p.xn; pl[2] = p.xs; pl[3] = p.yn; pl[4] = p.ys; pl[5] = pl[6] = 0;
        } else {
            const int z = (int)(row / h);
            const Planes3 p = border3_word(w, h, d, mask, z, (int)(row - (long long)z * h), k);
            pl[0] = p.mx; pl[1] = p.xn; pl[2] = p.xs; pl[3] = p.yn; pl[4] = p.ys; pl[5] = p.zn; pl[6] = p.zs;
        }
        const int n = (int)min(32LL, words - base);
        for (int q = 0; q < n; q++) {
            uint32_t b[7];
#pragma unroll
            for (int i = 0; i < (DIM == 2 ? 5 : 7); i++) b[i] = __shfl_sync(0xFFFFFFFFu, pl[i], q);
            const long long at = __shfl_sync(0xFFFFFFFFu, first, q) + lane;
            const int nq = __shfl_sync(0xFFFFFFFFu, live, q);
            if (lane < nq) {
                if (DIM == 2)
                    static_cast<uint32_t*>(dl)[at] = pack2(decode2(Planes2{b[0], b[1], b[2], b[3], b[4]}, lane));
                else
                    cell_store(static_cast<int16_t*>(dl), at,
                               decode3(Planes3{b[0], b[1], b[2], b[3], b[4], b[5], b[6]}, lane));
            }
        }
    }
}

template <class Cell, class P>
__device__ __forceinline__ void signed_dist_warps(const uint32_t* mask, const P* dl, float* out, int w, long long rows, int u,
                                                  int nu)
{
    const int lane = threadIdx.x & 31;
    const int ws = words_per_row(w);
    // rows of up to 16 cells: several at a time (2000 images of 2 x 400 1.19 ms row by
    // row, 0.89); four loads in flight (2000 images of 100 x 100 1.01 -> 0.84 ms)
    const int per = w <= 16 ? 32 / w : 1, sub = w <= 16 ? lane / w : 0;
    if (sub >= per) return;
    for (long long row = (long long)u * per + sub; row < rows; row += (long long)nu * per) {
        const long long first = row * w;
        for (int x0 = lane - sub * w; x0 < w; x0 += 128) {   // four cells in flight
            int l[4];
#pragma unroll
            for (int q = 0; q < 4; q++) l[q] = x0 + 32 * q < w ? (int)len(cell_load(dl, first + x0 + 32 * q)) : 0;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int x = x0 + 32 * q;
                if (x >= w) break;
                float r = __fdiv_rn(sqrtf((float)l[q]), 2.0f);
                if ((mask[row * ws + (x >> 5)] >> (x & 31)) & 1u) r = -r;
                out[first + x] = r;
            }
        }
    }
}

// Danielsson of one field by one warp: rows of at most 256 cells
template <int DIM>
__device__ __noinline__ void batch_dan_warp(void* dl, int w, int h, int d, unsigned char* strip)
{
    RowShared<1> none;
    if constexpr (DIM == 2) {   // (as single images: k_scan.cu)
        if (w < 32) return danielsson2_warp<1>(static_cast<uint32_t*>(dl), w, h, 2);
        if (w > 32 && w < 64) return danielsson2_warp<2>(static_cast<uint32_t*>(dl), w, h, 2);
    } else {
        if (w <= 32) return danielsson3_warp<1>(static_cast<int16_t*>(dl), w, h, d, 2);
        if (w <= 64) return danielsson3_warp<2>(static_cast<int16_t*>(dl), w, h, d, 2);
        if (w < 128) return danielsson3_warp<4>(static_cast<int16_t*>(dl), w, h, d, 2);
    }
    if (w <= 64) dan_serial<DIM, 2, 1>(dl, w, h, d, 2, strip, none);
    else if (w <= 128) dan_serial<DIM, 4, 1>(dl, w, h, d, 2, strip, none);
    else dan_serial<DIM, 8, 1>(dl, w, h, d, 2, strip, none);
}
// by a group of 4 warps: rows of at most 1024 cells
template <int DIM, int S>
__device__ __noinline__ void batch_dan_group(void* dl, int w, int h, int d, unsigned char* strip, RowShared<4>& sh)
{
    dan_serial<DIM, S, 4>(dl, w, h, d, 2, strip, sh);
}
// a volume by the whole CTA: rows of at most 128 cells, as many as fit in shared memory
template <int S, int NW>
__device__ __noinline__ void batch_dan_slices(void* dl, int w, int h, int d, unsigned char* smem)
{
    dan_slices<S, NW>(dl, w, h, d, 2, smem);
}

// an image processed by one warp
__device__ __noinline__ void batch_item_warp(const BatchItemDev& b, const uint32_t* masks, unsigned char* deltas,
                                             float* dist, unsigned char* strip)
{
    const uint32_t* m = masks + b.mask_off;
    uint32_t* dl = reinterpret_cast<uint32_t*>(deltas + b.delta_off);
    border_warps<2>(m, dl, b.w, b.h, 1, 0, 1);
    __syncwarp();
    batch_dan_warp<2>(dl, b.w, b.h, 1, strip);
    __syncwarp();
    if (dist && b.dist_off >= 0) signed_dist_warps<C2>(m, dl, dist + b.dist_off, b.w, b.h, 0, 1);
}

// Two queues.  Queue A (order[0 .. nv)) holds the volumes whose rows fit one
// warp (up to 256 cells), longest chain first; queue B (order[nv .. n)) the
// items with rows over 256 cells, then the narrow images.  A CTA (one per SM)
// takes queue A items while there are any, the slices' rows in parallel chunks
// (dan_slices.cuh), or, where a slice does not fit in shared memory, warp 0
// walking it serially.  Then it turns to queue B; items with wide rows come
// first, the first narrow image drawn switches to per-warp draining.
//   * up to kBatchFew items per CTA: 8 warps take one wide item at a time, 4 cells
//     per thread (2.7 us a row step: a wide image is a chain of steps, and the
//     largest ones decide when the batch ends; 200 volumes of 300 x 40 x 40 24.6 ms,
//     34.0 by 4 of the warps);
//   * more: each group of 4 warps takes items by itself (its own barrier), 11 us
//     a step but four images at a time.
// Milliseconds, 8 warps | groups (images only, sides up to 1024 x 2047): 16 images
// 5.3 | 8.1 (5.6 with 256 threads per item and as many CTAs as fit), 200 15 | 32
// (16.4), 900 16 | 42 (17.9), 2000 37 | 43 (39), 4096 71 | 50 (75); 16 warps per
// item: 20 at 200, 93 at 4096.  4096 images and 64 volumes: 98 ms with every
// volume walked serially by one warp, 55 ms.
// counter: [0] queue B, [1] queue A, [2] nv (written by dol_batch_prepare).
constexpr size_t kBatchSmem = 216 * 1024;
constexpr int kBatchFew = 16;
constexpr int kBatchStrip = (int)SerialIO<3, 8>::kBytes;   // a warp's strips in queue B, the widest

// an image with rows of at most 1024 cells by 8 warps, 4 cells per thread
__device__ __noinline__ void batch_dan_image(uint32_t* dl, int w, int h, ScanShared<C2>& sh)
{
    danielsson2_cta<4>(dl, w, h, 2, sh);
}

// a volume likewise
__device__ __noinline__ void batch_dan_volume(int16_t* dl, int w, int h, int d, ScanShared<C3>& sh)
{
    danielsson3_cta<4>(dl, w, h, d, 2, sh);
}

// an item of queue B with rows of more than 256 cells, by the CTA's 8 warps
__device__ __noinline__ void batch_item_cta(const BatchItemDev& b, const uint32_t* masks, unsigned char* deltas, float* dist,
                                            unsigned char* smem)
{
    const int warp = threadIdx.x >> 5;
    const uint32_t* m = masks + b.mask_off;
    void* dl = deltas + b.delta_off;
    if (b.d <= 1) {
        border_warps<2>(m, dl, b.w, b.h, 1, warp, 8);
        __syncthreads();
        batch_dan_image(static_cast<uint32_t*>(dl), b.w, b.h, *reinterpret_cast<ScanShared<C2>*>(smem));
        __syncthreads();
        if (dist && b.dist_off >= 0)
            signed_dist_warps<C2>(m, static_cast<uint32_t*>(dl), dist + b.dist_off, b.w, b.h, warp, 8);
    } else {
        border_warps<3>(m, dl, b.w, b.h, b.d, warp, 8);
        __syncthreads();
        batch_dan_volume(static_cast<int16_t*>(dl), b.w, b.h, b.d, *reinterpret_cast<ScanShared<C3>*>(smem));
        __syncthreads();
        if (dist && b.dist_off >= 0)
            signed_dist_warps<C3>(m, static_cast<int16_t*>(dl), dist + b.dist_off, b.w, (long long)b.h * b.d, warp, 8);
    }
}

template <int NW>
__global__ void __launch_bounds__(32 * NW) k_batch_sdf(const BatchItemDev* __restrict__ items,
                                                       const int* __restrict__ order, int n,
                                                       const uint32_t* __restrict__ masks,
                                                       unsigned char* __restrict__ deltas, float* __restrict__ dist,
                                                       int* __restrict__ counter)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ RowShared<4> sh[NW / 4];
    __shared__ int s_item[NW / 4 + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nv = counter[2];
    for (;;) {
        if (threadIdx.x == 0) s_item[0] = atomicAdd(counter + 1, 1);
        __syncthreads();
        const int it = s_item[0];
        __syncthreads();
        if (it >= nv) break;
        const BatchItemDev b = items[order[it]];
        const uint32_t* m = masks + b.mask_off;
        int16_t* dl = reinterpret_cast<int16_t*>(deltas + b.delta_off);
        border_warps<3>(m, dl, b.w, b.h, b.d, warp, NW);
        __syncthreads();
        if (b.w <= 64 && SliceIO<2>::bytes(b.h, NW) <= kBatchSmem) batch_dan_slices<2, NW>(dl, b.w, b.h, b.d, smem);
        else if (b.w <= 128 && SliceIO<4>::bytes(b.h, NW) <= kBatchSmem)
            batch_dan_slices<4, NW>(dl, b.w, b.h, b.d, smem);
        else if (warp == 0) batch_dan_warp<3>(dl, b.w, b.h, b.d, smem);
        __syncthreads();
        if (dist && b.dist_off >= 0)
            signed_dist_warps<C3>(m, dl, dist + b.dist_off, b.w, (long long)b.h * b.d, warp, NW);
        __syncthreads();
    }
    unsigned char* strip = smem + warp * kBatchStrip;
    if (n - nv <= kBatchFew * (int)gridDim.x) {
        if (warp >= 8) return;   // (barriers count the threads that are left)
        for (;;) {
            __syncthreads();
            if (threadIdx.x == 0) s_item[0] = nv + atomicAdd(counter, 1);
            __syncthreads();
            const int it = s_item[0];
            if (it >= n) return;
            const BatchItemDev b = items[order[it]];
            if (b.w <= 256) {
                // narrow images from here on: the first warp takes this item, every warp then drains the queue
                int mine = warp == 0 ? it : -1;
                for (;;) {
                    if (mine < 0) {
                        int v = 0;
                        if (lane == 0) v = nv + atomicAdd(counter, 1);
                        mine = __shfl_sync(0xFFFFFFFFu, v, 0);
                        if (mine >= n) return;
                    }
                    batch_item_warp(items[order[mine]], masks, deltas, dist, strip);
                    mine = -1;
                }
            }
            batch_item_cta(b, masks, deltas, dist, smem);
        }
    }
    const int group = warp >> 2, gw = warp & 3;
    RowShared<4>& gsh = sh[group];
    if ((threadIdx.x & 127) == 0) gsh.bar = 1 + group;
    auto sync = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory"); };
    for (;;) {
        if ((threadIdx.x & 127) == 0) s_item[1 + group] = nv + atomicAdd(counter, 1);
        sync();
        const int it = s_item[1 + group];
        sync();
        if (it >= n) return;
        const BatchItemDev b = items[order[it]];
        if (b.w <= 256) {
            // narrow images from here on: the group's first warp takes this item, every warp then drains the queue
            int mine = gw == 0 ? it : -1;
            for (;;) {
                if (mine < 0) {
                    int v = 0;
                    if (lane == 0) v = nv + atomicAdd(counter, 1);
                    mine = __shfl_sync(0xFFFFFFFFu, v, 0);
                    if (mine >= n) return;
                }
                batch_item_warp(items[order[mine]], masks, deltas, dist, strip);
                mine = -1;
            }
        }
        const uint32_t* m = masks + b.mask_off;
        void* dl = deltas + b.delta_off;
        const long long rows = (long long)b.h * b.d;
        if (b.d <= 1) {
            border_warps<2>(m, dl, b.w, b.h, 1, gw, 4);
            sync();
            if (b.w <= 512) batch_dan_group<2, 4>(dl, b.w, b.h, 1, strip, gsh);
            else batch_dan_group<2, 8>(dl, b.w, b.h, 1, strip, gsh);
            sync();
            if (dist && b.dist_off >= 0)
                signed_dist_warps<C2>(m, static_cast<uint32_t*>(dl), dist + b.dist_off, b.w, rows, gw, 4);
        } else {
            border_warps<3>(m, dl, b.w, b.h, b.d, gw, 4);
            sync();
            if (b.w <= 512) batch_dan_group<3, 4>(dl, b.w, b.h, b.d, strip, gsh);
            else batch_dan_group<3, 8>(dl, b.w, b.h, b.d, strip, gsh);
            sync();
            if (dist && b.dist_off >= 0)
                signed_dist_warps<C3>(m, static_cast<int16_t*>(dl), dist + b.dist_off, b.w, rows, gw, 4);
        }
        sync();
    }
}

static_assert(sizeof(BatchItemDev) == 40, "batch item layout (dol_batch_item)");

void launch_batch_sdf(const void* items, const int* order, int n, const uint32_t* masks, void* deltas, float* dist,
                      int* counter, cudaStream_t st)
{
    ProfScope ps("batch_sdf", st);
    // 16 warps per CTA, or 8
    auto run = [&](auto kern, int warps) {
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBatchSmem);
        int per_sm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * warps, kBatchSmem);
        if (per_sm < 1) per_sm = 1;
        int grid = per_sm * g_num_sms;
        if (grid > n) grid = n;
        if (grid < 1) grid = 1;
        cudaMemsetAsync(counter, 0, 2 * sizeof(int), st);   // the queue heads; counter[2] (nv) stays
        kern<<<grid, 32 * warps, kBatchSmem, st>>>(static_cast<const BatchItemDev*>(items), order, n, masks,
                                                   static_cast<unsigned char*>(deltas), dist, counter);
    };
    if (tune_get(kTuneBatch, 1024) == 8)
        run(k_batch_sdf<8>, 8);
    else
        run(k_batch_sdf<16>, 16);
}

}  // namespace dolk
