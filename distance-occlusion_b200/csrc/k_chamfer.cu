// k_chamfer.cu -- Chamfer 3-4 distance propagation (Borgefors), as the
// reference's Chamfer (DistanceOcclusionLib.cpp:916-1016) on int16 / int32
// fields, plus the integer InitDistancesFromBitMask overloads (:183-222).
//
// The reference makes one raster pass down the rows and one back up.  On the
// way down, row y first takes min(v, above-left + 4, above + 3, above-right + 4)
// per cell (fewer neighbours at the row ends), then a left-to-right pass takes
// min(v, left + 3).  The second step is a prefix min-plus scan:
//     r[x] = min over j <= x of (u[j] + 3 (x - j)) = 3x + min over j <= x of (u[j] - 3j)
// so a row is one block-wide prefix min.  Every step is a min of exact integer
// sums, so the order of evaluation cannot change the result: int16 sums are
// done in int (as the reference's promotion does) and never wrap; int32 sums
// are done in 64 bits, which equals the reference as long as its own int32
// sums do not wrap (every input at most INT32_MAX - 4).  The way up mirrors it
// (suffix min, right neighbour).
//
// A CTA walks a run of rows (each row needs the one before); a thread owns 4
// consecutive cells, so rows of up to 4096 cells.  The previous row stays in
// registers, its neighbours across threads come by shuffle, across warps from
// the row's own scan, so a row costs one barrier.  Fields of more than a few rows
// (chamfer_block_rows) run in blocks of 8 rows, all blocks at once (see below);
// smaller ones, or when the small boundary scratch cannot be had, in one CTA.
#include <limits.h>

#include <type_traits>

#include "common.cuh"
#include "grid_barrier.cuh"
#include "kernels.h"

namespace dolk {

constexpr int kChamferCells = 4;

template <typename T>
struct ChamferKey {
    using K = int;
    static constexpr int kInf = 1 << 29;
};
template <>
struct ChamferKey<int32_t> {
    using K = long long;
    static constexpr long long kInf = 1LL << 62;
};

template <typename K>
__device__ __forceinline__ K shfl_up_k(K v, int o)
{
    return __shfl_up_sync(0xFFFFFFFFu, v, o);
}
template <typename K>
__device__ __forceinline__ K shfl_down_k(K v, int o)
{
    return __shfl_down_sync(0xFFFFFFFFu, v, o);
}

// The min over the lanes whose `on` holds
__device__ __forceinline__ int warp_min_k(int v, bool on) { return __reduce_min_sync(0xFFFFFFFFu, on ? v : INT_MAX); }
__device__ __forceinline__ long long warp_min_k(long long v, bool on)
{
    long long m = on ? v : LLONG_MAX;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = min(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
    return m;
}

// Inclusive scan of m over the thread's cells and the warp's lanes before it in
// scan direction (kFwd: lower lanes); returns the exclusive part.
template <typename K, bool kFwd>
__device__ __forceinline__ K warp_excl_min(K tot, K inf, K* incl_out)
{
    const int lane = threadIdx.x & 31;
    K incl = tot;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const K v = kFwd ? shfl_up_k(incl, o) : shfl_down_k(incl, o);
        if (kFwd ? lane >= o : lane + o < 32) incl = min(incl, v);
    }
    *incl_out = incl;
    const K excl = kFwd ? shfl_up_k(incl, 1) : shfl_down_k(incl, 1);
    return (kFwd ? lane == 0 : lane == 31) ? inf : excl;
}

// Shared words of a row's scan: per warp its total and the key of the cell that
// the warp on the other side of it needs, double-buffered by row parity
template <typename K>
struct ChamferShared {
    K tot[2][32];
    K edge[2][32];
};

// Rows ya, ya + dir, ..., yb of one pass (dir = +1 down, -1 up); one CTA, a
// thread per 4 consecutive cells.  `before`: the row before ya (null: none).
// kWrite: rows go back to dist.  `last`: receives the last row (null: not wanted).
template <typename T, bool kFwd, bool kWrite>
__device__ __forceinline__ void chamfer_rows(T* __restrict__ dist, int w, int ya, int yb,
                                             const typename ChamferKey<T>::K* before, typename ChamferKey<T>::K* last,
                                             ChamferShared<typename ChamferKey<T>::K>& sh)
{
    using K = typename ChamferKey<T>::K;
    constexpr K kInf = ChamferKey<T>::kInf;
    constexpr int C = kChamferCells;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int x0 = threadIdx.x * C;
    K r[C], re = kInf, le = kInf;   // the previous row's cells x0 .. x0+3, x0+4 and x0-1
#pragma unroll
    for (int c = 0; c < C; c++) r[c] = kInf;
    bool have = before != nullptr;
    if (have) {
#pragma unroll
        for (int c = 0; c < C; c++)
            if (x0 + c < w) r[c] = before[x0 + c];
        if (x0 > 0 && x0 <= w) le = before[x0 - 1];
        if (x0 + C < w) re = before[x0 + C];
    }
    const int dir = kFwd ? 1 : -1;
    K nv[C];
    auto fetch = [&](int y) {
#pragma unroll
        for (int c = 0; c < C; c++) nv[c] = x0 + c < w ? (K)dist[(long long)y * w + x0 + c] : kInf;
    };
    fetch(ya);
    int b = 0;
    __syncthreads();   // an earlier walk of this CTA may still read the shared words
    for (int y = ya;; y += dir, b ^= 1) {
        K m[C];
#pragma unroll
        for (int c = 0; c < C; c++) {
            K u = nv[c];
            if (have) u = min(u, min(min(c ? r[c - 1] : le, c < C - 1 ? r[c + 1] : re) + 4, r[c] + 3));
            m[c] = x0 + c < w ? (kFwd ? u - 3 * (K)(x0 + c) : u + 3 * (K)(x0 + c)) : kInf;
        }
        if (y != yb) fetch(y + dir);   // the next row's cells, while this one is scanned
        const K own_edge = kFwd ? m[0] : m[C - 1];
        if (kFwd) {
#pragma unroll
            for (int c = 1; c < C; c++) m[c] = min(m[c - 1], m[c]);
        } else {
#pragma unroll
            for (int c = C - 2; c >= 0; c--) m[c] = min(m[c + 1], m[c]);
        }
        K incl;
        const K excl = warp_excl_min<K, kFwd>(kFwd ? m[C - 1] : m[0], kInf, &incl);
        if (lane == (kFwd ? 31 : 0)) sh.tot[b][wid] = incl;
        if (lane == (kFwd ? 0 : 31)) sh.edge[b][wid] = own_edge;
        __syncthreads();
        // the min over the warps before mine (kInf: none)
        const K wex = min(kInf, warp_min_k(lane < nw ? sh.tot[b][lane] : kInf, kFwd ? lane < wid : lane > wid));
        const K ex = min(excl, wex);
#pragma unroll
        for (int c = 0; c < C; c++) {
            const int x = x0 + c;
            r[c] = x < w ? (kFwd ? min(ex, m[c]) + 3 * (K)x : min(ex, m[c]) - 3 * (K)x) : kInf;
        }
        if (kWrite) {
#pragma unroll
            for (int c = 0; c < C; c++)
                if (x0 + c < w) dist[(long long)y * w + x0 + c] = (T)r[c];
        }
        if (y == yb) break;
        // neighbours in this row for the next: by shuffle inside the warp; the
        // cell before the warp in scan order is the scan of all warps before,
        // the cell after it the scan through this warp and that cell's own key
        le = shfl_up_k(r[C - 1], 1);
        re = shfl_down_k(r[0], 1);
        const K thru = min(wex, sh.tot[b][wid]);
        if (lane == 0)
            le = wid == 0 ? kInf : (kFwd ? wex : min(thru, sh.edge[b][wid - 1])) + (kFwd ? 3 : -3) * (K)(x0 - 1);
        if (lane == 31)
            re = x0 + C >= w ? kInf : (kFwd ? min(thru, sh.edge[b][wid + 1]) : wex) + (kFwd ? 3 : -3) * (K)(x0 + C);
        have = true;
    }
    if (last) {
#pragma unroll
        for (int c = 0; c < C; c++)
            if (x0 + c < w) last[x0 + c] = r[c];
    }
}

// the whole field in one CTA: down the rows, then back up
template <typename T>
__global__ void __launch_bounds__(1024) k_chamfer2(T* __restrict__ dist, int w, int h)
{
    using K = typename ChamferKey<T>::K;
    __shared__ ChamferShared<K> sh;
    chamfer_rows<T, true, true>(dist, w, 0, h - 1, nullptr, nullptr, sh);
    chamfer_rows<T, false, true>(dist, w, h - 1, 0, nullptr, nullptr, sh);
}

// ---- the same passes over blocks of R rows ----
// A pass only takes mins of sums of exact integers, so it is min-plus linear:
// a block's last row is the min of (a) its last row when nothing comes before
// the block and (b) the true last row of the block before carried through R
// rows of "no value".  The carry has a closed form: a cell gets min over j of
// in[j] + c(x - j), c the cheapest path of the pass's steps (3 straight, 4
// diagonal, along the row only in the scan direction): 3 R + |dx| for
// |dx| <= R, 3 |dx| + R beyond that on the side the row scan comes from.  A
// row that went through the row scan never rises by more than 3 from one cell
// to the next, so the far side never beats the window's edge cell, and the
// carry is  carry_r(in)[x] = 3 r + min over |dx| <= r of in[x - dx] + |dx|.
// Carries compose (carry_a after carry_b is carry_(a + b)), so the blocks'
// true last rows are a scan over the blocks: with s = 1, 4, 16, ...
//     row_k <- min(row_k, carry_(sR) of row_(k-s), carry_(2sR) of row_(k-2s),
//                  carry_(3sR) of row_(k-3s))
// makes row_k right for 4s blocks.  One cooperative launch, a CTA per block:
//   1. run the block with nothing before it, keep its last row;
//   2. the scan, one grid barrier per level;
//   3. run the block again from the previous block's true last row, writing it;
// and the same upwards.
//
// What bounds it: the barrier and shuffle latency of the 4 R rows a CTA walks
// and the scan's grid barriers.  1024 x 1024 int16: 0.47 ms when one CTA
// carried the rows from block to block and each cell searched its window;
// 0.10 ms now; with blocks of 4, 6, 12 or 16 rows 0.11 - 0.12 ms.  2048 x 2048
// int32: 0.26 ms (2.87 ms).
constexpr int kChamferBlockRows = 8;

template <typename K>
struct ChamferCoop {
    K* rows;          // [2][nb][w]: the scan's rows, by level parity
    unsigned* ctl;    // arrivals at the grid barrier
    int* err;
    int w, h, R, nb;
};

// in <- carry of `in` by r rows, less its 3 r: window minima by doubling,
// D_2a[x] = min(D_a[x], D_a[x - a] + a, D_a[x + a] + a).  Returns the buffer
// that holds the result.
template <typename K>
__device__ __forceinline__ K* chamfer_window(K* in, K* out, int w, int r)
{
    constexpr K kInf = sizeof(K) == 8 ? (K)(1LL << 62) : (K)(1 << 29);
    for (int have = 0; have < r && have < w;) {
        const int o = have ? have : 1;   // window 0 -> 1 -> 2 -> 4 ... -> r
        for (int x = threadIdx.x; x < w; x += blockDim.x) {
            const K l = x >= o ? in[x - o] : kInf, g = x + o < w ? in[x + o] : kInf;
            out[x] = min(in[x], min(l, g) + (K)o);
        }
        __syncthreads();
        K* t = in;
        in = out;
        out = t;
        have += o;
    }
    return in;
}

// One way (down or up) of the field.  Returns false when a grid barrier gave up.
template <typename T, bool kFwd>
__device__ __forceinline__ bool chamfer_way(T* __restrict__ dist, const ChamferCoop<typename ChamferKey<T>::K>& p,
                                            ChamferShared<typename ChamferKey<T>::K>& sh,
                                            typename ChamferKey<T>::K* buf, int& parity, unsigned& passed)
{
    using K = typename ChamferKey<T>::K;
    const int w = p.w;
    const int pos = kFwd ? blockIdx.x : p.nb - 1 - blockIdx.x;   // the block's place in scan order
    const int y0 = blockIdx.x * p.R, y1 = min(p.h, y0 + p.R);
    auto row = [&](int which, int q) { return p.rows + ((size_t)which * p.nb + q) * w; };
    K* mine = buf;             // this block's row
    K* wa = buf + w;           // two window buffers
    K* wb = buf + 2 * w;
    // a last block of fewer than R rows is last downwards (no block needs its
    // row) and first upwards (its row is its whole result)
    chamfer_rows<T, kFwd, false>(dist, w, kFwd ? y0 : y1 - 1, kFwd ? y1 - 1 : y0, nullptr, mine, sh);
    __syncthreads();
    for (int s = 1; s < p.nb; s *= 4) {
        parity ^= 1;
        for (int x = threadIdx.x; x < w; x += blockDim.x) row(parity, pos)[x] = mine[x];
        if (!grid_barrier(p.ctl, passed, p.err)) return false;
        const int terms = min(3, pos / s);
        if (terms > 0) {
            const int r = s * p.R;
            K* in = wa;
            for (int t = terms; t > 0; t--) {   // the farthest first, each carried s more blocks with the next
                K* other = in == wa ? wb : wa;
                for (int x = threadIdx.x; x < w; x += blockDim.x) {
                    const K v = __ldcg(row(parity, pos - t * s) + x);
                    in[x] = t == terms ? v : min(v, in[x] + 3 * (K)r);
                }
                __syncthreads();
                in = chamfer_window(in, other, w, r);
            }
            for (int x = threadIdx.x; x < w; x += blockDim.x) mine[x] = min(mine[x], in[x] + 3 * (K)r);
            __syncthreads();
        }
    }
    parity ^= 1;
    for (int x = threadIdx.x; x < w; x += blockDim.x) row(parity, pos)[x] = mine[x];
    if (!grid_barrier(p.ctl, passed, p.err)) return false;
    if (pos > 0) {
        for (int x = threadIdx.x; x < w; x += blockDim.x) mine[x] = __ldcg(row(parity, pos - 1) + x);
        __syncthreads();
    }
    chamfer_rows<T, kFwd, true>(dist, w, kFwd ? y0 : y1 - 1, kFwd ? y1 - 1 : y0, pos ? mine : nullptr, nullptr, sh);
    return true;
}

template <typename T>
__global__ void __launch_bounds__(1024) k_chamfer_coop(T* __restrict__ dist, ChamferCoop<typename ChamferKey<T>::K> p)
{
    using K = typename ChamferKey<T>::K;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ ChamferShared<K> sh;
    K* buf = reinterpret_cast<K*>(smem_raw);   // three rows
    int parity = 0;
    unsigned passed = 0;
    if (!chamfer_way<T, true>(dist, p, sh, buf, parity, passed)) return;
    __syncthreads();
    chamfer_way<T, false>(dist, p, sh, buf, parity, passed);   // a block's rows are its own: no barrier in between
}

template <typename T>
__global__ void __launch_bounds__(256) k_init_distances_int(const uint32_t* __restrict__ mask, T* __restrict__ dist,
                                                            int w, long long rows, T max_d)
{
    const int ws = words_per_row(w);
    const long long n = rows * w;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const long long y = i / w;
        const int x = (int)(i - y * w);
        dist[i] = ((__ldg(mask + y * ws + (x >> 5)) >> (x & 31)) & 1u) ? (T)0 : max_d;
    }
}

int chamfer_threads(int w)
{
    const int t = (w + kChamferCells - 1) / kChamferCells;
    return ((t + 31) / 32) * 32;
}

// Rows from which the blocks are faster than one CTA's walk: their scan costs some
// 20 - 30 us, a row 0.5 - 3 us by its width (one CTA against blocks, us, int16: 250
// x 16 19, 33; 250 x 32 33, 41; 1000 x 20 36, 41; 1000 x 24 42, 40; 2000 x 18 45, 47; 2000 x
// 20 51, 47; 4096 x 16 69, 58; int32 250 x 32 50, 55; 2000 x 18 72, 74)
static int chamfer_block_rows(int w) { return w <= 512 ? 33 : w <= 1024 ? 24 : w <= 2048 ? 20 : 16; }

template <typename T>
void launch_chamfer_2d(T* dist, int w, int h, int* err, size_t scratch_cap, cudaStream_t st)
{
    using K = typename ChamferKey<T>::K;
    const int threads = chamfer_threads(w);
    ProfScope ps("chamfer_2d", st);
    if (h >= chamfer_block_rows(w)) {
        const size_t smem = 3 * (size_t)w * sizeof(K);
        // (always: the static shared memory counts towards the 48 KB that need no asking)
        cudaFuncSetAttribute(k_chamfer_coop<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        int per_sm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_chamfer_coop<T>, threads, smem);
        // every block's CTA has to be resident: longer blocks for taller fields
        const long long resident = (long long)per_sm * g_num_sms;
        int R = kChamferBlockRows;
        while (resident > 0 && (h + R - 1) / R > resident) R *= 2;
        const int nb = (h + R - 1) / R;
        void* scratch = nullptr;
        const size_t rows = 2 * (size_t)nb * w * sizeof(K);
        if (resident > 0 && nb >= 2 && (!scratch_cap || rows + 256 <= scratch_cap) &&
            cudaMallocAsync(&scratch, rows + 256, st) == cudaSuccess) {
            ChamferCoop<K> p{static_cast<K*>(scratch), reinterpret_cast<unsigned*>(static_cast<char*>(scratch) + rows),
                             err, w, h, R, nb};
            cudaMemsetAsync(p.ctl, 0, sizeof(unsigned), st);
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(nb);
            cfg.blockDim = dim3(threads);
            cfg.dynamicSmemBytes = smem;
            cfg.stream = st;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeCooperative;
            attr[0].val.cooperative = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            const bool ok = cudaLaunchKernelEx(&cfg, k_chamfer_coop<T>, dist, p) == cudaSuccess;
            cudaFreeAsync(scratch, st);
            if (ok) return;
        }
        cudaGetLastError();   // no scratch or no cooperative launch: walk the whole field in one CTA
    }
    k_chamfer2<T><<<1, threads, 0, st>>>(dist, w, h);
}

template <typename T>
void launch_init_distances_int(const uint32_t* mask, T* dist, int w, long long rows, T max_d, cudaStream_t st)
{
    long long n = rows * w;
    long long blocks = (n + 255) / 256;
    long long cap = (long long)g_num_sms * 32;
    k_init_distances_int<T><<<(int)(blocks < cap ? blocks : cap), 256, 0, st>>>(mask, dist, w, rows, max_d);
}

template void launch_chamfer_2d<int16_t>(int16_t*, int, int, int*, size_t, cudaStream_t);
template void launch_chamfer_2d<int32_t>(int32_t*, int, int, int*, size_t, cudaStream_t);
template void launch_init_distances_int<int16_t>(const uint32_t*, int16_t*, int, long long, int16_t, cudaStream_t);
template void launch_init_distances_int<int32_t>(const uint32_t*, int32_t*, int, long long, int32_t, cudaStream_t);

}  // namespace dolk
