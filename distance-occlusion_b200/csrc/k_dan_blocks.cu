// k_dan_blocks.cu -- Danielsson (2D and 3D) as a fixed-point iteration over
// blocks of rows, bit-identical to the serial sweeps.
//
// The reference's Danielsson (DistanceOcclusionLib.cpp:702-778 2D,
// :2264-2394 3D) is one long chain: every row needs the previous row, every
// slice the previous slice after its full 2D sweep, every cell of an x pass
// the cell before it.  Cut each sweep phase (the 2D image; each z direction of
// a volume) into blocks of 32 S columns, R rows and Z slices, a warp each.  A
// block runs the reference's steps over its own cells -- slice by slice the z
// pull, rows y0..y1-1 going down, then y1-1..y0 going up, each with its x
// passes -- from the inputs that other blocks produce:
//
//   Z  the previous slice's cells after its sweep               (block k-1)
//   D  row y0-1 after the down sweep                            (block c-1)
//   U  row y1 after the up sweep                                (block c+1)
//   L  per row and sweep, the cell left of the block after the
//      pass to the right                                        (block xb-1)
//   R  the cell right of it after the pass to the left          (block xb+1)
//
// Every block starts from guesses (the phase input's own rows, no cell at the
// sides), all blocks run in parallel, and each round recomputes exactly the
// blocks whose inputs changed in the round before.  At the stop every block's
// inputs equal its producers' outputs, so by induction along the serial order
// (split into the half sweeps and their passes it is acyclic) every output is
// the serial one.  Round r finalises at least one more piece of the chain, so
// the iteration ends; in practice after about as many rounds as the longest
// distance in blocks that a seed's influence travels.
//
// What bounds it: rounds x the latency of a block, one dependent row step after
// another, and with all blocks busy the integer pipe (some 400 instructions per
// step of 128 cells).  Short segments make short steps, and cutting rows into
// x blocks costs no rounds (a model of the iteration on the 256^3 volume of
// boxes and spheres: 19 + 14 rounds at 256 and at 128 columns, 20 + 15 at 64,
// with 9 / 8 / 7 times the serial work), while it takes the exchange between
// the warps of a row out of every pass.
// 256^3 boxes and spheres 17.4 -> 8.8 ms, 1024^2 with 100 points 1.41 -> 0.51 ms
// against one CTA per block of whole rows.
//
// Outputs alternate between two version buffers per block, so a round reads
// only the previous round's outputs; a block's version flips whenever it runs,
// and the cells that other blocks read are compared with their old values to
// find the blocks that have to run again.  One cooperative launch runs all
// rounds, each closed by one grid barrier (bounded waits).  With a warp for
// every block a block that changed marks its dependents for the next round;
// larger fields take blocks from a work list.
#include "dan_rounds.h"
#include "dan_serial.cuh"
#include "grid_barrier.cuh"
#include "kernels.h"

namespace dolk {

constexpr int kBlkMaxWidth = 2048;
constexpr int kBlkMaxRows = 16;    // rows of a block: a lane per row and sweep

struct DanBlk {
    const void* A;         // phase input, unchanged during the phase
    void* V[2];            // output versions (cells, same layout as A)
    void* DB[2];           // per slice, chunk of rows and version: its last row after the down sweep
    uint2* XR[2];          // per row, sweep, x block and version: its last cell after the pass to the right (xy, z)
    uint2* XL[2];          // its first cell after the pass to the left
    unsigned* state;       // per block: round it last ran in + 1, version after and before that (block_state)
    uint8_t* dirty[2];     // few blocks: per block, to run in the round of that parity
    int* stamp;            // many blocks: per block, last round it was queued for
    int* wl[2];            // and the work lists by round parity
    unsigned* ctl;         // by round modulo 3: [0..2] a block changed / work-list size, [3..5] work counter;
                           // [6] grid barrier, [7] rounds used (0: not done)
    int* err;
    int w, h, d, R, nc, nx, cw;
    int dir;      // +1: slices zfirst, zfirst+1, ...; -1: downwards
    int zfirst;   // first slice of the phase's chain (the slice before it keeps its input)
    int nchain;   // slices in the chain (2D: 1)
    int Z;        // slices per block
    int nk;       // blocks along the chain: ceil(nchain / Z)
    int nblocks;  // nk * nc * nx, block (k, c, xb) at (k * nc + c) * nx + xb
    int max_rounds;
    bool rest;    // a field that is not done by then is left to k_dan_rest
};

// A block's state word: the round it last ran in plus 1, the version that holds
// its output since and the one before (2: none yet, the input's rows stand).
// One word, so that a reader of the same round sees either it or the word
// before it, and takes the output of before this round from both.
__device__ __forceinline__ unsigned block_state(int round, int now, int before)
{
    return ((unsigned)(round + 1) << 4) | ((unsigned)now << 2) | (unsigned)before;
}
__device__ __forceinline__ int block_version(unsigned state, int round)
{
    return (int)((state >> 4) == (unsigned)(round + 1) ? state & 3u : (state >> 2) & 3u);
}

// what a run changed for other blocks
constexpr int kChgLast = 1;    // a row of the block's last slice changed  -> block (k+1, c)
constexpr int kChgFirst = 2;   // row y0 of some slice changed             -> block (k, c-1)
constexpr int kChgDown = 4;    // the down-sweep row y1-1 of some slice    -> block (k, c+1)
constexpr int kChgRight = 8;   // a last cell after a pass to the right    -> block xb+1
constexpr int kChgLeft = 16;   // a first cell after a pass to the left    -> block xb-1

template <int DIM, int S>
using BlockIO = RowIO<DIM, S, 2>;

// Shared memory of a warp: its RowIO strips, then its part of the block's R
// rows, cell s of lane l at [row][s][l]: after the down sweep a row's down
// result, after the up sweep its result, which the next slice pulls from.
template <int DIM, int S>
__host__ __device__ constexpr size_t dan_warp_bytes(int R)
{
    return BlockIO<DIM, S>::kBytes + (size_t)R * S * 32 * (DIM == 3 ? 6 : 4);
}

template <int DIM, int S>
struct BlockRows;
template <int S>
struct BlockRows<2, S> {
    uint32_t* c;

    DOL_DI void put(int r, const Cells<2, S>& v) const
    {
#pragma unroll
        for (int s = 0; s < S; s++) c[(r * S + s) * 32 + (threadIdx.x & 31)] = v.xy[s];
    }
    DOL_DI void get(int r, uint32_t (&xy)[S], int (&z)[S]) const
    {
#pragma unroll
        for (int s = 0; s < S; s++) {
            xy[s] = c[(r * S + s) * 32 + (threadIdx.x & 31)];
            z[s] = 0;
        }
    }
};
template <int S>
struct BlockRows<3, S> {
    uint32_t* c;
    int16_t* zz;

    DOL_DI void put(int r, const Cells<3, S>& v) const
    {
#pragma unroll
        for (int s = 0; s < S; s++) {
            c[(r * S + s) * 32 + (threadIdx.x & 31)] = v.xy[s];
            zz[(r * S + s) * 32 + (threadIdx.x & 31)] = (int16_t)v.z[s];
        }
    }
    DOL_DI void get(int r, uint32_t (&xy)[S], int (&z)[S]) const
    {
#pragma unroll
        for (int s = 0; s < S; s++) {
            xy[s] = c[(r * S + s) * 32 + (threadIdx.x & 31)];
            z[s] = zz[(r * S + s) * 32 + (threadIdx.x & 31)];
        }
    }
};

// One block by one warp; returns what changed (bits above, per lane).
template <int DIM, int S>
__device__ __forceinline__ int dan_block(const DanBlk& p, int b, int round, const BlockIO<DIM, S>& io,
                                         const BlockRows<DIM, S>& T)
{
    using IO = BlockIO<DIM, S>;
    using Row = Cells<DIM, S>;
    const int lane = threadIdx.x & 31;
    const int w = p.w, h = p.h, cw = p.cw;
    const int xb = b % p.nx, kc = b / p.nx;
    const int k = kc / p.nc;
    const int c = kc - k * p.nc;
    const int xw = xb * 32 * S;
    const int y0 = c * p.R, y1 = min(y0 + p.R, h), L = y1 - y0;
    const long long plane = (long long)w * h;
    const long long abytes = plane * p.d * IO::kCell, dbytes = (long long)p.nc * p.d * w * IO::kCell;
    // neighbour blocks' versions (fixed for the whole round): lane i looks one up
    int nb = b;
    if (lane == 1) nb = c > 0 ? b - p.nx : -1;
    if (lane == 2) nb = y1 < h ? b + p.nx : -1;
    if (lane == 3) nb = DIM == 3 && k > 0 ? b - p.nc * p.nx : -1;
    if (lane == 4) nb = xb > 0 ? b - 1 : -1;
    if (lane == 5) nb = xb + 1 < p.nx ? b + 1 : -1;
    const int ver = lane < 6 && nb >= 0 ? block_version(__ldcg(p.state + nb), round) : 2;
    const int vo = __shfl_sync(0xFFFFFFFFu, ver, 0), vn = vo == 0 ? 1 : 0;
    const int vd = __shfl_sync(0xFFFFFFFFu, ver, 1), vu = __shfl_sync(0xFFFFFFFFu, ver, 2);
    const int vz = __shfl_sync(0xFFFFFFFFu, ver, 3);
    const int vl = __shfl_sync(0xFFFFFFFFu, ver, 4), vr = __shfl_sync(0xFFFFFFFFu, ver, 5);
    const int dz = -p.dir * cw;
    const int pos0 = k * p.Z, nsl = min(p.Z, p.nchain - pos0);
    auto arr = [&](int v) { return static_cast<unsigned char*>(v == 2 ? const_cast<void*>(p.A) : p.V[v]); };
    auto cell_at = [&](int z, int y) { return ((long long)z * plane + (long long)y * w + xw) * IO::kCell; };
    auto fetch_a = [&](int r, int v, int z, int y) {
        unsigned char* q = arr(v);
        io.fetch(r, q + cell_at(z, y), q, q + abytes);
    };
    // the down-boundary row of chunk cc of slice z in version v (2: the input's row yy)
    auto fetch_d = [&](int r, int v, int z, int cc, int yy) -> const unsigned char* {
        if (v == 2) {
            fetch_a(r, 2, z, yy);
            return arr(2) + cell_at(z, yy);
        }
        unsigned char* q = static_cast<unsigned char*>(p.DB[v]);
        const unsigned char* a = q + (((long long)z * p.nc + cc) * w + xw) * IO::kCell;
        io.fetch(r, a, q, q + dbytes);
        return a;
    };
    auto cells_xyz = [&](int r, const unsigned char* a, uint32_t (&xy)[S], int (&z)[S]) {
        uint32_t wd[IO::kWords];
        io.words(wd, r, a);
        IO::split(wd, xy, z);
    };
    // does the fetched row differ from c in one of this lane's cells?
    auto differs = [&](int r, const unsigned char* a, const Row& c) -> bool {
        uint32_t xy[S];
        int z[S];
        cells_xyz(r, a, xy, z);
        const int n = io.live();
        bool d = false;
#pragma unroll
        for (int s = 0; s < S; s++) d |= s < n && (xy[s] != c.xy[s] || (DIM == 3 && z[s] != c.z[s]));
        return d;
    };

    // a row as candidate only: cells that win against none when shifted by +-cw in y
    auto absent = [&](Row& r) {
#pragma unroll
        for (int s = 0; s < S; s++) {
            r.xy[s] = 0;
            r.z[s] = 0;
            r.W[s] = 0;
            r.L[s] = INT_MAX - cw * cw;
        }
    };
    Row P, C;
    // strips: the next step's row; the row beside it (slice before, block
    // below); the row above the block, in the strip that stores use: it is
    // loaded after a slice's last store and read before the next one's first
    constexpr int rc = 0, rq = 1, rd = IO::kStrips - 1;
    int bits = 0;
    const bool has_d = c > 0, has_u = y1 < h;
    const unsigned char* ad = nullptr;
    auto first_rows = [&](int j) {   // what the first step of slice j needs
        const int z = p.zfirst + p.dir * (pos0 + j);
        if (has_d) ad = fetch_d(rd, vd, z, c - 1, y0 - 1);
        fetch_a(rc, 2, z, y0);
        if (DIM == 3 && j == 0) fetch_a(rq, vz, z - p.dir, y0);
    };
    // the sides: lane t holds the cells of step t of a slice
    const bool sides = p.nx > 1;
    const int yt = lane < L ? y0 + lane : y0 + 2 * L - 1 - lane;
    auto side_at = [&](int z) { return (((long long)z * h + yt) * 2 + (lane < L ? 0 : 1)) * p.nx + xb; };
    const uint2 kNoCell = make_uint2(0x80000000u, 0x80000000u);   // (z is never that: 16 bits)
    uint2 inL = kNoCell, inR = kNoCell, nextL = kNoCell, nextR = kNoCell;
    auto load_sides = [&](int j) {
        const int z = p.zfirst + p.dir * (pos0 + j);
        if (lane < 2 * L) {
            if (vl != 2) nextL = __ldcg(p.XR[vl] + side_at(z) - 1);
            if (vr != 2) nextR = __ldcg(p.XL[vr] + side_at(z) + 1);
        }
    };
    auto side_input = [&](const uint2& in, int t) -> Chain {
        const uint32_t xy = __shfl_sync(0xFFFFFFFFu, in.x, t);
        const int z = (int)__shfl_sync(0xFFFFFFFFu, in.y, t);
        if (z == (int)0x80000000u) return chain_none(cw);
        return Chain{xy, w_of<DIM>(xy, z), z};
    };
    __syncwarp();
    first_rows(0);
    if (sides) load_sides(0);

    for (int j = 0; j < nsl; j++) {
        const int z = p.zfirst + p.dir * (pos0 + j);
        const bool last = j == nsl - 1;
        uint2 outR = kNoCell, outL = kNoCell;   // lane t: this block's own side cells of step t
        inL = nextL;
        inR = nextR;
        // the row above the block after its down sweep is the first step's candidate
        if (has_d) io.cells_of(P, rd, ad, cw);
        else absent(P);
        // steps 0 .. L-1 go down the rows, L .. 2L-1 back up
#pragma unroll 1
        for (int i = 0; i < 2 * L; i++) {
            const bool down = i < L;
            const int q = down ? i : 2 * L - 1 - i, y = y0 + q;
            uint32_t xy[S];
            int zz[S];
            if (down) {   // its own cells, then the slice before
                io.cells_of(C, rc, arr(2) + cell_at(z, y), cw);
                if constexpr (DIM == 3) {
                    if (j == 0) cells_xyz(rq, arr(vz) + cell_at(z - p.dir, y), xy, zz);
                    else T.get(q, xy, zz);
                    pull_z<S>(C, xy, zz, dz);
                }
            } else if (i > L) {   // its down result
                T.get(q, xy, zz);
#pragma unroll
                for (int s = 0; s < S; s++) {
                    C.xy[s] = xy[s];
                    C.z[s] = zz[s];
                    C.W[s] = w_of<DIM>(xy[s], zz[s]);
                    C.L[s] = len_of(xy[s], C.W[s]);
                }
                const int n = io.live();
                if (n < S) {
#pragma unroll
                    for (int s = 0; s < S; s++)
                        if (s >= n) set_none(C, s, cw);
                }
            } else {   // the turn: its down result is at hand, the candidate is the row below the block
                C = P;
                if (has_u) io.cells_of(P, rq, arr(vu) + cell_at(z, y1), cw);
                else absent(P);
            }
            // old results are compared where another block reads them: the
            // block below reads the last down row, the block above the first
            // row, the next block in z the last slice
            const bool cmp_d = has_u && i == L - 1;
            const bool cmp_u = !down && ((last && k + 1 < p.nk) || (q == 0 && has_d));
            const unsigned char* ao = nullptr;
            // loaded behind this step's passes: the old result, what the next step needs
            if (i + 1 < L) {
                fetch_a(rc, 2, z, y + 1);
                if (DIM == 3 && j == 0) fetch_a(rq, vz, z - p.dir, y + 1);
            } else if (i == L - 1) {
                if (has_u) {
                    ao = fetch_d(rc, vo, z, c, y);
                    fetch_a(rq, vu, z, y1);
                }
            } else if (cmp_u) {
                fetch_a(rc, vo, z, y);
                ao = arr(vo) + cell_at(z, y);
            }
            merge_y<DIM, S>(P, C, down ? -cw : cw);
            if (down ? y > 0 : y < h - 1) {
                RowShared<1> none;
                int par = 0;
                Chain wl = chain_none(cw), wr = wl;
                if (sides) {
                    wl = side_input(inL, i);
                    wr = side_input(inR, i);
                }
                row_pass_w<DIM, S, 1, +1, NoDiag>(P, NoDiag{}, cw, none, par, wl);
                if (sides) {
                    const uint32_t oxy = __shfl_sync(0xFFFFFFFFu, P.xy[S - 1], 31);
                    const int oz = DIM == 3 ? __shfl_sync(0xFFFFFFFFu, P.z[S - 1], 31) : 0;
                    if (lane == i) outR = make_uint2(oxy, (uint32_t)oz);
                }
                row_pass_w<DIM, S, 1, -1, NoDiag>(P, NoDiag{}, cw, none, par, wr);
                if (sides) {
                    const uint32_t oxy = __shfl_sync(0xFFFFFFFFu, P.xy[0], 0);
                    const int oz = DIM == 3 ? __shfl_sync(0xFFFFFFFFu, P.z[0], 0) : 0;
                    if (lane == i) outL = make_uint2(oxy, (uint32_t)oz);
                }
            }
            if (DIM == 3 || down) T.put(q, P);
            if (cmp_d) {
                if (differs(rc, ao, P)) bits |= kChgDown;
                unsigned char* db = static_cast<unsigned char*>(p.DB[vn]);
                io.put_cells(db + (((long long)z * p.nc + c) * w + xw) * IO::kCell, P);
            }
            if (!down) {
                if (cmp_u && differs(rc, ao, P)) bits |= (last ? kChgLast : 0) | (q == 0 ? kChgFirst : 0);
                io.put_cells(static_cast<unsigned char*>(p.V[vn]) + cell_at(z, y), P);
            }
            if (sides && i == L && !last) load_sides(j + 1);
            if (i == 2 * L - 1 && !last) first_rows(j + 1);
        }
        if (sides && lane < 2 * L) {
            const long long at = side_at(z);
            auto post = [&](uint2* const (&x)[2], const uint2& v) -> bool {
                const uint2 o = vo == 2 ? kNoCell : __ldcg(x[vo == 1 ? 1 : 0] + at);
                x[vn][at] = v;
                return o.x != v.x || o.y != v.y;
            };
            if (xb + 1 < p.nx && post(p.XR, outR)) bits |= kChgRight;
            if (xb > 0 && post(p.XL, outL)) bits |= kChgLeft;
        }
    }
    __syncwarp();   // every lane's stores, before the state word that shows them
    if (lane == 0) __stcg(p.state + b, block_state(round, vn, vo));
    return bits;
}

constexpr int kBlkWarps = 4;   // per CTA, each taking blocks by itself

template <int DIM, int S>
__global__ void __launch_bounds__(32 * kBlkWarps, 4) k_dan_blocks(DanBlk p)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31;
    unsigned char* mine = smem_raw + (threadIdx.x >> 5) * dan_warp_bytes<DIM, S>(p.R);
    BlockRows<DIM, S> T;
    T.c = reinterpret_cast<uint32_t*>(mine + BlockIO<DIM, S>::kBytes);
    if constexpr (DIM == 3) T.zz = reinterpret_cast<int16_t*>(T.c + p.R * S * 32);
    const int warp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int warps = (int)((gridDim.x * blockDim.x) >> 5);
    const bool own = p.nblocks <= warps;   // a warp per block: no lists
    unsigned passed = 0;
    int round = 0;
    for (;; round++) {
        const int cur = round & 1, r3 = round % 3, n3 = (round + 1) % 3;
        if (round >= p.max_rounds) {
            if (!p.rest && blockIdx.x == 0 && threadIdx.x == 0) atomicExch(p.err, 3);
            return;
        }
        const unsigned nwork = own || round == 0 ? (unsigned)p.nblocks : __ldcg(p.ctl + (round + 2) % 3);
        for (bool first = true;; first = false) {
            int b;
            if (own) {
                if (!first || warp >= p.nblocks || (round > 0 && __ldcg(p.dirty[cur] + warp) == 0)) break;
                b = warp;
                if (lane == 0) p.dirty[cur][b] = 0;
            } else {
                unsigned it = 0;
                if (lane == 0) it = atomicAdd(p.ctl + 3 + r3, 1u);
                it = __shfl_sync(0xFFFFFFFFu, it, 0);
                if (it >= nwork) break;
                b = round == 0 ? (int)it : __ldcg(p.wl[cur] + it);
            }
            const int xb = b % p.nx;
            const BlockIO<DIM, S> io{mine, min(32 * S, p.w - xb * 32 * S)};
            const unsigned bits = __reduce_or_sync(0xFFFFFFFFu, (unsigned)dan_block<DIM, S>(p, b, round, io, T));
            if (lane < 5 && ((bits >> lane) & 1u)) {   // lane i queues the dependent of bit i
                const int k = b / p.nx / p.nc, c = b / p.nx - k * p.nc;
                int dep = -1;
                if (lane == 0 && k + 1 < p.nk) dep = b + p.nc * p.nx;
                if (lane == 1 && c > 0) dep = b - p.nx;
                if (lane == 2 && c + 1 < p.nc) dep = b + p.nx;
                if (lane == 3 && xb + 1 < p.nx) dep = b + 1;
                if (lane == 4 && xb > 0) dep = b - 1;
                if (dep >= 0) {
                    if (own) {
                        p.dirty[cur ^ 1][dep] = 1;
                        __stcg(p.ctl + r3, 1u);
                    } else if (atomicMax(p.stamp + dep, round + 1) < round + 1) {
                        p.wl[cur ^ 1][atomicAdd(p.ctl + r3, 1u)] = dep;
                    }
                }
            }
            __syncwarp();
        }
        if (blockIdx.x == 0 && threadIdx.x == 0) {   // the next round's words: last read two barriers ago
            __stcg(p.ctl + n3, 0u);
            __stcg(p.ctl + 3 + n3, 0u);
        }
        if (!grid_barrier(p.ctl + 6, passed, p.err)) return;
        if (__ldcg(p.ctl + r3) == 0) break;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) p.ctl[7] = (unsigned)(round + 1);
}

// every block takes its rows from the input; the first round runs all
__global__ void k_dan_blocks_init(DanBlk p)
{
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < p.nblocks; b += gridDim.x * blockDim.x) {
        p.state[b] = (2u << 2) | 2u;
        p.dirty[0][b] = 0;
        p.dirty[1][b] = 0;
        p.stamp[b] = 0;
    }
    if (blockIdx.x == 0 && threadIdx.x < 8) p.ctl[threadIdx.x] = 0;
}

// the converged outputs back into the caller's array, by 16-bit halves: kCell
// of them per cell, x blocks of bx cells
template <int kCell>
__global__ void k_dan_blocks_store(DanBlk p, uint16_t* __restrict__ dl, int bx)
{
    if (p.ctl[7] == 0) return;   // not done
    const long long row_halves = (long long)p.w * kCell;
    const long long rows = (long long)p.h * p.d;
    for (long long r = blockIdx.x; r < rows; r += gridDim.x) {
        const int z = (int)(r / p.h), y = (int)(r - (long long)z * p.h);
        const int pos = (z - p.zfirst) * p.dir;
        if (pos < 0 || pos >= p.nchain) continue;   // the fixed slice
        const unsigned* state = p.state + ((pos / p.Z) * p.nc + y / p.R) * p.nx;
        const uint16_t* s0 = static_cast<const uint16_t*>(p.V[0]) + r * row_halves;
        const uint16_t* s1 = static_cast<const uint16_t*>(p.V[1]) + r * row_halves;
        uint16_t* dst = dl + r * row_halves;
        const int span = bx * kCell;   // a multiple of 64 halves
        if ((((uintptr_t)s0 | (uintptr_t)s1 | (uintptr_t)dst) & 15) == 0 && row_halves % 8 == 0) {
            for (int i = threadIdx.x; i < row_halves / 8; i += blockDim.x)
                reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(state[8 * i / span] >> 2 & 1u ? s1 : s0)[i];
        } else {
            for (int i = threadIdx.x; i < row_halves; i += blockDim.x) dst[i] = (state[i / span] >> 2 & 1u ? s1 : s0)[i];
        }
    }
}

// The phase by the serial walk, on the caller's cells, when its rounds ran out
template <int DIM, int S, int NW>
__global__ void __launch_bounds__(32 * NW) k_dan_rest(const unsigned* __restrict__ ctl, void* __restrict__ dl, int w,
                                                      int h, int d, int cw, int way)
{
    extern __shared__ __align__(16) unsigned char strips[];
    __shared__ RowShared<NW> sh;
    if (ctl[7] != 0) return;
    if constexpr (NW > 1) {
        if (threadIdx.x == 0) sh.bar = 0;
        __syncthreads();
    }
    dan_serial<DIM, S, NW>(dl, w, h, d, cw, strips + (NW > 1 ? threadIdx.x >> 5 : 0) * SerialIO<DIM, S>::kBytes, sh, way);
}

template <int DIM>
static void launch_dan_rest(const DanBlk& p, void* dl, cudaStream_t st)
{
    auto run = [&](auto kern, int warps, size_t strips) {
        if (strips > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)strips);
        kern<<<1, 32 * warps, strips, st>>>(p.ctl, dl, p.w, p.h, p.d, p.cw, p.dir > 0 ? 0 : 1);
    };
    if (p.w <= 64) run(k_dan_rest<DIM, 2, 1>, 1, SerialIO<DIM, 2>::kBytes);
    else if (p.w <= 128) run(k_dan_rest<DIM, 4, 1>, 1, SerialIO<DIM, 4>::kBytes);
    else if (p.w <= 256) run(k_dan_rest<DIM, 8, 1>, 1, SerialIO<DIM, 8>::kBytes);
    else if (p.w <= 512) run(k_dan_rest<DIM, 8, 2>, 2, 2 * SerialIO<DIM, 8>::kBytes);
    else if (p.w <= 1024) run(k_dan_rest<DIM, 8, 4>, 4, 4 * SerialIO<DIM, 8>::kBytes);
    else run(k_dan_rest<DIM, 8, 8>, 8, 8 * SerialIO<DIM, 8>::kBytes);
}

static size_t al256(size_t b) { return (b + 255) & ~(size_t)255; }

int dan_blocks_rows(int dim, int w, int h, int d)
{
    const int tv = tune_get(kTuneDanRows, w);
    if (tv > 0) return tv >= kDanSerial ? kDanSerial : min(tv, kBlkMaxRows);
    // Fields of a short chain go to the serial engine: the blocks take some 20
    // rounds and three launches however short it is.  Images (noise of lattice 51
    // | 20, and 40 points, us serial against blocks): 64 x 64 76 | 121, 119 against
    // 157 | 156, 105; 64 x 128 158 | 236, 205 against 285 | 135, 121; 128 x 64 160 |
    // 147, 119 against 156 | 145, 109; 256 x 32 82 | 100, 88 against 179 | 146, 131;
    // 96 x 96 280 | 346, 252 against 285 | 219, 146; lattice 20 and 30 points: 400 x 16
    // 101, 92 against 114, 101; 700 x 16 123, 93 against 138, 124; 700 x 24 184, 134
    // against 177, 148).  Volumes: a row step takes the serial engine about 0.5 us
    // and 2 ns a cell; blocks from 4 (h - 1) (d - 1) steps that sum to 140 us,
    // 220 where slices outnumber rows, each a step of the rounds' chain (the same
    // contents: 64 x 4 x 16 137, 137 against 229, 208; 64 x 8 x 16 311, 285
    // against 295, 265; 16 x 16 x 4 132, 118 against 168, 122; 16 x 16 x 8 295, 257
    // against 212, 182; 256 x 8 x 4 119, 116 against 172, 156; 256 x 16 x 4 244, 224
    // against 228, 197; 1000 x 4 x 6 257, 231 against 254, 233; 32 x 3
    // x 40 234, 206 against 336, 234); one row per slice has
    // no passes at all (64 x 1 x 40 0.04 against 0.27 ms).
    const long long cells = (long long)w * h * (dim == 3 ? d : 1);
    if (cells < 1024 || w > kBlkMaxWidth) return kDanSerial;
    if (dim == 3 && (h == 1 || 4LL * (h - 1) * (d - 1) * (250 + w) < (d > h ? 110000 : 70000))) return kDanSerial;
    if (dim == 2 && ((w <= 256 && h <= 32) || (w <= 128 && h <= 64) || (w <= 64 && h <= 200) || (w <= 32 && h <= 512) ||
                     h < 24))
        return kDanSerial;
    // 8 rows; tall images of several x blocks 16.  8 | 16 rows on 1024 columns,
    // noise of lattice 20, of lattice 51, 100 points, us: 700 high 240 | 286, 394 |
    // 446, 469 | 414; 1000 high 305 | 291, 410 | 453, 572 | 522; 1600 high 0.88, 0.95, 0.77
    // of the time (on 300 columns 1.14, 1.0, 0.85): even somewhere between 850 and
    // 1100 rows, by content.  Volumes whose
    // blocks of 4 rows do not outnumber the resident warps by much 4 (101 x 77
    // x 90: 1.6 against 2.0 ms; 256^3: 9.3 against 8.8)
    if (dim == 2) return w > 256 && h >= 1024 ? 16 : 8;
    return cells <= (1 << 21) ? 4 : 8;
}

// Cells per lane.  Images of up to 512 columns take x blocks of 64 (256^2 noise,
// lattice 51: 0.32 ms, 0.35 with 128, 0.44 as one block; 96 x 192 0.37 against
// 0.49; 400 x 256 0.36 either way), but 128 columns one block (128 x 256 noise,
// lattice 20: 0.16 against 0.18 ms); wider ones blocks of 128 (1024^2, 100 points:
// 0.51 ms, 0.64 with 256); volumes blocks of 64 (256^3 boxes and spheres: 8.8
// ms, 9.4 with 128 and 11.8 with 256), from 512 columns on 128.
static int dan_blocks_s(int dim, int w)
{
    int s = tune_get(dim == 2 ? kTuneDan2 : kTuneDan3, w);
    if (s != 2 && s != 4 && s != 8) {
        if (dim == 2) s = w <= 512 && (w <= 112 || w > 128) ? 2 : 4;
        else s = w < 512 ? 2 : 4;
    }
    return s;
}

// Bytes of the pieces of the workspace.  The control words need 32 of the last
// piece's; the rest lets the first piece start at a 16-byte boundary whatever the
// caller's workspace is aligned to (side cells move 8 bytes at a time).
constexpr size_t kCtlBytes = 256, kWsAlign = 16;
struct DanSizes {
    size_t field, down, side, flag, list, total;
};
static DanSizes dan_sizes(int dim, int w, int h, int d, int R)
{
    const size_t cb = dim == 3 ? 6 : 4;
    const size_t nd = dim == 3 ? d : 1;
    const int bx = 32 * dan_blocks_s(dim, w);
    const size_t nc = (h + R - 1) / R, nx = (w + bx - 1) / bx;
    DanSizes z;
    z.field = al256((size_t)w * h * nd * cb);
    z.down = al256(nc * nd * w * cb);
    z.side = nx > 1 ? al256(nd * h * 2 * nx * sizeof(uint2)) : 0;
    z.flag = al256(nc * nd * nx);
    z.list = al256(nc * nd * nx * sizeof(int));
    z.total = 2 * z.field + 2 * z.down + 4 * z.side + 2 * z.flag + 4 * z.list + kCtlBytes;
    return z;
}

size_t dan_blocks_workspace_bytes(int dim, int w, int h, int d, int R)
{
    return dan_sizes(dim, w, h, d, min(R, kBlkMaxRows)).total;
}

template <int kDim, int S>
static bool run_phase(DanBlk& p, void* dl, cudaStream_t st)
{
    auto kern = k_dan_blocks<kDim, S>;
    const size_t warp_bytes = dan_warp_bytes<kDim, S>(p.R);
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kBlkWarps * warp_bytes));
    cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * kBlkWarps, kBlkWarps * warp_bytes) !=
            cudaSuccess ||
        per_sm < 1)
        return false;
    const int resident = per_sm * g_num_sms * kBlkWarps;   // warps
    // slices per block: 2 while that gives at most two blocks per resident warp
    // (101 x 77 x 90: 1.6 ms, 1.8 with 4), 1 for up to 16 slices then (noise | 30
    // points: 64 x 400 x 8 0.45 | 0.94 ms, 0.52 | 1.44 with 2; 200 x 400 x 4 0.43 | 0.95,
    // 0.54 | 1.32; but 8 x 400 x 100 1.45 | 3.26, 1.29 | 3.60), else 4, more where there
    // would be over 8 blocks per resident warp, at most 16
    int Z = tune_get(kTuneDanSlices, p.w);
    if (Z < 1) {
        Z = (int)((long long)p.nchain * p.nc * p.nx / (8LL * resident));
        const bool few = (long long)p.nchain * p.nc * p.nx <= 4LL * resident;
        Z = max(few ? (p.nchain <= 16 ? 1 : 2) : 4, min(Z, 16));
    }
    if (Z > p.nchain) Z = p.nchain;
    p.Z = Z;
    p.nk = (p.nchain + Z - 1) / Z;
    p.nblocks = p.nk * p.nc * p.nx;
    p.max_rounds = p.rest ? dan_round_budget(kDim, p.nchain, p.h, p.nc, p.nk, p.nx) : dan_max_rounds(p.nchain, p.h, p.nx);
    k_dan_blocks_init<<<min((p.nblocks + 255) / 256, g_num_sms * 8), 256, 0, st>>>(p);
    // a warp per CTA while that spreads the blocks over more SMs
    const int warps = p.nblocks <= 2 * g_num_sms ? 1 : kBlkWarps;
    const int ctas = (p.nblocks + warps - 1) / warps;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(min(per_sm * g_num_sms, ctas));
    cfg.blockDim = dim3(32 * warps);
    cfg.dynamicSmemBytes = warps * warp_bytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, kern, p) != cudaSuccess) return false;
    long long gb = (long long)p.h * p.d;
    if (gb > (long long)g_num_sms * 32) gb = (long long)g_num_sms * 32;
    k_dan_blocks_store<kDim == 3 ? 3 : 2>
        <<<(int)gb, p.w >= 128 ? 256 : 64, 0, st>>>(p, static_cast<uint16_t*>(dl), 32 * S);
    if (p.rest) launch_dan_rest<kDim>(p, dl, st);
    return true;
}

template <int kDim, int S>
static bool run_all(int w, int h, int d, int cw, int R, bool initial, void* deltas, void* ws, int* err, cudaStream_t st)
{
    const DanSizes z = dan_sizes(kDim, w, h, d, R);
    static_assert(8 * sizeof(unsigned) + kWsAlign <= kCtlBytes, "the control words follow the shifted pieces");
    char* q = reinterpret_cast<char*>(((uintptr_t)ws + kWsAlign - 1) & ~(uintptr_t)(kWsAlign - 1));
    auto take = [&](size_t bytes) {
        char* r = q;
        q += bytes;
        return r;
    };
    DanBlk p{};
    p.A = deltas;
    for (int v = 0; v < 2; v++) p.V[v] = take(z.field);
    for (int v = 0; v < 2; v++) p.DB[v] = take(z.down);
    for (int v = 0; v < 2; v++) p.XR[v] = reinterpret_cast<uint2*>(take(z.side));
    for (int v = 0; v < 2; v++) p.XL[v] = reinterpret_cast<uint2*>(take(z.side));
    p.state = reinterpret_cast<unsigned*>(take(z.list));
    for (int v = 0; v < 2; v++) p.dirty[v] = reinterpret_cast<uint8_t*>(take(z.flag));
    p.stamp = reinterpret_cast<int*>(take(z.list));
    p.wl[0] = reinterpret_cast<int*>(take(z.list));
    p.wl[1] = reinterpret_cast<int*>(take(z.list));
    p.ctl = reinterpret_cast<unsigned*>(q);
    p.err = err;
    p.w = w;
    p.h = h;
    p.d = d;
    p.R = R;
    p.nc = (h + R - 1) / R;
    p.nx = (w + 32 * S - 1) / (32 * S);
    p.cw = cw;
    p.rest = !initial;
    if (kDim == 2) {
        p.dir = 1;
        p.zfirst = 0;
        p.nchain = 1;
        return run_phase<kDim, S>(p, deltas, st);
    }
    // slices 1..d-1 pull from the slice before, then d-2..0 from the slice after
    p.dir = 1;
    p.zfirst = 1;
    p.nchain = d - 1;
    if (!run_phase<kDim, S>(p, deltas, st)) return false;
    p.dir = -1;
    p.zfirst = d - 2;
    return run_phase<kDim, S>(p, deltas, st);
}

size_t danielsson_workspace_bytes(int dim, int w, int h, int d)
{
    if (dim == 3 && d < 2) return 0;   // nothing to sweep
    const int R = dan_blocks_rows(dim, w, h, d);
    if (R >= kDanSerial || w > kBlkMaxWidth) return 0;
    return dan_blocks_workspace_bytes(dim, w, h, d, R);
}

bool run_danielsson(int dim, void* deltas, int w, int h, int d, int cw, bool initial, void* ws, size_t ws_bytes,
                    int* err, cudaStream_t st)
{
    const int R = dan_blocks_rows(dim, w, h, d);
    if (ws && R < kDanSerial && ws_bytes >= dan_blocks_workspace_bytes(dim, w, h, d, R) &&
        launch_danielsson_blocks(dim, deltas, w, h, d, cw, R, initial, ws, err, st))
        return true;
    launch_danielsson(dim, deltas, w, h, d, cw, st);
    return false;
}

bool launch_danielsson_blocks(int dim, void* deltas, int w, int h, int d, int cw, int R, bool initial, void* ws, int* err,
                              cudaStream_t st)
{
    if (dim == 3 && d < 2) return true;   // the reference's slice loops do not run
    if (w > kBlkMaxWidth) return false;
    R = min(R, kBlkMaxRows);
    ProfScope ps("danielsson_blocks", st);
    switch (dan_blocks_s(dim, w)) {
        case 2:
            return dim == 2 ? run_all<2, 2>(w, h, 1, cw, R, initial, deltas, ws, err, st)
                            : run_all<3, 2>(w, h, d, cw, R, initial, deltas, ws, err, st);
        case 4:
            return dim == 2 ? run_all<2, 4>(w, h, 1, cw, R, initial, deltas, ws, err, st)
                            : run_all<3, 4>(w, h, d, cw, R, initial, deltas, ws, err, st);
        default:
            return dim == 2 ? run_all<2, 8>(w, h, 1, cw, R, initial, deltas, ws, err, st)
                            : run_all<3, 8>(w, h, d, cw, R, initial, deltas, ws, err, st);
    }
}

}  // namespace dolk
