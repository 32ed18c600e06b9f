// row.cuh -- rows of delta cells held by warps, and the reference's serial x
// passes over them, exact.
//
// Every delta sweep ends each row with serial passes along x (Danielsson
// DistanceOcclusionLib.cpp:722-738, FastSweep :669-693, :2245-2255):
//
//     v[i] = closer(v[i], v[i-dir] shifted by -dir*cw in x)      (+ a fixed
//            candidate D[i] from the previous row in FastSweep 2D)
//
// `closer` keeps the incumbent on ties, and which of two deltas is closer can
// change along the row, so this is not an associative scan: the result depends
// on the exact chain of replacements.  It is a composition of per-cell
// functions, so a row cut into segments (S cells per lane) is solved by
// iterating the segments' inputs to the unique fixed point:
//
//   round 0   a segment's input is its predecessor's boundary cell as it was
//             before the pass;
//   round r   its input is the output of the nearest segment before it that is
//             not transparent (transparent: the input took the first cell and
//             comes out at the end, shifted by the segment length), shifted
//             across the transparent segments in between;
//   stop      when no segment would see another input.  An input only matters
//             if it takes the segment's first cell: one that does not is as
//             good as any other that does not.
//
// At the stop every segment saw what the serial pass would feed it, so the
// result is bit-identical.  It terminates: if segments 0..k are right after
// round r, segment k+1 is right after round r+1.
//
// In a warp the exchange is a shuffle and the stop a vote.  Rows wider than 32 S
// cells take several warps, each settled by itself from a first input of
// "none"; the warps then exchange their outputs through shared memory by the
// same rules, one barrier per exchange.
//
// What a cell needs for that is kept
// beside it in registers: x in the high half of a word (a shift is one add and
// wraps as int16 does), the sum of the other components' squares, and its
// squared length.
#pragma once

#include <limits.h>

#include <type_traits>

#include "common.cuh"

namespace dolk {

#define DOL_DI __device__ __forceinline__

// S cells of a lane.  xy: x in the high half, y in the low; W: y^2 (+ z^2);
// L: squared length, all in the reference's 32-bit arithmetic.
template <int DIM, int S>
struct Cells {
    uint32_t xy[S];
    uint32_t W[S];
    int L[S];
    int z[S];   // 3D only
};

// A candidate on its way along the row
struct Chain {
    uint32_t xy, W;
    int z;
};

// Cells past the row's end, and the input of its first cell: never replaced,
// and one step away exactly as long as an int can be, so that it replaces
// nothing.
DOL_DI Chain chain_none(int cw) { return Chain{0u, (uint32_t)INT_MAX - (uint32_t)(cw * cw), 0}; }

template <int DIM, int S>
DOL_DI void set_none(Cells<DIM, S>& c, int s, int cw)
{
    c.xy[s] = 0;
    c.W[s] = (uint32_t)INT_MAX - (uint32_t)(cw * cw);
    c.L[s] = INT_MIN;
    c.z[s] = 0;
}

template <int DIM>
DOL_DI uint32_t w_of(uint32_t xy, int z)
{
    const int y = (int)(int16_t)xy;
    return DIM == 3 ? (uint32_t)(y * y) + (uint32_t)(z * z) : (uint32_t)(y * y);
}
DOL_DI int len_of(uint32_t xy, uint32_t W)
{
    const int x = (int)xy >> 16;
    return (int)((uint32_t)(x * x) + W);
}
// y + dy, wrapping as int16
DOL_DI uint32_t y_shift(uint32_t xy, int dy) { return __byte_perm(xy, xy + (uint32_t)dy, 0x3254); }

// c[s] = closer(c[s], (xy, z))
template <int DIM, int S>
DOL_DI void consider(Cells<DIM, S>& c, int s, uint32_t xy, int z)
{
    const uint32_t W = w_of<DIM>(xy, z);
    const int l = len_of(xy, W);
    const bool t = c.L[s] > l;
    c.xy[s] = t ? xy : c.xy[s];
    c.W[s] = t ? W : c.W[s];
    c.L[s] = t ? l : c.L[s];
    if (DIM == 3) c.z[s] = t ? z : c.z[s];
}

// FastSweep 2D's candidates from the previous row's diagonal
template <int S>
struct Diag {
    uint32_t xy[S];
    uint32_t W[S];
    int L[S];   // INT_MAX: none
};
struct NoDiag {};

template <int DIM>
DOL_DI Chain shfl_chain(const Chain& c, int src)
{
    Chain r;
    r.xy = __shfl_sync(0xFFFFFFFFu, c.xy, src);
    r.W = __shfl_sync(0xFFFFFFFFu, c.W, src);
    r.z = DIM == 3 ? __shfl_sync(0xFFFFFFFFu, c.z, src) : 0;
    return r;
}

template <int DIM>
DOL_DI bool same_chain(const Chain& a, const Chain& b)
{
    return a.xy == b.xy && (DIM == 2 || a.z == b.z);
}

// c = closer(c, p shifted by dy in y), the result in p: the row of a sweep from
// the row before it (p) and its own cells (c)
template <int DIM, int S>
DOL_DI void merge_y(Cells<DIM, S>& p, const Cells<DIM, S>& c, int dy)
{
#pragma unroll
    for (int s = 0; s < S; s++) {
        const uint32_t xy = y_shift(p.xy[s], dy);
        const uint32_t W = w_of<DIM>(xy, DIM == 3 ? p.z[s] : 0);
        const int l = (int)(W + ((uint32_t)p.L[s] - p.W[s]));   // its x did not change
        const bool t = c.L[s] > l;
        p.xy[s] = t ? xy : c.xy[s];
        p.W[s] = t ? W : c.W[s];
        p.L[s] = t ? l : c.L[s];
        if (DIM == 3) p.z[s] = t ? p.z[s] : c.z[s];
    }
}

// One pass of a warp over its 32 S cells, in place.
//
// Most rows of a sweep are changed by a pass in a few cells or none (a row that
// took the relaxed row before it has little left to relax: on the 256^3 volume
// of boxes and spheres 61 % of the passes change nothing and 95 % need one
// round), so every cell is first tested against its neighbour as it stands, all
// of them at once; only a row where one of those tests succeeds is walked.
template <int DIM, int S, int DIR, class D>
struct WarpPass {
    Chain in, out;   // this lane's input and output
    bool e;          // the input took the first cell
    bool walked;     // O holds the row before the pass
    uint32_t step;   // shift of one cell, in the high half
    Cells<DIM, S> O;

    static constexpr bool kDiag = !std::is_same<D, NoDiag>::value;
    static constexpr int kFirst = DIR > 0 ? 0 : S - 1, kLast = DIR > 0 ? S - 1 : 0;

    DOL_DI bool first_lane(int lane) const { return lane == (DIR > 0 ? 0 : 31); }

    // the segment's serial pass from `in`: O -> V
    DOL_DI void walk(Cells<DIM, S>& V, const D& diag)
    {
        Chain c = in;
#pragma unroll
        for (int u = 0; u < S; u++) {
            const int s = DIR > 0 ? u : S - 1 - u;
            const uint32_t xy = c.xy + step;
            const int l = len_of(xy, c.W);
            const bool t = O.L[s] > l;
            if (u == 0) e = t;
            c.xy = t ? xy : O.xy[s];
            c.W = t ? c.W : O.W[s];
            if (DIM == 3) c.z = t ? c.z : O.z[s];
            int L = t ? l : O.L[s];
            if constexpr (kDiag) {
                const bool td = L > diag.L[s];
                c.xy = td ? diag.xy[s] : c.xy;
                c.W = td ? diag.W[s] : c.W;
                L = td ? diag.L[s] : L;
            }
            V.xy[s] = c.xy;
            V.W[s] = c.W;
            V.L[s] = L;
            if (DIM == 3) V.z[s] = c.z;
        }
        out = c;
    }

    // the pass from first-lane input `win`; leaves `out` right for every lane
    DOL_DI void run(Cells<DIM, S>& V, const D& diag, const Chain& win, int cw)
    {
        const int lane = threadIdx.x & 31, pl = DIR > 0 ? (lane + 31) & 31 : (lane + 1) & 31;
        step = (uint32_t)(-DIR * cw) << 16;
        out = Chain{V.xy[kLast], V.W[kLast], DIM == 3 ? V.z[kLast] : 0};
        in.xy = __shfl_sync(0xFFFFFFFFu, out.xy, pl);
        in.W = __shfl_sync(0xFFFFFFFFu, out.W, pl);
        if (first_lane(lane)) {
            in.xy = win.xy;
            in.W = win.W;
        }
        bool any = false;
#pragma unroll
        for (int u = 0; u < S; u++) {
            const int s = DIR > 0 ? u : S - 1 - u, q = DIR > 0 ? s - 1 : s + 1;
            const uint32_t xy = (u ? V.xy[u ? q : s] : in.xy) + step;
            const int l = len_of(xy, u ? V.W[u ? q : s] : in.W);
            any |= V.L[s] > l;
            if constexpr (kDiag) any |= V.L[s] > diag.L[s];
        }
        e = false;
        walked = false;
        if (!__any_sync(0xFFFFFFFFu, any)) return;
        walked = true;
        O = V;
        in.z = DIM == 3 ? __shfl_sync(0xFFFFFFFFu, out.z, pl) : 0;
        if (DIM == 3 && first_lane(lane)) in.z = win.z;
        const Chain edge = out;
        walk(V, diag);
        // every input was its predecessor's edge cell as it stood: right unless an edge cell changed
        if (!__any_sync(0xFFFFFFFFu, !same_chain<DIM>(edge, out))) return;
        guess(V, diag, win);
        settle(V, diag, win);
    }

    // Better inputs before the rounds, for chains that run over several lanes: a
    // scan of `closer` over the lanes' outputs.  It is what the serial pass
    // gives unless a candidate that some lane drops would have come first
    // again further on; the rounds find out.
    DOL_DI void guess(Cells<DIM, S>& V, const D& diag, const Chain& win)
    {
        const int lane = threadIdx.x & 31;
        Chain c = out;
        int l = len_of(c.xy, c.W);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            Chain q;
            const int src = DIR > 0 ? (lane - o) & 31 : (lane + o) & 31;
            q = shfl_chain<DIM>(c, src);
            q.xy += (uint32_t)(S * o) * step;
            const int ql = len_of(q.xy, q.W);
            const bool t = (DIR > 0 ? lane >= o : lane + o < 32) && l > ql;
            c.xy = t ? q.xy : c.xy;
            c.W = t ? q.W : c.W;
            if (DIM == 3) c.z = t ? q.z : c.z;
            l = t ? ql : l;
        }
        Chain g = shfl_chain<DIM>(c, DIR > 0 ? (lane + 31) & 31 : (lane + 1) & 31);
        if (first_lane(lane)) g = win;
        const bool te = O.L[kFirst] > len_of(g.xy + step, g.W);
        if (te ? !e || !same_chain<DIM>(g, in) : e) {
            in = g;
            walk(V, diag);
        }
    }

    // rounds until no lane would see another input; win: the first lane's
    DOL_DI void settle(Cells<DIM, S>& V, const D& diag, const Chain& win)
    {
        const int lane = threadIdx.x & 31;
        if (!walked) {
            walked = true;
            O = V;
        }
        for (int r = 0; r < 36; r++) {   // (the fixed point is reached within 33 rounds)
            const bool trans = e && out.xy == in.xy + (uint32_t)S * step && (DIM == 2 || out.z == in.z);
            const uint32_t nt = __ballot_sync(0xFFFFFFFFu, !trans);
            int j, gap;   // the nearest lane before this one that is not transparent
            if (DIR > 0) {
                const uint32_t m = nt & ((1u << lane) - 1u);
                j = m ? 31 - __clz(m) : -1;
                gap = lane - j - 1;
            } else {
                const uint32_t m = lane == 31 ? 0u : nt >> (lane + 1);
                j = m ? lane + __ffs(m) : 32;
                gap = j - lane - 1;
            }
            const bool from_win = j < 0 || j > 31;
            Chain c = shfl_chain<DIM>(out, j & 31);
            if (from_win) c = win;
            c.xy += (uint32_t)(S * gap) * step;
            const bool te = O.L[kFirst] > len_of(c.xy + step, c.W);
            const bool need = te ? !e || !same_chain<DIM>(c, in) : e;
            if (!__any_sync(0xFFFFFFFFu, need)) break;
            if (need) {
                in = c;
                walk(V, diag);
            }
        }
    }
};

// What the warps of a row exchange, by parity of the exchange
struct WarpPost {
    uint32_t oxy, oW, ixy;
    int oz, iz, L;
    uint32_t flags;   // bit 0: transparent, bit 1: its input took the first cell
    uint32_t pad;
};
template <int NW>
struct RowShared {
    WarpPost post[2][NW];
    int bar;   // the barrier of the row's NW warps (0: the CTA's, which they then are)

    DOL_DI void sync() const { asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(32 * NW) : "memory"); }
};
template <>
struct RowShared<1> {};

// One pass over a row of NW warps (32 S cells each), in place.  `par`: the
// exchange parity, kept by the caller over all the passes that use `sh`.
// `first` (one warp only): the input of the row's first cell.
template <int DIM, int S, int NW, int DIR, class D>
DOL_DI void row_pass_w(Cells<DIM, S>& V, const D& diag, int cw, RowShared<NW>& sh, int& par, const Chain& first)
{
    using PassT = WarpPass<DIM, S, DIR, D>;
    PassT p;
    Chain win = NW > 1 ? chain_none(cw) : first;
    const int first_L = V.L[PassT::kFirst];
    p.run(V, diag, win, cw);
    if constexpr (NW > 1) {
        const int lane = threadIdx.x & 31, wi = (threadIdx.x >> 5) & (NW - 1);
        const uint32_t span = (uint32_t)(32 * S) * p.step;
        for (int r = 0; r < NW + 3; r++, par ^= 1) {
            // the first lane in scan order knows the warp's input, the last its output
            const int fl = DIR > 0 ? 0 : 31, ll = 31 - fl;
            const bool e0 = __shfl_sync(0xFFFFFFFFu, (int)p.e, fl) != 0;
            if (lane == ll) {
                WarpPost& o = sh.post[par][wi];
                o.oxy = p.out.xy;
                o.oW = p.out.W;
                o.oz = p.out.z;
                const bool trans = e0 && p.out.xy == win.xy + span && (DIM == 2 || p.out.z == win.z);
                o.flags = (trans ? 1u : 0u) | (e0 ? 2u : 0u);
                o.ixy = win.xy;
                o.iz = win.z;
            }
            if (lane == fl) sh.post[par][wi].L = first_L;
            sh.sync();
            // every warp looks at all of them: lane k decides for warp k
            const int k = lane < NW ? lane : NW - 1;
            const WarpPost mine = sh.post[par][k];
            const uint32_t nt = __ballot_sync(0xFFFFFFFFu, lane < NW && !(mine.flags & 1u));
            int j, gap;
            if (DIR > 0) {
                const uint32_t m = nt & ((1u << k) - 1u);
                j = m ? 31 - __clz(m) : -1;
                gap = k - j - 1;
            } else {
                const uint32_t m = k == 31 ? 0u : nt >> (k + 1);
                j = m ? k + __ffs(m) : NW;
                gap = j - k - 1;
            }
            Chain c = chain_none(cw);
            if (j >= 0 && j < NW) {
                const WarpPost& o = sh.post[par][j];
                c = Chain{o.oxy + (uint32_t)gap * span, o.oW, o.oz};
            }
            const bool e = (mine.flags & 2u) != 0;
            const bool te = mine.L > len_of(c.xy + p.step, c.W);
            const bool need = lane < NW && (te ? !e || c.xy != mine.ixy || (DIM == 3 && c.z != mine.iz) : e);
            const uint32_t needs = __ballot_sync(0xFFFFFFFFu, need);
            if (!needs) {
                par ^= 1;
                break;
            }
            const Chain nw = shfl_chain<DIM>(c, wi);
            if ((needs >> wi) & 1u) {
                win = nw;
                p.settle(V, diag, win);
            }
        }
    }
}

// ---- rows in global memory -----------------------------------------------------------
//
// A warp's part of a row is 32 S cells of 4 (2D) or 6 (3D) bytes at any 4- or
// 2-byte boundary.  It moves as the aligned 16-byte pieces that hold it,
// coalesced over the warp, and is turned through a strip of shared memory into
// S cells per lane.  Loads are asynchronous copies into one of LOADS strips
// (a row in flight takes no registers), stores go through one more.
// Pieces that reach past the array's ends, and pieces that hold a neighbour's
// cells when storing, go by halves.
template <int DIM, int S, int LOADS>   // LOADS: rows in flight at a time
struct RowIO {
    static constexpr int kCell = DIM == 3 ? 6 : 4;
    static constexpr int kLane = S * kCell;                       // bytes per lane
    static constexpr int kPieces = (32 * kLane + 15 + 511) / 512;   // per lane
    static constexpr int kWords = kLane / 4;
    static constexpr int kStrip = (32 * kLane + 16 + 15) / 16 * 16 + 16;   // bytes of shared memory per warp
    static_assert(kLane % 4 == 0, "whole words per lane");

    static constexpr int kStrips = LOADS + 1;
    static constexpr size_t kBytes = (size_t)kStrips * kStrip;   // shared memory per warp

    unsigned char* strips;   // this warp's
    int cells;               // of this warp in a row (<= 32 S, may be <= 0)

    DOL_DI static void copy16(unsigned char* dst, const unsigned char* src)
    {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                     "l"(src)
                     : "memory");
    }

    static __device__ __noinline__ uint4 load_edge(const unsigned char* a, const unsigned char* lo, const unsigned char* hi)
    {
        uint32_t w[4] = {0, 0, 0, 0};
        for (int i = 0; i < 8; i++) {
            const unsigned char* q = a + 2 * i;
            if (q >= lo && q + 2 <= hi)
                w[i >> 1] |= (uint32_t)__ldcg(reinterpret_cast<const unsigned short*>(q)) << (16 * (i & 1));
        }
        return make_uint4(w[0], w[1], w[2], w[3]);
    }

    // a warp's full part of a row at a 16-byte boundary: whole pieces, no edges
    DOL_DI bool whole(const unsigned char* a) const { return ((uintptr_t)a & 15) == 0 && cells == 32 * S; }

    // start loading a row into strip k; a: the address of the warp's first cell;
    // [lo, hi): the array
    DOL_DI void fetch(int k, const unsigned char* a, const unsigned char* lo, const unsigned char* hi) const
    {
        const int lane = threadIdx.x & 31;
        unsigned char* strip = strips + k * kStrip;
        const int sh = (int)((uintptr_t)a & 15), end = sh + cells * kCell;
        const unsigned char* b = a - sh;
        __syncwarp();   // the strip's last use
        if (whole(a)) {
#pragma unroll
            for (int i = 0; i < kPieces; i++) {
                const int off = 16 * (lane + 32 * i);
                if (32 * kLane >= 512 * (i + 1) || off < 32 * kLane) copy16(strip + off, a + off);
            }
            return;
        }
#pragma unroll
        for (int i = 0; i < kPieces; i++) {
            const int off = 16 * (lane + 32 * i);
            if (off < end && cells > 0) {
                const unsigned char* q = b + off;
                if (q >= lo && q + 16 <= hi) copy16(strip + off, q);
                else *reinterpret_cast<uint4*>(strip + off) = load_edge(q, lo, hi);
            }
        }
    }

    // the lane's words of the row in strip k
    DOL_DI void words(uint32_t (&w)[kWords], int k, const unsigned char* a) const
    {
        const int lane = threadIdx.x & 31;
        const int sh = (int)((uintptr_t)a & 15);
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
        const unsigned char* strip = strips + k * kStrip;
        const unsigned char* q = strip + lane * kLane + (sh & ~3);
        if (kLane % 16 == 0 && sh == 0) {
#pragma unroll
            for (int i = 0; i < kWords / 4; i++) {
                const uint4 v = reinterpret_cast<const uint4*>(q)[i];
                w[4 * i] = v.x;
                w[4 * i + 1] = v.y;
                w[4 * i + 2] = v.z;
                w[4 * i + 3] = v.w;
            }
        } else {
            const uint32_t* q4 = reinterpret_cast<const uint32_t*>(q);
#pragma unroll
            for (int i = 0; i < kWords; i++) w[i] = q4[i];
            if (sh & 2) {   // 3D rows of odd cells
                const uint32_t tail = q4[kWords];
#pragma unroll
                for (int i = 0; i < kWords; i++)
                    w[i] = __funnelshift_r(w[i], i + 1 < kWords ? w[i + 1 < kWords ? i + 1 : i] : tail, 16);
            }
        }
    }

    // words <-> (xy, z)
    static DOL_DI void split(const uint32_t (&w)[kWords], uint32_t (&xy)[S], int (&z)[S])
    {
        if constexpr (DIM == 2) {
#pragma unroll
            for (int s = 0; s < S; s++) {
                xy[s] = __byte_perm(w[s], 0, 0x1032);
                z[s] = 0;
            }
        } else {
#pragma unroll
            for (int k = 0; k < S / 2; k++) {
                const uint32_t a = w[3 * k], b = w[3 * k + 1], c = w[3 * k + 2];   // y0:x0, x1:z0, z1:y1
                xy[2 * k] = __byte_perm(a, 0, 0x1032);
                z[2 * k] = (int)(int16_t)b;
                xy[2 * k + 1] = __byte_perm(b, c, 0x3254);
                z[2 * k + 1] = (int)c >> 16;
            }
        }
    }
    static DOL_DI void join(uint32_t (&w)[kWords], const uint32_t (&xy)[S], const int (&z)[S])
    {
        if constexpr (DIM == 2) {
#pragma unroll
            for (int s = 0; s < S; s++) w[s] = __byte_perm(xy[s], 0, 0x1032);
        } else {
#pragma unroll
            for (int k = 0; k < S / 2; k++) {
                w[3 * k] = __byte_perm(xy[2 * k], 0, 0x1032);
                w[3 * k + 1] = __byte_perm((uint32_t)z[2 * k], xy[2 * k + 1], 0x7610);
                w[3 * k + 2] = __byte_perm(xy[2 * k + 1], (uint32_t)z[2 * k + 1], 0x5410);
            }
        }
    }

    // number of this lane's cells that lie in the row
    DOL_DI int live() const { return max(0, min(S, cells - (int)(threadIdx.x & 31) * S)); }

    // the row in strip k as cells, those past its end as "none"
    DOL_DI void cells_of(Cells<DIM, S>& c, int k, const unsigned char* a, int cw) const
    {
        uint32_t w[kWords];
        words(w, k, a);
        split(w, c.xy, c.z);
#pragma unroll
        for (int s = 0; s < S; s++) {
            c.W[s] = w_of<DIM>(c.xy[s], c.z[s]);
            c.L[s] = len_of(c.xy[s], c.W[s]);
        }
        const int n = live();
        if (n < S) {
#pragma unroll
            for (int s = 0; s < S; s++)
                if (s >= n) set_none(c, s, cw);
        }
    }

    // store the lane's words at a
    DOL_DI void put(unsigned char* a, const uint32_t (&w)[kWords]) const
    {
        const int lane = threadIdx.x & 31;
        const int sh = (int)((uintptr_t)a & 15), end = sh + cells * kCell;
        unsigned char* strip = strips + (kStrips - 1) * kStrip;
        __syncwarp();   // the strip's last use
        unsigned char* q = strip + lane * kLane + sh;
        if (kLane % 16 == 0 && sh == 0) {
#pragma unroll
            for (int i = 0; i < kWords / 4; i++)
                reinterpret_cast<uint4*>(q)[i] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
        } else if (!(sh & 2)) {
#pragma unroll
            for (int i = 0; i < kWords; i++) reinterpret_cast<uint32_t*>(q)[i] = w[i];
        } else {
#pragma unroll
            for (int i = 0; i < kWords; i++) {
                reinterpret_cast<unsigned short*>(q)[2 * i] = (unsigned short)w[i];
                reinterpret_cast<unsigned short*>(q)[2 * i + 1] = (unsigned short)(w[i] >> 16);
            }
        }
        __syncwarp();
        unsigned char* b = a - sh;
        if (whole(a)) {
#pragma unroll
            for (int i = 0; i < kPieces; i++) {
                const int off = 16 * (lane + 32 * i);
                if (off < 32 * kLane)
                    *reinterpret_cast<uint4*>(a + off) = *reinterpret_cast<const uint4*>(strip + off);
            }
            return;
        }
#pragma unroll
        for (int i = 0; i < kPieces; i++) {
            const int off = 16 * (lane + 32 * i);
            if (off >= sh && off + 16 <= end) {
                *reinterpret_cast<uint4*>(b + off) = *reinterpret_cast<const uint4*>(strip + off);
            } else if (off + 16 > sh && off < end) {
                for (int k = max(off, sh); k < min(off + 16, end); k += 2)
                    *reinterpret_cast<unsigned short*>(b + k) = *reinterpret_cast<const unsigned short*>(strip + k);
            }
        }
    }
    DOL_DI void put_cells(unsigned char* a, const Cells<DIM, S>& c) const
    {
        uint32_t w[kWords];
        join(w, c.xy, c.z);
        put(a, w);
    }
};

}  // namespace dolk
