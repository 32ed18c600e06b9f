// k_fastsweep3.cu -- FastSweep 3D (DistanceOcclusionLib.cpp:2186-2260) as one
// launch of columns that stream along z.
//
// An octant sweep replaces a cell by the closest of itself and its three
// neighbours of the same sweep, in z, y, x order (:2216-2255); the first row and
// the first slice keep their cells.  So a cell needs (x-1, y, z), (x, y-1, z),
// (x, y, z-1) in sweep order and nothing else, and a sweep is a wavefront of
// w + h + d steps.  The field is cut into columns of 16 x 16 cells over all
// slices; a CTA takes a (sweep, column) and marches: at step s lane (i, j)
// updates slice s - i - j.  The cell behind is the lane's own last value, the
// other two come from the lanes beside it through shared memory.
//   * Faces.  A column's outer lanes write their cells, as they are made, to face
//     words in global memory (8 bytes: cell and the sweep's tag), which the next
//     columns' face warp polls: the data is its own flag, so a column runs about
//     16 steps and one trip through L2 behind the one before it.  Words are
//     indexed by step, so a step's words lie side by side.
//   * The field.  Before the sweeps the cells are copied into tiles, a column's
//     slice side by side (x and y words, then z), so that any width stages by
//     16-byte pieces in order; after them they are copied back.  Only the
//     column's own CTA touches its cells, so sweeps are ordered by a progress
//     count per sweep and column.  Two warps stage chunks of 8 slices into a ring
//     in shared memory, two more store what is finished.  A chunk of sweep s
//     waits until the column's own sweep s - 1 is past it (all of it where z turns
//     round), and likewise the columns that read this one's face words in sweep
//     s - 1, whose words it is about to overwrite.
//   * Columns are claimed in order of sweep and diagonal, so a claimed column
//     waits only for earlier ones, and sweeps overlap as far as the waits allow.
// Every wait is bounded.
//
// Lengths.  A neighbour at offset o along an axis has length L + o (2 c + o), c
// its component: one multiply-add instead of three.  That holds while no
// component wraps at 16 bits.  A cell's component differs from that of the cell it
// came from by cw times the cells between them, so cells that start further than
// cw times the field's extent from the limits never get there; the copy into
// tiles checks that, and a field with others is swept in the wrapping form.
//
// What bounds it: latency along the wavefront -- a step is ~0.2 us (two shared
// loads, two dependent compares with their selects, a barrier), a hop to the next
// column ~16 steps and ~1 us through L2, a sweep that turns y starts after the
// one before has crossed the field.  The copies to and from tiles are 0.1 ms.
// 256^3 boxes and spheres, eight sweeps: 1.96 ms; 3.3 ms with a warp per slice
// that passes whole rows on, two sweeps at a time; 11.2 ms with a CTA per slice,
// one sweep per launch and a flag per row.  255 x 256 x 256: 1.95 ms (7.7 ms with
// cells staged from the field itself, whose rows of 6-byte cells then lie on any
// even byte).  Columns of 16 x 8 cells: 2.5 ms (more hops); three such CTAs per
// SM gained nothing.  Face words taken 2 or 8 steps at a time: 2.1 ms; by two
// warps in turn: 2.1 ms.
#include "common.cuh"
#include "kernels.h"

namespace dolk {

constexpr int kTX = 16, kTY = 16;         // a column
constexpr int kCompute = kTX * kTY;       // its lanes
constexpr int kLoaders = 2, kStorers = 2;   // warps that take chunks in turn
constexpr int kFs3Threads = kCompute + 32 * (1 + kLoaders + kStorers);   // (1: the face warp)
constexpr int kChunk = 8, kRing = 56;     // slices staged at a time, slices in shared memory
constexpr int kSliceZ = kCompute * 4;     // a tile: x and y of its cells, then z
constexpr int kSliceBytes = kCompute * 6;
constexpr int kFaceRing = 32;             // steps of face words in shared memory
constexpr int kFaceLanes = kTX + kTY;

struct Fs3 {
    unsigned char* cells;           // the field
    unsigned char* tiles;           // per column: [chunks * kChunk] slices
    unsigned* counter;              // columns taken
    int* wraps;                     // a component may wrap
    int* progress;                  // per sweep, column and storing warp: chunks stored
    unsigned long long* xface;      // per column: [d + kTY][kTY]
    unsigned long long* yface;      // per column: [d + kTX][kTX]
    int* err;
    int w, h, d, cw;
    int nbx, nby, nch;
    int safe;                       // largest component that cannot wrap on its way
    int stall;                      // sweep whose waits are made to run out, or -1
    unsigned limit;                 // polls of a wait
};

struct Fs3Smem {
    unsigned char ring[kRing * kSliceBytes];   // slice z at z % kRing
    int4 face[kFaceRing][kFaceLanes];    // by step: rows above (by column), columns beside (by row)
    int4 edge[2][kTY][kTX];              // the lanes' cells of the step before
    int item;
    volatile int step;                   // steps done
    volatile int staged[kLoaders];       // per loading warp: its last chunk there + 1
    volatile int faces;                  // steps whose face cells are there
    volatile int stored[kStorers];       // per storing warp: chunks stored
    volatile int broken;                 // a wait inside the CTA has given up
};
constexpr int kAll = 1 << 30;             // faces: all there are

__device__ __forceinline__ int acquire_load(const int* p)
{
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// until *v >= need.  The other side gets there, its own waits being bounded; the
// bound here only keeps a logic error from looping on the device.  A waiting warp
// sleeps between polls, so as to leave its issue slots to those it waits for.
template <int kSleep>
__device__ __forceinline__ int smem_wait(const volatile int* v, int need, Fs3Smem& sm, int* err)
{
    auto load = [&] {
        int x;
        asm volatile("ld.acquire.cta.shared.s32 %0, [%1];"
                     : "=r"(x)
                     : "r"((uint32_t)__cvta_generic_to_shared(const_cast<const int*>(v)))
                     : "memory");
        return x;
    };
    int x = load();
    for (unsigned polls = 0; x < need; polls++) {
        if (sm.broken || polls >= (1u << 25)) {
            atomicExch(err, 1);
            sm.broken = 1;
            break;
        }
        if (kSleep >= 50 || polls > 16) __nanosleep(kSleep);
        x = load();
    }
    return x;
}

__device__ __forceinline__ void smem_post(const volatile int* v, int x)
{
    asm volatile("st.release.cta.shared.s32 [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(const_cast<const int*>(v))),
                 "r"(x)
                 : "memory");
}

// One sweep's view of a column
struct Fs3Column {
    int sweep, tx, ty, col;
    int x0, y0, ni, nj;      // cells in memory
    int sx, sy, sz;          // directions: 1 = downwards
    int bx, by;              // place in sweep order

    __device__ Fs3Column(const Fs3& p, int item)
    {
        const int n = p.nbx * p.nby;
        sweep = item / n;
        int r = item - sweep * n;
        sx = sweep & 1;
        sy = (sweep >> 1) & 1;
        sz = (sweep >> 2) & 1;
        // r-th in order of diagonals bx + by
        int l = 0;
        for (;; l++) {
            const int lo = max(0, l - (p.nby - 1)), hi = min(l, p.nbx - 1);
            const int c = hi - lo + 1;
            if (r < c) {
                bx = lo + r;
                by = l - bx;
                break;
            }
            r -= c;
        }
        tx = sx ? p.nbx - 1 - bx : bx;
        ty = sy ? p.nby - 1 - by : by;
        col = ty * p.nbx + tx;
        x0 = tx * kTX;
        y0 = ty * kTY;
        ni = min(kTX, p.w - x0);
        nj = min(kTY, p.h - y0);
    }
    // chunk q in sweep order: its first slice in memory, and in sweep order, where the next starts
    __device__ int chunk_z(const Fs3& p, int q) const { return kChunk * (sz ? p.nch - 1 - q : q); }
    __device__ int chunk_end(const Fs3& p, int q) const
    {
        return sz ? p.d - kChunk * (p.nch - 1 - q) : min(p.d, kChunk * (q + 1));
    }
};

struct Fs3Cell {
    int x, y, z, l;
};

__device__ __forceinline__ int len3(int x, int y, int z) { return (int)((unsigned)(x * x) + (unsigned)(y * y) + (unsigned)(z * z)); }

// loading warps: bring chunk after chunk into the ring
static __device__ void fs3_load(const Fs3& p, const Fs3Column& c, Fs3Smem& sm, int wl, bool& up)
{
    const int lane = threadIdx.x & 31;
    // what a chunk waits for: lane -> progress word
    const int* dep = nullptr;
    if (c.sweep > 0 && lane < 3 * kStorers) {
        const int* prog = p.progress + (long long)kStorers * (c.sweep - 1) * p.nbx * p.nby + lane % kStorers;
        const int ps = c.sweep - 1, nx = c.tx + (ps & 1 ? -1 : 1), ny = c.ty + (ps & 2 ? -1 : 1);
        const int which = lane / kStorers;
        if (which == 0) dep = prog + kStorers * c.col;
        else if (which == 1 && nx >= 0 && nx < p.nbx) dep = prog + kStorers * (c.ty * p.nbx + nx);
        else if (which == 2 && ny >= 0 && ny < p.nby) dep = prog + kStorers * (ny * p.nbx + c.tx);
    }
    const bool turned = c.sweep == 4;   // z turns round: the sweep before must be through
    const unsigned char* tiles = p.tiles + (long long)c.col * p.nch * kChunk * kSliceBytes + 16 * lane;
    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(sm.ring) + 16 * lane;
    int seen = dep ? -1 : INT_MAX;
    for (int q = wl; q < p.nch; q += kLoaders) {
        // room: the chunk that was in these slots is stored
        if (q >= kRing / kChunk) {
            const int old = q - kRing / kChunk;
            smem_wait<100>(&sm.stored[old % kStorers], old / kStorers + 1, sm, p.err);
        }
        if (c.sweep > 0) {
            const int by = lane % kStorers;   // chunks that storing warp `by` must have stored
            const int need = turned ? (p.nch - by + kStorers - 1) / kStorers : (q % kStorers == by ? q / kStorers + 1 : 0);
            const bool never = c.sweep == p.stall;
            for (unsigned polls = 0;; polls++) {
                if (seen < need) seen = acquire_load(dep);
                if (__all_sync(0xFFFFFFFFu, seen >= need && !never)) break;
                if (!up || polls >= p.limit) {
                    if (up && lane == 0) atomicExch(p.err, 1);
                    up = false;
                    break;
                }
                __nanosleep(64);
            }
            __syncwarp();
        }
        const int z0 = c.chunk_z(p, q);
        const unsigned char* src = tiles + (long long)z0 * kSliceBytes;
        const uint32_t dst = ring + (z0 % kRing) * kSliceBytes;
#pragma unroll
        for (int e = 0; e < kChunk * kSliceBytes; e += 512)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + e), "l"(src + e) : "memory");
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
        if (lane == 0) smem_post(&sm.staged[wl], q + 1);
    }
}

// storing warps: write chunk after chunk back
static __device__ void fs3_store(const Fs3& p, const Fs3Column& c, Fs3Smem& sm, int wl)
{
    const int lane = threadIdx.x & 31;
    unsigned char* tiles = p.tiles + (long long)c.col * p.nch * kChunk * kSliceBytes + 16 * lane;
    int* progress = p.progress + (long long)kStorers * (c.sweep * p.nbx * p.nby + c.col) + wl;
    for (int q = wl; q < p.nch; q += kStorers) {
        smem_wait<60>(&sm.step, c.chunk_end(p, q) + c.ni - 1 + c.nj - 1, sm, p.err);
        __syncwarp();
        const int z0 = c.chunk_z(p, q);
        const unsigned char* src = sm.ring + (z0 % kRing) * kSliceBytes + 16 * lane;
        unsigned char* dst = tiles + (long long)z0 * kSliceBytes;
        constexpr int kBatch = 8, kPieces = kChunk * kSliceBytes / 512;
        static_assert(kPieces % kBatch == 0, "");
#pragma unroll
        for (int e = 0; e < kPieces; e += kBatch) {
            uint4 v[kBatch];
#pragma unroll
            for (int u = 0; u < kBatch; u++) v[u] = *reinterpret_cast<const uint4*>(src + 512 * (e + u));
#pragma unroll
            for (int u = 0; u < kBatch; u++) *reinterpret_cast<uint4*>(dst + 512 * (e + u)) = v[u];
        }
        __syncwarp();
        if (lane == 0) {
            __threadfence();
            asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(progress), "r"(q / kStorers + 1) : "memory");
            smem_post(&sm.stored[wl], q / kStorers + 1);
        }
    }
}

// the face warp: lane i < kTX the row above the column, lane kTX + j the column beside it
static __device__ void fs3_faces(const Fs3& p, const Fs3Column& c, Fs3Smem& sm, bool& up)
{
    const int lane = threadIdx.x & 31;
    const int steps = p.d + c.ni - 1 + c.nj - 1;
    if (c.bx + c.by == 0) {
        if (lane == 0) sm.faces = kAll;
        return;
    }
    const unsigned tag = c.sweep == p.stall ? 0x10000u : (unsigned)c.sweep + 1;
    const bool above = lane < kTX;
    const int me = above ? lane : lane - kTX;
    const bool mine = above ? c.by > 0 && me < c.ni : c.bx > 0 && me < c.nj;
    const unsigned long long* src = nullptr;
    int pitch = 0;
    if (mine && above) {
        const int from = (c.ty + (c.sy ? 1 : -1)) * p.nbx + c.tx;
        src = p.yface + (long long)from * (p.d + kTX) * kTX + me;
        pitch = kTX;
    } else if (mine) {
        const int from = c.ty * p.nbx + c.tx + (c.sx ? 1 : -1);
        src = p.xface + (long long)from * (p.d + kTY) * kTY + me;
        pitch = kTY;
    }
    constexpr int kAhead = 4;
    unsigned polls = 0;
    for (int s = 0; s < steps;) {
        smem_wait<100>(&sm.step, s + kAhead - kFaceRing, sm, p.err);   // room for kAhead more
        unsigned long long v[kAhead];
        int n = 0;
#pragma unroll
        for (int u = 0; u < kAhead; u++) {
            v[u] = 0;
            if (mine && (unsigned)(s + u - me) < (unsigned)p.d)
                asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v[u]) : "l"(src + (long long)(s + u) * pitch)
                             : "memory");
        }
#pragma unroll
        for (int u = 0; u < kAhead; u++) {
            const bool wanted = mine && (unsigned)(s + u - me) < (unsigned)p.d;
            const bool ok = __all_sync(0xFFFFFFFFu, !wanted || (unsigned)(v[u] >> 48) == tag);
            if ((ok || !up) && n == u) {
                n = u + 1;
                const int x = (int)(int16_t)(v[u]), y = (int)(int16_t)(v[u] >> 16), z = (int)(int16_t)(v[u] >> 32);
                if (lane < kFaceLanes) sm.face[(s + u) % kFaceRing][lane] = make_int4(x, y, z, len3(x, y, z));
            }
        }
        if (n) {
            polls = 0;
            s += n;
            __syncwarp();
            if (lane == 0) smem_post(&sm.faces, s < steps ? s : kAll);
        } else if (++polls > p.limit) {
            if (up && lane == 0) atomicExch(p.err, 1);
            up = false;
        } else if (polls > 16) {
            __nanosleep(40);
        }
    }
}

// one cell's update in wrapping arithmetic
static __device__ __noinline__ Fs3Cell fs3_wrapping(Fs3Cell own, Fs3Cell back, Fs3Cell above, Fs3Cell left, int ox, int oy,
                                                    int oz, bool upd, bool has_left)
{
    auto take = [&](int x, int y, int z) {
        const int l = len3(x, y, z);
        if (own.l > l) own = Fs3Cell{x, y, z, l};
    };
    if (upd) {
        take(back.x, back.y, trunc16(back.z + oz));
        take(above.x, trunc16(above.y + oy), above.z);
        if (has_left) take(trunc16(left.x + ox), left.y, left.z);
    }
    return own;
}

__device__ __forceinline__ int4 lds_cell(uint32_t a)
{
    int4 v;
    asm volatile("ld.shared.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
    return v;
}
// What lane (i, j) needs at every step
struct Fs3Lane {
    int ij, nk;
    bool row_upd, has_left;
    uint32_t cell, cell_z;               // its cell in the ring's slice 0: x and y, z
    uint32_t slice_step, slice_wrap;     // to the next slice; where the ring goes on
    uint32_t above, above_mask, above_pitch, left, left_mask, left_pitch;   // by step
    uint32_t edge;                       // where its own go, odd steps (even ones kEdgeBytes on)
    unsigned long long *fx, *fy;         // face words by step of this lane's slice
    unsigned out_x, out_y;               // writes them
    unsigned long long tag;
    int ox, oy, oz;
};
constexpr uint32_t kEdgeBytes = kTX * kTY * 16;

// a cell's x and y, and z, from the ring
__device__ __forceinline__ void fs3_own(const Fs3Lane& q, uint32_t slice, uint32_t& xy, int& z)
{
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(xy) : "r"(q.cell + slice) : "memory");
    asm volatile("{ .reg .s16 h; ld.shared.s16 h, [%1]; cvt.s32.s16 %0, h; }" : "=r"(z) : "r"(q.cell_z + slice) : "memory");
}

// Steps s .. e-1.  A step's own cell is loaded before the barrier that ends the
// step before it (all of it is staged), its length and the cell behind worked in
// while the neighbours' cells are on their way.
template <bool kWraps>
__device__ __forceinline__ void fs3_steps(const Fs3Lane& q, Fs3Cell& v, uint32_t& slice, int s, int e)
{
    uint32_t xy;
    Fs3Cell n;
    fs3_own(q, slice, xy, n.z);
    uint32_t above = q.above + ((unsigned)s & q.above_mask) * q.above_pitch;
    uint32_t left = q.left + ((unsigned)s & q.left_mask) * q.left_pitch;
    for (;;) {
        const int4 ea = lds_cell(above), el = lds_cell(left);
        const int k = s - q.ij;
        const bool upd = q.row_upd && k > 0;
        n.x = (int)(int16_t)xy;
        n.y = (int)xy >> 16;
        n.l = len3(n.x, n.y, n.z);
        if (!kWraps) {
            const int lb = (int)((unsigned)v.l + (unsigned)q.oz * (unsigned)(2 * v.z + q.oz));
            const bool b = upd && n.l > lb;
            n.x = b ? v.x : n.x;
            n.y = b ? v.y : n.y;
            n.z = b ? v.z + q.oz : n.z;
            n.l = b ? lb : n.l;
            const int la = (int)((unsigned)ea.w + (unsigned)q.oy * (unsigned)(2 * ea.y + q.oy));
            const int ll = (int)((unsigned)el.w + (unsigned)q.ox * (unsigned)(2 * el.x + q.ox));
            const bool a = upd && n.l > la;
            n.x = a ? ea.x : n.x;
            n.y = a ? ea.y + q.oy : n.y;
            n.z = a ? ea.z : n.z;
            n.l = a ? la : n.l;
            const bool l = upd && q.has_left && n.l > ll;
            n.x = l ? el.x + q.ox : n.x;
            n.y = l ? el.y : n.y;
            n.z = l ? el.z : n.z;
            n.l = l ? ll : n.l;
        } else {
            n = fs3_wrapping(n, v, Fs3Cell{ea.x, ea.y, ea.z, ea.w}, Fs3Cell{el.x, el.y, el.z, el.w}, q.ox, q.oy, q.oz,
                             upd, q.has_left);
        }
        v = n;
        const unsigned on = (unsigned)k < (unsigned)q.nk;
        xy = (uint32_t)n.y << 16 | (uint32_t)(uint16_t)n.x;
        const unsigned long long word = q.tag | (unsigned long long)(uint16_t)n.z << 32 | xy;
        asm volatile(
            "{ .reg .pred p, px, py; .reg .s16 h;\n"
            "setp.ne.u32 p, %0, 0; setp.ne.and.u32 px, %1, 0, p; setp.ne.and.u32 py, %2, 0, p;\n"
            "@p st.shared.v4.s32 [%3], {%6, %7, %8, %9};\n"
            "@p st.shared.u32 [%4], %12;\n"
            "cvt.s16.s32 h, %8; @p st.shared.s16 [%5], h;\n"
            "@px st.relaxed.gpu.global.u64 [%10], %13;\n"
            "@py st.relaxed.gpu.global.u64 [%11], %13; }" ::"r"(on),
            "r"(q.out_x), "r"(q.out_y), "r"(q.edge + (((unsigned)s & 1) ^ 1) * kEdgeBytes), "r"(q.cell + slice),
            "r"(q.cell_z + slice), "r"(n.x), "r"(n.y), "r"(n.z), "r"(n.l), "l"(q.fx + s * kTY), "l"(q.fy + s * kTX),
            "r"(xy), "l"(word)
            : "memory");
        slice += q.slice_step;
        if (slice >= kRing * kSliceBytes) slice = q.slice_wrap;
        if (++s == e) break;
        fs3_own(q, slice, xy, n.z);
        above = q.above + ((unsigned)s & q.above_mask) * q.above_pitch;
        left = q.left + ((unsigned)s & q.left_mask) * q.left_pitch;
        asm volatile("bar.sync 1, %0;" ::"n"(kCompute) : "memory");
    }
    asm volatile("bar.sync 1, %0;" ::"n"(kCompute) : "memory");
}

static __device__ void fs3_compute(const Fs3& p, const Fs3Column& c, Fs3Smem& sm)
{
    const int t = threadIdx.x, i = t & (kTX - 1), j = t / kTX;
    const int steps = p.d + c.ni - 1 + c.nj - 1;
    const bool live = i < c.ni && j < c.nj;
    auto shared = [](const void* a) { return (uint32_t)__cvta_generic_to_shared(a); };
    Fs3Lane q;
    q.ij = i + j;
    q.nk = live ? p.d : 0;
    q.has_left = c.bx > 0 || i > 0;
    q.row_upd = c.by > 0 || j > 0;
    q.ox = c.sx ? p.cw : -p.cw;
    q.oy = c.sy ? p.cw : -p.cw;
    q.oz = c.sz ? p.cw : -p.cw;
    // place in the ring: memory order
    const int im = c.sx ? c.ni - 1 - i : i, jm = c.sy ? c.nj - 1 - j : j, place = live ? jm * kTX + im : 0;
    q.cell = shared(sm.ring) + 4 * place;
    q.cell_z = shared(sm.ring) + kSliceZ + 2 * place;
    q.slice_step = c.sz ? -(uint32_t)kSliceBytes : kSliceBytes;
    q.slice_wrap = c.sz ? (kRing - 1) * kSliceBytes : 0;
    // step 0 is slice -(i + j) of the sweep
    uint32_t slice = (uint32_t)((c.sz ? p.d - 1 + q.ij : kRing - q.ij) % kRing) * kSliceBytes;
    q.above = j ? shared(&sm.edge[0][j - 1][i]) : shared(&sm.face[0][i]);
    q.above_mask = j ? 1u : kFaceRing - 1;
    q.above_pitch = j ? kEdgeBytes : kFaceLanes * 16;
    q.left = i ? shared(&sm.edge[0][j][i - 1]) : shared(&sm.face[0][kTX + j]);
    q.left_mask = i ? 1u : kFaceRing - 1;
    q.left_pitch = i ? kEdgeBytes : kFaceLanes * 16;
    q.edge = shared(&sm.edge[0][j][i]);
    q.tag = (unsigned long long)(unsigned)(c.sweep + 1) << 48;
    // face words by step of the reader: row j's slice k at k + j = s - i, column i's at k + i = s - j
    const bool out_x = live && i == c.ni - 1 && c.bx + 1 < p.nbx, out_y = live && j == c.nj - 1 && c.by + 1 < p.nby;
    q.fx = p.xface + (long long)c.col * (p.d + kTY) * kTY + j - i * kTY;
    q.fy = p.yface + (long long)c.col * (p.d + kTX) * kTX + i - j * kTX;
    q.out_x = out_x;
    q.out_y = out_y;
    Fs3Cell v{0, 0, 0, 0};
    const bool wraps = *p.wraps != 0;
    int s = 0, next = 0, end = 0;   // chunk `next` starts at slice `end`
    while (s < steps) {
        if (s == end && next < p.nch) {
            smem_wait<20>(&sm.staged[next % kLoaders], next + 1, sm, p.err);
            end = c.chunk_end(p, next++);
        }
        int e = min(steps, smem_wait<20>(&sm.faces, s + 1, sm, p.err));
        e = max(s + 1, min(e, s < p.d ? end : s + kChunk));   // (max: a wait gave up)
        if (!wraps)
            fs3_steps<false>(q, v, slice, s, e);
        else
            fs3_steps<true>(q, v, slice, s, e);
        s = e;
        if (t == 0) smem_post(&sm.step, s);
    }
}

// the field into tiles (kIn) or back; a CTA takes a column's chunk
template <bool kIn>
__global__ void __launch_bounds__(kCompute) k_fastsweep3_tiles(Fs3 p)
{
    const int i = threadIdx.x & (kTX - 1), j = threadIdx.x / kTX;
    const int col = blockIdx.x, z0 = blockIdx.y * kChunk, nk = min(kChunk, p.d - z0);
    const int x = (col % p.nbx) * kTX + i, y = (col / p.nbx) * kTY + j;
    const bool live = x < p.w && y < p.h;
    unsigned char* tile = p.tiles + ((long long)col * p.nch * kChunk + z0) * kSliceBytes;
    short* cell = reinterpret_cast<short*>(p.cells) + (((long long)z0 * p.h + y) * p.w + x) * 3;
    const long long plane = 3LL * p.w * p.h;
    if (kIn) {
        short v[kChunk][3];
#pragma unroll
        for (int k = 0; k < kChunk; k++)
#pragma unroll
            for (int a = 0; a < 3; a++) v[k][a] = live && k < nk ? __ldcs(cell + k * plane + a) : (short)0;
        bool far = false;
#pragma unroll
        for (int k = 0; k < kChunk; k++) {
            reinterpret_cast<uint32_t*>(tile + k * kSliceBytes)[threadIdx.x] =
                (uint32_t)(uint16_t)v[k][1] << 16 | (uint32_t)(uint16_t)v[k][0];
            reinterpret_cast<short*>(tile + k * kSliceBytes + kSliceZ)[threadIdx.x] = v[k][2];
            far |= max(max(abs((int)v[k][0]), abs((int)v[k][1])), abs((int)v[k][2])) > p.safe;
        }
        if (far) *p.wraps = 1;
    } else if (live) {
        uint32_t xy[kChunk];
        short z[kChunk];
#pragma unroll
        for (int k = 0; k < kChunk; k++) {
            xy[k] = __ldcs(reinterpret_cast<const uint32_t*>(tile + k * kSliceBytes) + threadIdx.x);
            z[k] = __ldcs(reinterpret_cast<const short*>(tile + k * kSliceBytes + kSliceZ) + threadIdx.x);
        }
#pragma unroll
        for (int k = 0; k < kChunk; k++)
            if (k < nk) {
                cell[k * plane] = (short)(xy[k] & 0xFFFFu);
                cell[k * plane + 1] = (short)(xy[k] >> 16);
                cell[k * plane + 2] = z[k];
            }
    }
}

__global__ void __launch_bounds__(kFs3Threads, 2) k_fastsweep3_columns(Fs3 p)
{
    extern __shared__ __align__(16) unsigned char smem[];
    Fs3Smem& sm = *reinterpret_cast<Fs3Smem*>(smem);
    const int t = threadIdx.x, wi = t >> 5;
    if (t == 0) sm.broken = 0;
    const int items = 8 * p.nbx * p.nby;
    bool up = true;   // no wait of this warp has given up
    for (;;) {
        __syncthreads();   // the column before is stored
        if (t == 0) {
            sm.item = (int)atomicAdd(p.counter, 1u);
            sm.step = 0;
            for (int l = 0; l < kLoaders; l++) sm.staged[l] = 0;
            for (int l = 0; l < kStorers; l++) sm.stored[l] = 0;
            sm.faces = 0;
        }
        __syncthreads();
        const int item = sm.item;
        if (item >= items) return;
        const Fs3Column c(p, item);
        if (wi < kCompute / 32) fs3_compute(p, c, sm);
        else if (wi == kCompute / 32) fs3_faces(p, c, sm, up);
        else if (wi < kCompute / 32 + 1 + kLoaders) fs3_load(p, c, sm, wi - kCompute / 32 - 1, up);
        else fs3_store(p, c, sm, wi - kCompute / 32 - 1 - kLoaders);
    }
}

// workspace: counter, flag, progress, face words, tiles
struct Fs3Layout {
    long long cols;
    int nch;
    size_t progress, xface, yface, tiles, bytes;
};

static Fs3Layout fs3_layout(int w, int h, int d)
{
    Fs3Layout l;
    l.cols = (long long)((w + kTX - 1) / kTX) * ((h + kTY - 1) / kTY);
    l.nch = (d + kChunk - 1) / kChunk;
    l.progress = 256;
    l.xface = l.progress + ((size_t)l.cols * 8 * kStorers * sizeof(int) + 255) / 256 * 256;
    l.yface = l.xface + (size_t)l.cols * (d + kTY) * kTY * 8;
    l.tiles = (l.yface + (size_t)l.cols * (d + kTX) * kTX * 8 + 255) / 256 * 256;
    l.bytes = l.tiles + (size_t)l.cols * l.nch * kChunk * kSliceBytes;
    return l;
}

// Volumes of few rows and slices go to the slices (k_sweep.cu, a CTA per slice that
// walks its rows): those take a row's time for each row and slice of each sweep,
// some 1.3 us and 4.5 ns a cell, whatever the width, while x turns round with
// every sweep, so that the eight sweeps cross the columns of a row one after
// another, some 6 us each.  Columns against slices, us: 256 x 4 x 4 749, 142; 256 x 8 x
// 32 812, 707; 256 x 32 x 32 846, 1148; 2000 x 2 x 2 5709, 133; 2000 x 32 x 32 5995, 4816;
// 2000 x 128 x 8 5839, 10462; 64 x 8 x 8 216, 194; 64 x 8 x 32 251, 561.
bool fastsweep3_by_slices(int w, int h, int d)
{
    return (h + d - 2.0) * (10.4 + 0.036 * w) < 50.0 * ((w + kTX - 1) / kTX);
}

// what the columns need, whether or not they are to run
size_t fastsweep3_columns_most(int w, int h, int d)
{
    if (h < 2 || d < 2) return 0;
    const Fs3Layout l = fs3_layout(w, h, d);
    return 8 * l.cols > (1 << 28) || l.nch > 65535 ? 0 : l.bytes;
}

size_t fastsweep3_columns_bytes(int w, int h, int d)
{
    const int tuned = tune_get(kTuneFs3, w);   // positive: columns, negative: the anti-diagonal wavefront
    return tuned < 0 || (tuned == 0 && fastsweep3_by_slices(w, h, d)) ? 0 : fastsweep3_columns_most(w, h, d);
}

// false: the workspace is too small; nothing has been queued then
bool launch_fastsweep_3d_columns(void* deltas, int w, int h, int d, int cw, void* ws, size_t ws_bytes, int* err,
                                 cudaStream_t st)
{
    const size_t bytes = fastsweep3_columns_bytes(w, h, d);
    if (!bytes || ws_bytes < bytes || ((uintptr_t)ws & 15) != 0) return false;
    const Fs3Layout l = fs3_layout(w, h, d);
    const size_t smem = sizeof(Fs3Smem);
    cudaFuncSetAttribute(k_fastsweep3_columns, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaFuncSetAttribute(k_fastsweep3_columns, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_fastsweep3_columns, kFs3Threads, smem) != cudaSuccess ||
        per_sm < 1)
        return false;
    unsigned char* b = static_cast<unsigned char*>(ws);
    const WaitHooks hooks = wait_hooks();
    Fs3 p{};
    p.cells = static_cast<unsigned char*>(deltas);
    p.counter = reinterpret_cast<unsigned*>(b);
    p.wraps = reinterpret_cast<int*>(b + 128);
    p.progress = reinterpret_cast<int*>(b + l.progress);
    p.xface = reinterpret_cast<unsigned long long*>(b + l.xface);
    p.yface = reinterpret_cast<unsigned long long*>(b + l.yface);
    p.tiles = b + l.tiles;
    p.err = err;
    p.w = w;
    p.h = h;
    p.d = d;
    p.cw = cw;
    p.nbx = (w + kTX - 1) / kTX;
    p.nby = (h + kTY - 1) / kTY;
    p.nch = l.nch;
    // (one step more than the extent: candidates that are not taken)
    const long long reach = (long long)(cw < 0 ? -(long long)cw : cw) * (max(w, max(h, d)) + 1);
    p.safe = reach < 32767 ? (int)(32767 - reach) : -1;
    p.stall = hooks.stall_sweep;
    p.limit = hooks.limit;
    ProfScope ps("fastsweep_3d", st);
    cudaMemsetAsync(ws, 0, l.tiles, st);   // no tag is 0; the counts start at 0
    k_fastsweep3_tiles<true><<<dim3((unsigned)l.cols, l.nch), kCompute, 0, st>>>(p);
    const long long grid = min((long long)per_sm * g_num_sms, 8 * l.cols);
    k_fastsweep3_columns<<<(int)grid, kFs3Threads, smem, st>>>(p);
    k_fastsweep3_tiles<false><<<dim3((unsigned)l.cols, l.nch), kCompute, 0, st>>>(p);
    return true;
}

}  // namespace dolk
