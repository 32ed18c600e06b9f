// k_fastsweep3.cu -- FastSweep 3D (DistanceOcclusionLib.cpp:2186-2260) as a
// pipeline of single-warp slices, two octant sweeps per row step and four per
// launch.
//
// An octant sweep updates row (y, z) from row (y, z - dz) and row (y - dy, z) of
// the same sweep, then along x.  The order of the eight sweeps (dx innermost,
// dz outermost) allows more overlap than one sweep after the other:
//   * sweeps 2p and 2p + 1 differ in dx only and visit rows in the same order.
//     Row (y, z) of sweep 2p + 1 needs itself after sweep 2p and its neighbours
//     after sweep 2p + 1, so both passes run back to back on a row, with two
//     sets of neighbour rows;
//   * sweeps 2, 3 (6, 7) walk the same slices in the same order with y turned
//     round.  A slice may start them when its own rows are through sweeps 0, 1
//     and the slice before is ahead in sweeps 2, 3: both hold when the same
//     warp goes on to them, since the slice after takes what it needs of the
//     earlier rows as they are made, not from the field.
// So a launch runs dz = +1 (then one dz = -1): warp k owns slice k and walks its
// rows twice, one row step behind warp k - 1.
//
// A row keeps its y neighbours in registers (the warp's own last results).  The
// z neighbours come from the warp before through a ring of row slots, in shared
// memory inside a CTA of kG warps, in global memory (L2) from the CTA before.
// Every 8-byte word of a slot carries its cell and the row step's tag, so the
// reader polls the data itself: no flag, no fence, one trip.  A writer reuses a
// slot when the reader's progress count has passed it.  All CTAs are resident
// (cooperative launch) and every wait is bounded.
//
// What bounds it: the chain of 2 (h - 1) + d - 1 row steps per launch, two x
// passes each. 
// 256^3 boxes and spheres, eight sweeps: 3.3 ms; 11.2 ms with a CTA per slice,
// one sweep per launch and a flag per row between CTAs.
#include "dan_serial.cuh"
#include "kernels.h"

namespace dolk {

constexpr int kG = 4;            // slices (warps) per CTA
constexpr int kSmemSlots = 4;    // rows in a ring inside the CTA
constexpr int kGlobSlots = 16;   // rows in a ring between CTAs
constexpr int kFs3MaxRows = 8192;   // row steps of the eight sweeps stay below the 16-bit tags

struct Fs3 {
    void* cells;
    unsigned long long* rings;   // per CTA: [kGlobSlots][2][S][32] words
    int* taken;                  // per CTA: row steps its first warp has taken (32 ints apart)
    int* err;
    int w, h, d, cw;
    int dz;
    unsigned tag0;               // row steps of the launches before
    int stall;                   // sweep pair of this launch whose waits are made to run out, or -1
    unsigned limit;              // polls of a wait
};

template <bool kShared>
DOL_DI unsigned long long ring_load(const unsigned long long* p)
{
    unsigned long long v;
    if (kShared)
        asm volatile("ld.volatile.shared.u64 %0, [%1];" : "=l"(v) : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
    else
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
template <bool kShared>
DOL_DI void ring_store(unsigned long long* p, unsigned long long v)
{
    if (kShared)
        asm volatile("st.volatile.shared.u64 [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(p)), "l"(v) : "memory");
    else
        asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// The two rows of a slot, when all their words carry `tag`; false: gave up
template <int S, bool kShared>
DOL_DI bool ring_take(const unsigned long long* slot, unsigned tag, unsigned limit, uint32_t (&xy0)[S], int (&z0)[S],
                      uint32_t (&xy1)[S], int (&z1)[S])
{
    const int lane = threadIdx.x & 31;
    for (unsigned polls = 0;; polls++) {
        bool ok = true;
#pragma unroll
        for (int s = 0; s < S; s++) {
            const unsigned long long a = ring_load<kShared>(slot + s * 32 + lane);
            const unsigned long long b = ring_load<kShared>(slot + (S + s) * 32 + lane);
            xy0[s] = (uint32_t)a;
            xy1[s] = (uint32_t)b;
            z0[s] = (int)(int16_t)(a >> 32);
            z1[s] = (int)(int16_t)(b >> 32);
            ok &= (unsigned)(a >> 48) == tag && (unsigned)(b >> 48) == tag;
        }
        if (__all_sync(0xFFFFFFFFu, ok)) return true;
        if (polls >= limit) return false;
        if (!kShared) __nanosleep(32);
    }
}

template <int S, bool kShared>
DOL_DI void ring_put(unsigned long long* slot, unsigned tag, int row, const Cells<3, S>& c)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int s = 0; s < S; s++)
        ring_store<kShared>(slot + (row * S + s) * 32 + lane,
                            ((unsigned long long)((tag << 16) | (uint32_t)(uint16_t)c.z[s]) << 32) | c.xy[s]);
}

// Until *count reaches need; `seen`: its last known value.  false: gave up
DOL_DI bool wait_taken(const int* count, int need, unsigned limit, int& seen, bool shared)
{
    for (unsigned polls = 0; seen < need; polls++) {
        if (shared)
            asm volatile("ld.volatile.shared.s32 %0, [%1];"
                         : "=r"(seen)
                         : "r"((uint32_t)__cvta_generic_to_shared(count))
                         : "memory");
        else
            asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(seen) : "l"(count) : "memory");
        if (seen >= need) break;
        if (polls >= limit) return false;
        if (!shared) __nanosleep(32);
    }
    return true;
}

template <int S>
__global__ void __launch_bounds__(32 * kG) k_fastsweep3_pipe(Fs3 p)
{
    using IO = SerialIO<3, S>;
    using Row = Cells<3, S>;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_taken[kG];   // row steps that warp g has taken from its ring
    const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
    constexpr int kSlot = 2 * S * 32;   // words
    // ring g (shared): from warp g to warp g + 1
    unsigned long long* ring_sh = reinterpret_cast<unsigned long long*>(smem + kG * IO::kBytes);
    for (int i = threadIdx.x; i < (kG - 1) * kSmemSlots * kSlot; i += blockDim.x) ring_sh[i] = 0;   // no tag is 0
    if (threadIdx.x < kG) s_taken[threadIdx.x] = 0;
    __syncthreads();
    const int H = p.h - 1, Dd = p.d - 1;
    const int kk = blockIdx.x * kG + g + 1;   // this warp's slice, in sweep order
    if (kk > Dd) return;
    const bool has_next = kk < Dd;
    Field<3, S> f;
    f.lo = static_cast<unsigned char*>(p.cells);
    f.hi = f.lo + (long long)p.w * p.h * p.d * IO::kCell;
    f.w = p.w;
    f.h = p.h;
    f.xw = 0;
    const IO io{smem + g * IO::kBytes, p.w};
    constexpr int rc = 0, rz = 1;   // strips: the next row, the first slice's row
    const int cw = p.cw, oz = -cw * p.dz;
    const int z = p.dz > 0 ? kk : p.d - 1 - kk, zprev = z - p.dz;
    const bool from_field = kk == 1;   // the slice before is not updated by these sweeps
    const bool in_shared = g > 0, out_shared = g < kG - 1;
    const unsigned long long* in_ring = in_shared ? ring_sh + (g - 1) * kSmemSlots * kSlot
                                                  : p.rings + (long long)(blockIdx.x - 1) * kGlobSlots * kSlot;
    unsigned long long* out_ring =
        out_shared ? ring_sh + g * kSmemSlots * kSlot : p.rings + (long long)blockIdx.x * kGlobSlots * kSlot;
    int* my_taken = in_shared ? &s_taken[g] : p.taken + (long long)blockIdx.x * 32;
    const int* next_taken = out_shared ? &s_taken[g + 1 < kG ? g + 1 : 0] : p.taken + (long long)(blockIdx.x + 1) * 32;
    const int out_slots = out_shared ? kSmemSlots : kGlobSlots;
    int seen = 0;        // the reader's progress, as last seen
    bool up = true;      // no wait has given up
    RowShared<1> none;
    int par = 0;

    Row P0, P1, C;   // the row before after the first and the second sweep of the pair; the row
    int step = 0;
    for (int pair = 0; pair < 2; pair++) {
        const int dy = pair == 0 ? 1 : -1, oy = -cw * dy;
        const int yb = dy > 0 ? 0 : H;
        if (pair == 0) {   // the first row is not updated (:2208, :2214 start at 1)
            io.fetch(rc, f.row(z, yb), f.lo, f.hi);
            io.cells_of(P0, rc, f.row(z, yb), cw);
            P1 = P0;
        } else {
            P0 = P1;       // the last row of the pair before is the first of this one
        }
        __syncwarp();
        io.fetch(rc, f.row(z, yb + dy), f.lo, f.hi);
        if (from_field) io.fetch(rz, f.row(zprev, yb + dy), f.lo, f.hi);
#pragma unroll 1
        for (int jj = 1; jj <= H; jj++) {
            const int y = yb + jj * dy;
            step++;
            const unsigned tag = (p.tag0 + (unsigned)step) & 0xFFFFu;
            io.cells_of(C, rc, f.row(z, y), cw);
            uint32_t zx0[S], zx1[S];
            int zz0[S], zz1[S];
            if (from_field) {
                uint32_t wd[IO::kWords];
                io.words(wd, rz, f.row(zprev, y));
                IO::split(wd, zx0, zz0);
#pragma unroll
                for (int s = 0; s < S; s++) {
                    zx1[s] = zx0[s];
                    zz1[s] = zz0[s];
                }
            }
            if (jj < H) {   // the next rows, behind this one's passes
                io.fetch(rc, f.row(z, y + dy), f.lo, f.hi);
                if (from_field) io.fetch(rz, f.row(zprev, y + dy), f.lo, f.hi);
            }
            if (!from_field) {
                const unsigned want = pair == p.stall ? 0x10000u : tag;   // (a tag no word can carry)
                const unsigned limit = up ? p.limit : 0;
                bool ok;
                if (in_shared)
                    ok = ring_take<S, true>(in_ring + (step % kSmemSlots) * kSlot, want, limit, zx0, zz0, zx1, zz1);
                else
                    ok = ring_take<S, false>(in_ring + (step % kGlobSlots) * kSlot, want, limit, zx0, zz0, zx1, zz1);
                if (!ok && up) {
                    up = false;
                    if (lane == 0) atomicExch(p.err, 1);
                }
                if (lane == 0) {
                    if (in_shared)
                        asm volatile("st.volatile.shared.s32 [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(my_taken)),
                                     "r"(step)
                                     : "memory");
                    else
                        asm volatile("st.relaxed.gpu.global.s32 [%0], %1;" ::"l"(my_taken), "r"((int)p.tag0 + step)
                                     : "memory");
                }
            }
            unsigned long long* slot = out_ring + (step % out_slots) * kSlot;
            if (has_next && step > out_slots) {   // the slot is free when the row step before in it was taken
                const int base = out_shared ? 0 : (int)p.tag0;
                if (!wait_taken(next_taken, base + step - out_slots, up ? p.limit : 0, seen, out_shared) && up) {
                    up = false;
                    if (lane == 0) atomicExch(p.err, 1);
                }
            }
            // first sweep of the pair: to the right
            pull_z<S>(C, zx0, zz0, oz);
            merge_y<3, S>(P0, C, oy);
            row_pass_w<3, S, 1, +1, NoDiag>(P0, NoDiag{}, cw, none, par, chain_none(cw));
            if (has_next) {
                if (out_shared) ring_put<S, true>(slot, tag, 0, P0);
                else ring_put<S, false>(slot, tag, 0, P0);
            }
            // second: to the left
            C = P0;
            pull_z<S>(C, zx1, zz1, oz);
            merge_y<3, S>(P1, C, oy);
            row_pass_w<3, S, 1, -1, NoDiag>(P1, NoDiag{}, cw, none, par, chain_none(cw));
            if (has_next) {
                if (out_shared) ring_put<S, true>(slot, tag, 1, P1);
                else ring_put<S, false>(slot, tag, 1, P1);
            }
            io.put_cells(f.row(z, y), P1);
        }
    }
}

// cells per lane, 0: rows too wide for a warp
static int pipe_s(int w)
{
    const int tv = tune_get(kTuneFs3, w);
    if ((tv == 2 || tv == 4 || tv == 8) && 32 * tv >= w) return tv;
    return w <= 64 ? 2 : (w <= 128 ? 4 : (w <= 256 ? 8 : 0));
}

static size_t pipe_bytes(int w, int d, int s)
{
    const size_t ctas = (size_t)(d - 1 + kG - 1) / kG;
    const size_t rings = ctas * kGlobSlots * 2 * s * 32 * sizeof(unsigned long long);
    (void)w;
    return rings + (ctas + 1) * 32 * sizeof(int) + 256;
}

size_t fastsweep3_pipe_bytes(int w, int h, int d)
{
    const int s = pipe_s(w);
    if (!s || h < 2 || d < 2 || h > kFs3MaxRows || tune_get(kTuneFs3, w) < 0) return 0;
    return pipe_bytes(w, d, s);
}

template <int S>
static bool run_pipe(Fs3 p, size_t bytes, cudaStream_t st)
{
    auto kern = k_fastsweep3_pipe<S>;
    const size_t smem = kG * SerialIO<3, S>::kBytes + (size_t)(kG - 1) * kSmemSlots * 2 * S * 32 * 8;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * kG, smem) != cudaSuccess) return false;
    const int ctas = (p.d - 1 + kG - 1) / kG;
    if ((long long)per_sm * g_num_sms < ctas) return false;   // every slice needs its warp resident
    cudaMemsetAsync(p.rings, 0, bytes, st);   // no tag is 0; the counts start at 0
    const WaitHooks hooks = wait_hooks();
    p.limit = hooks.limit;
    for (int dir = 0; dir < 2; dir++) {
        p.dz = dir == 0 ? 1 : -1;
        p.tag0 = (unsigned)(2 * (p.h - 1) * dir);
        p.stall = hooks.stall_sweep >= 4 * dir && hooks.stall_sweep < 4 * dir + 4 ? (hooks.stall_sweep - 4 * dir) / 2 : -1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(ctas);
        cfg.blockDim = dim3(32 * kG);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (cudaLaunchKernelEx(&cfg, kern, p) != cudaSuccess) {
            if (dir == 0) return false;   // nothing has run
            break;                        // half the sweeps have: the caller reports the launch error
        }
    }
    return true;
}

// false: not for this field (rows too wide, more slices than resident warps) or
// the workspace is too small; nothing has been queued then
bool launch_fastsweep_3d_pipe(void* deltas, int w, int h, int d, int cw, void* ws, size_t ws_bytes, int* err,
                              cudaStream_t st)
{
    const size_t bytes = fastsweep3_pipe_bytes(w, h, d);
    if (!bytes || ws_bytes < bytes || ((uintptr_t)ws & 7) != 0) return false;
    const int s = pipe_s(w);
    const size_t ctas = (size_t)(d - 1 + kG - 1) / kG;
    Fs3 p{};
    p.cells = deltas;
    p.rings = static_cast<unsigned long long*>(ws);
    p.taken = reinterpret_cast<int*>(p.rings + ctas * kGlobSlots * 2 * s * 32);
    p.err = err;
    p.w = w;
    p.h = h;
    p.d = d;
    p.cw = cw;
    ProfScope ps("fastsweep_3d", st);
    return s == 2 ? run_pipe<2>(p, bytes, st) : (s == 4 ? run_pipe<4>(p, bytes, st) : run_pipe<8>(p, bytes, st));
}

}  // namespace dolk
