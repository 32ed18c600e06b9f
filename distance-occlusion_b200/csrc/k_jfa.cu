// k_jfa.cu -- JumpFlood passes and deltas -> distances.
//
// JumpFlood (DistanceOcclusionLib.cpp:782-908 for 2D, :2398-2472 for 3D) is a
// ping-pong stencil: every cell of a pass reads only the previous pass, so one
// thread per cell with the reference's fixed candidate order reproduces it
// exactly.  The driver keeps the reference's pass schedule: steps from
// FloorPow2(max dim - 1) halving to 1, plus one extra step-1 pass back into the
// caller's buffer when the last result sits in the ping-pong buffer.
#include <limits.h>

#include "common.cuh"
#include "grid_barrier.cuh"
#include "kernels.h"

namespace dolk {

// One cell of a 2D pass.  kCoherent: the pass before ran in the same launch.
template <bool kCoherent>
__device__ __forceinline__ uint32_t jfa2_cell(const uint32_t* in, int w, int h, int s, int cw, int x, int y)
{
    const int o = cw * s;
    auto at = [&](int xx, int yy) {
        const uint32_t* p = in + (long long)yy * w + xx;
        return unpack2(kCoherent ? __ldcg(p) : __ldg(p));
    };
    C2 best = at(x, y);
    int32_t bl = len(best);   // the incumbent's squared length, kept between candidates
    // closer(): a candidate wins only when strictly shorter
    auto consider = [&](C2 cand) {
        const int32_t cl = len(cand);
        if (bl > cl) {
            best = cand;
            bl = cl;
        }
    };
    // candidate order of :794-868
    if (x - s >= 0) {
        consider(add(at(x - s, y), -o, 0));
        if (y - s >= 0) consider(add(at(x - s, y - s), -o, -o));
        if (y + s < h) consider(add(at(x - s, y + s), -o, +o));
    }
    if (x + s < w) {
        consider(add(at(x + s, y), +o, 0));
        if (y - s >= 0) consider(add(at(x + s, y - s), +o, -o));
        if (y + s < h) consider(add(at(x + s, y + s), +o, +o));
    }
    if (y - s >= 0) consider(add(at(x, y - s), 0, -o));
    if (y + s < h) consider(add(at(x, y + s), 0, +o));
    return pack2(best);
}

__global__ void __launch_bounds__(512) k_jfa2(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, int w,
                                              int h, int s, int cw)
{
    const int x = blockIdx.x * 32 + (threadIdx.x & 31);
    const int y = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (x >= w || y >= h) return;
    out[(long long)y * w + x] = jfa2_cell<false>(in, w, h, s, cw, x, y);
}

struct JfaSteps {
    int n, s[40];
};

// All passes of an image in one cooperative launch, a grid barrier between them:
// a pass over few cells takes less than its launch (512 x 512, 10 passes: 60 us
// as launches, 46 us).
__global__ void __launch_bounds__(1024) k_jfa2_all(uint32_t* a, uint32_t* b, int w, int h, int cw, JfaSteps st,
                                                  unsigned* count, int* err)
{
    const int tx = (w + 31) / 32, ty = (h + 31) / 32;
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    unsigned passed = 0;
    for (int pass = 0; pass < st.n; pass++) {
        for (int t = blockIdx.x; t < tx * ty; t += gridDim.x) {
            const int by = t / tx, x = (t - by * tx) * 32 + lane, y = by * 32 + wi;
            if (x < w && y < h) b[(long long)y * w + x] = jfa2_cell<true>(a, w, h, st.s[pass], cw, x, y);
        }
        if (pass + 1 < st.n && !grid_barrier(count, passed, err)) return;
        uint32_t* c = a;
        a = b;
        b = c;
    }
}

__device__ __forceinline__ C3 load3(const int16_t* p, long long i)
{
    const int16_t* c = p + 3 * i;
    return C3{__ldg(c), __ldg(c + 1), __ldg(c + 2)};
}
__device__ __forceinline__ void store3(int16_t* p, long long i, C3 v)
{
    int16_t* c = p + 3 * i;
    c[0] = (int16_t)v.x;
    c[1] = (int16_t)v.y;
    c[2] = (int16_t)v.z;
}
// Between its first and last pass the 3D JumpFlood keeps cells in 8 bytes
// (x, y, z, unused): one aligned load per neighbour instead of three.
__device__ __forceinline__ C3 load3w(const uint2* p, long long i)
{
    const uint2 u = __ldg(p + i);
    return C3{(int)(int16_t)(u.x & 0xFFFFu), (int)(int16_t)(u.x >> 16), (int)(int16_t)(u.y & 0xFFFFu)};
}
__device__ __forceinline__ void store3w(uint2* p, long long i, C3 v)
{
    p[i] = make_uint2((uint32_t)(uint16_t)v.x | ((uint32_t)(uint16_t)v.y << 16), (uint32_t)(uint16_t)v.z);
}

// kWideIn / kWideOut: 8-byte cells (the ping-pong buffers) or the caller's 6-byte cells
template <bool kWideIn, bool kWideOut>
__global__ void __launch_bounds__(512) k_jfa3(const void* __restrict__ in, void* __restrict__ out, int w, int h, int d,
                                              int s, int cw)
{
    const int x = blockIdx.x * 32 + (threadIdx.x & 31);
    const int y = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int z = blockIdx.z;
    if (x >= w || y >= h) return;
    const long long plane = (long long)w * h;
    const long long idx = z * plane + (long long)y * w + x;
    auto ld = [&](long long i) -> C3 {
        return kWideIn ? load3w(static_cast<const uint2*>(in), i) : load3(static_cast<const int16_t*>(in), i);
    };
    C3 best = ld(idx);
    int32_t bl = len(best);   // the incumbent's squared length, kept between candidates
    // all offsets in {-s, 0, +s}^3 that stay inside, z outermost, x innermost,
    // skipping neighbours still at max (:2419-2438); a candidate wins only
    // when strictly shorter (closer())
    // (unrolled over the 27 offsets; an offset leaving the field is skipped)
    const bool zlo = z - s >= 0, zhi = z + s < d, ylo = y - s >= 0, yhi = y + s < h, xlo = x - s >= 0,
               xhi = x + s < w;
    const long long oz = (long long)s * plane, oy = (long long)s * w;
#pragma unroll
    for (int iz = -1; iz <= 1; iz++) {
        const bool vz = iz == 0 || (iz < 0 ? zlo : zhi);
#pragma unroll
        for (int iy = -1; iy <= 1; iy++) {
            const bool vy = iy == 0 || (iy < 0 ? ylo : yhi);
#pragma unroll
            for (int ix = -1; ix <= 1; ix++) {
                const bool vx = ix == 0 || (ix < 0 ? xlo : xhi);
                if (!(vz && vy && vx)) continue;
                const C3 c = ld(idx + iz * oz + iy * oy + ix * s);
                if (c.x == kMax3) continue;
                const C3 cand = add(c, cw * s * ix, cw * s * iy, cw * s * iz);
                const int32_t cl = len(cand);
                if (bl > cl) {
                    best = cand;
                    bl = cl;
                }
            }
        }
    }
    if (kWideOut)
        store3w(static_cast<uint2*>(out), idx, best);
    else
        store3(static_cast<int16_t*>(out), idx, best);
}

// The same pass walking z: a thread takes one column (x, y) and the cells
// z = r + i s of one residue class r (a chunk of kJfaChunk of them), and visits
// the slices r + j s in order, each slice's 9 neighbours of the column loaded
// once and applied to the three cells that read them -- as offset +s for cell
// j - 1, 0 for cell j and -s for cell j + 1.  A cell thus meets its candidates
// in the reference's order (its own value first, then the slice below, its
// own slice, the slice above, y then x within each), and the pass loads ~10
// values per cell instead of 27.
constexpr int kJfaChunk = 32;

// kSame: the pass before ran in the same launch (no read-only loads; the grid
// barrier between them orders plain ones)
template <bool kWideIn, bool kSame>
__device__ __forceinline__ C3 jfa_ld(const void* in, long long i)
{
    if (!kSame) return kWideIn ? load3w(static_cast<const uint2*>(in), i) : load3(static_cast<const int16_t*>(in), i);
    if (kWideIn) {
        const uint2 u = static_cast<const uint2*>(in)[i];
        return C3{(int)(int16_t)(u.x & 0xFFFFu), (int)(int16_t)(u.x >> 16), (int)(int16_t)(u.y & 0xFFFFu)};
    }
    const int16_t* c = static_cast<const int16_t*>(in) + 3 * i;
    return C3{c[0], c[1], c[2]};
}

template <bool kWideIn, bool kWideOut, bool kSame>
__device__ __forceinline__ void jfa3z_column(const void* in, void* out, int w, int h, int d, int s, int cw, int run,
                                             int nchunk, int x, int y, int rc)
{
    if (x >= w || y >= h) return;
    const int r = rc / nchunk, chunk = rc % nchunk;
    const int m = (d - r + s - 1) / s;   // cells r + i s < d
    const int i0 = chunk * run, i1 = min(m, i0 + run);
    if (i0 >= i1) return;
    const long long plane = (long long)w * h;
    const long long col = (long long)y * w + x;
    const bool ylo = y - s >= 0, yhi = y + s < h, xlo = x - s >= 0, xhi = x + s < w;
    const int o = cw * s;
    // the three cells a slice serves: A = j - 1 (offset +s), B = j (0), C = j + 1 (-s)
    C3 bA{0, 0, 0}, bB{0, 0, 0}, bC{0, 0, 0};
    int32_t lA = 0, lB = 0, lC = 0;
    auto consider = [](C3& best, int32_t& bl, const C3& cand) {
        const int32_t cl = len(cand);
        if (bl > cl) {   // strictly shorter (closer())
            best = cand;
            bl = cl;
        }
    };
    for (int j = i0 - 1; j <= i1; j++) {
        const bool hasA = j - 1 >= i0, hasB = j >= i0 && j < i1, hasC = j + 1 < i1;
        if (hasC) {   // cell j + 1 starts from its own value
            bC = jfa_ld<kWideIn, kSame>(in, (long long)(r + (j + 1) * s) * plane + col);
            lC = len(bC);
        }
        if (j >= 0 && j < m) {   // slice r + j s exists: its 9 neighbours of the column
            const long long base = (long long)(r + j * s) * plane + col;
#pragma unroll
            for (int iy = -1; iy <= 1; iy++) {
                const bool vy = iy == 0 || (iy < 0 ? ylo : yhi);
#pragma unroll
                for (int ix = -1; ix <= 1; ix++) {
                    const bool vx = ix == 0 || (ix < 0 ? xlo : xhi);
                    if (!(vy && vx)) continue;
                    const C3 c = jfa_ld<kWideIn, kSame>(in, base + (long long)iy * s * w + ix * s);
                    if (c.x == kMax3) continue;
                    const int cx = trunc16(c.x + o * ix), cy = trunc16(c.y + o * iy);
                    if (hasC) consider(bC, lC, C3{cx, cy, trunc16(c.z - o)});
                    if (hasB) consider(bB, lB, C3{cx, cy, c.z});
                    if (hasA) consider(bA, lA, C3{cx, cy, trunc16(c.z + o)});
                }
            }
        }
        if (hasA) {   // cell j - 1 has seen its three slices
            const long long idx = (long long)(r + (j - 1) * s) * plane + col;
            if (kWideOut)
                store3w(static_cast<uint2*>(out), idx, bA);
            else
                store3(static_cast<int16_t*>(out), idx, bA);
        }
        bA = bB;
        lA = lB;
        bB = bC;
        lB = lC;
    }
}

template <bool kWideIn, bool kWideOut>
__global__ void __launch_bounds__(512) k_jfa3z(const void* __restrict__ in, void* __restrict__ out, int w, int h, int d,
                                               int s, int cw, int nchunk)
{
    jfa3z_column<kWideIn, kWideOut, false>(in, out, w, h, d, s, cw, kJfaChunk, nchunk, blockIdx.x * 32 + (threadIdx.x & 31),
                                           blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5), blockIdx.z);
}

// ---- packed 3D passes ---------------------------------------------------------------------
//
// A neighbour's candidate is its delta plus the offset to it, that is, the
// distance from this cell to the neighbour's site; cells at max (25000) are
// skipped and so stay as they are.  So a pass can keep sites instead of deltas:
// one 32-bit word per cell, the site's position in units of the cell width
// (cw * cell + delta, plus 1: border deltas reach one unit outside), 10 + 10 + 11
// bits, or kNoSite for a cell at max.  The squared length of a candidate is then
// exact integer arithmetic on positions with no int16 in between.
//
// Fields whose sides stay within kSiteSpan units qualify; there a site is less
// than 2^21 away in square and kNoSite's position more, so a cell without a
// site loses to any real one without a test.  Initial deltas always have this
// form; the caller's own are checked by the conversion (k_jfa3_pack), and if
// one does not, the packed passes do nothing and k_jfa3_general runs the
// passes on the cells as they are.
//
// What bounds a pass: integer instructions.  Walking z (as k_jfa3z) a neighbour
// is unpacked once for the three cells that read it; each of them costs a
// multiply-add and a share of a three-way min of length * 256 + order, the order being
// the reference's (own cell first, z outermost, x innermost), so that ties fall
// as there, and the winner's word is read again at the end.  256^3, a pass:
// 0.30 ms on 8-byte deltas with a compare and five selects per candidate,
// 0.16 ms.
constexpr int kSiteSpan = 600;
constexpr uint32_t kNoSite = 0xFFFFFFFFu;   // at (1023, 1023, 2047)

__device__ __forceinline__ uint32_t pack_site(int x, int y, int z)
{
    return (uint32_t)x | ((uint32_t)y << 10) | ((uint32_t)z << 21);
}

// deltas -> sites; *odd is set when a cell has no site in range and is not at max
__global__ void __launch_bounds__(256) k_jfa3_pack(const int16_t* __restrict__ in, uint32_t* __restrict__ out, int w,
                                                   int h, int d, int cw, int* __restrict__ odd)
{
    bool bad = false;
    const int rows = h * d, lane = threadIdx.x & 31, nw = (gridDim.x * blockDim.x) >> 5;
    for (int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < rows; row += nw) {
        const int z = row / h, y = row - z * h;
        for (int x = lane; x < w; x += 32) {
            const int i = row * w + x;
            const C3 c = load3(in, i);
            const int px = c.x + cw * x + 1, py = c.y + cw * y + 1, pz = c.z + cw * z + 1;
            const bool none = c.x == kMax3 && c.y == kMax3 && c.z == kMax3;
            if (!none)
                bad |= (unsigned)px > (unsigned)(cw * (w - 1) + 2) || (unsigned)py > (unsigned)(cw * (h - 1) + 2) ||
                       (unsigned)pz > (unsigned)(cw * (d - 1) + 2);
            out[i] = none ? kNoSite : pack_site(px & 1023, py & 1023, pz & 1023);
        }
    }
    if (odd && __any_sync(0xFFFFFFFFu, bad) && lane == 0) *odd = 1;
}

template <bool kLast>
__global__ void __launch_bounds__(512) k_jfa3p(const uint32_t* __restrict__ in, void* __restrict__ out, int w, int h,
                                               int d, int s, int cw, int len, int nchunk,
                                               const int* __restrict__ odd)
{
    if (odd && *odd) return;
    const int x = blockIdx.x * 32 + (threadIdx.x & 31);
    const int y = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (x >= w || y >= h) return;
    const int r = blockIdx.z / nchunk, chunk = blockIdx.z % nchunk;
    const int m = (d - r + s - 1) / s;   // cells r + i s < d
    const int i0 = chunk * len, i1 = min(m, i0 + len);
    if (i0 >= i1) return;
    const int plane = w * h;
    const int col = y * w + x;
    const int cx = cw * x + 1, cy = cw * y + 1;
    // the slice's nine neighbours; one outside the field stands for the middle
    // one, a candidate anyway
    const int oy[3] = {y - s >= 0 ? -s * w : 0, 0, y + s < h ? s * w : 0};
    const int ox[3] = {x - s >= 0 ? -s : 0, 0, x + s < w ? s : 0};
    __shared__ int s_off[9][512];
#pragma unroll
    for (int n = 0; n < 9; n++) s_off[n][threadIdx.x] = oy[n / 3] + ox[n % 3];
    // a cell's best so far: length * 256 + order (0: its own site)
    int kA = INT_MAX, kB = INT_MAX, kC = INT_MAX;
    // the cells s slices away from this slice's: (d +- t)^2 = d^2 +- 2 t d + t^2, in units of 1/16
    const int t = 16 * cw * s, t2 = t * t;
    for (int j = i0 - 1; j <= i1; j++) {
        kC = INT_MAX;   // cell j + 1 starts here
        if (j >= 0 && j < m) {
            const uint32_t* slice = in + ((r + j * s) * plane + col);
            const int zB = 16 * (cw * (r + j * s) + 1);
            int vA[9], vB[9], vC[9];   // cells j - 1, j, j + 1 (A, C less t2)
#pragma unroll
            for (int n = 0; n < 9; n++) {
                const uint32_t p = __ldg(slice + (oy[n / 3] + ox[n % 3]));
                const int dx = (int)(p & 1023u) * 16 - 16 * cx, dy = (int)((p >> 10) & 1023u) * 16 - 16 * cy;
                const int dz = (int)(p >> 21) * 16 - zB;
                const int b = dz * dz + (dy * dy + (dx * dx + n));
                vA[n] = dz * (2 * t) + b;
                vB[n] = b;
                vC[n] = dz * (-2 * t) + b;
            }
            auto min9 = [](const int (&v)[9]) {
                return __vimin3_s32(__vimin3_s32(v[0], v[1], v[2]), __vimin3_s32(v[3], v[4], v[5]),
                                    __vimin3_s32(v[6], v[7], v[8]));
            };
            const int own = vB[4] & ~255;
            kC = min9(vC) + t2 + 1;                              // orders 1 .. 9: the slice below
            vB[4] = vB[3];
            kB = __vimin3_s32(kB, min9(vB) + 10, own);           // 10 .. 18: its own slice
            kA = min(kA, min9(vA) + t2 + 19);                    // 19 .. 27: the slice above
        }
        if (j - 1 >= i0) {   // cell j - 1 has seen its three slices
            const int z = r + (j - 1) * s, idx = z * plane + col;
            const int o = (kA & 255) - 1;    // -1: its own
            int from = idx;
            if (o >= 0) {
                const int sl = (o * 57) >> 9;      // o / 9
                from = idx + (sl - 1) * (s * plane) + s_off[o - 9 * sl][threadIdx.x];
            }
            const uint32_t p = __ldg(in + from);
            if (kLast) {
                const C3 c = p == kNoSite ? C3{kMax3, kMax3, kMax3}
                                          : C3{(int)(p & 1023u) - cx, (int)((p >> 10) & 1023u) - cy,
                                               (int)(p >> 21) - (cw * z + 1)};
                store3(static_cast<int16_t*>(out), idx, c);
            } else {
                static_cast<uint32_t*>(out)[idx] = p;
            }
        }
        kA = kB;
        kB = kC;
    }
}

// All passes on the cells as they are, in one cooperative launch, when the
// conversion found a cell that the packed passes cannot hold: the z walk, between
// the caller's array and one buffer (the schedule has an even number of passes;
// the second buffer's start holds the flag and the barrier).  256^3 with one such
// cell: 5.68 ms with a cell per thread and 27 loads, 2.97 now (2.47 as launches of
// the z walk between two buffers, which only the host could choose); 64^3 0.16 ms,
// 0.13 (0.22).
__global__ void __launch_bounds__(256) k_jfa3_general(int16_t* cells, uint2* buf, int w, int h, int d, int cw,
                                                      JfaSteps st, int len, const int* odd, unsigned* count, int* err)
{
    if (!*odd) return;
    const int tx = (w + 31) / 32, ty = (h + 7) / 8;
    unsigned passed = 0;
    for (int pass = 0; pass < st.n; pass++) {
        const int s = st.s[pass];
        const int nchunk = ((d + s - 1) / s + len - 1) / len;
        const int items = tx * ty * min(s, d) * nchunk;
        for (int t = blockIdx.x; t < items; t += gridDim.x) {
            const int rc = t / (tx * ty), tile = t - rc * (tx * ty), by = tile / tx;
            const int x = (tile - by * tx) * 32 + (threadIdx.x & 31), y = by * 8 + (threadIdx.x >> 5);
            if (pass & 1) jfa3z_column<true, false, true>(buf, cells, w, h, d, s, cw, len, nchunk, x, y, rc);
            else jfa3z_column<false, true, true>(cells, buf, w, h, d, s, cw, len, nchunk, x, y, rc);
        }
        if (pass + 1 < st.n && !grid_barrier(count, passed, err)) return;
    }
}

size_t jumpflood_workspace_bytes(int dim, int w, int h, int d)
{
    const size_t cells = (size_t)w * h * (dim == 3 ? d : 1);
    if (dim == 2) return cells * sizeof(uint32_t);
    return 2 * (((cells * sizeof(uint2)) + 255) & ~(size_t)255);
}

static int floor_pow2(int v)
{
    v |= v >> 1;
    v |= v >> 2;
    v |= v >> 4;
    v |= v >> 8;
    v |= v >> 16;
    return (v + 1) >> 1;
}

// Cells up to which a 2D field runs all its passes in one launch
constexpr long long kJfaOneLaunch = 1 << 22;

static bool jfa2_one_launch(uint32_t* deltas, uint32_t* temp, int w, int h, int cw, const int* steps, int np, int* err,
                            cudaStream_t st)
{
    static_assert(sizeof(JfaSteps) < 256, "a kernel parameter");
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_jfa2_all, 1024, 0) != cudaSuccess || per_sm < 1)
        return false;
    void* count = nullptr;
    if (cudaMallocAsync(&count, sizeof(unsigned), st) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    cudaMemsetAsync(count, 0, sizeof(unsigned), st);
    JfaSteps js;
    js.n = np;
    for (int i = 0; i < np; i++) js.s[i] = steps[i];
    const long long tiles = (long long)((w + 31) / 32) * ((h + 31) / 32);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)min((long long)per_sm * g_num_sms, tiles));
    cfg.blockDim = dim3(1024);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    ProfScope ps("jumpflood_passes", st);
    const bool ok = cudaLaunchKernelEx(&cfg, k_jfa2_all, deltas, temp, w, h, cw, js, static_cast<unsigned*>(count), err) ==
                    cudaSuccess;
    if (!ok) cudaGetLastError();
    cudaFreeAsync(count, st);
    return ok;
}

// The packed passes in the workspace of the 8-byte ones: their two buffers take
// the first half, the check's flag and the general passes' barrier the start of
// the second.
static bool run_packed(void* deltas, void* temp, size_t half, int w, int h, int d, int cw, const int* steps, int np,
                       int ry, bool checked, int* err, cudaStream_t st)
{
    const size_t cells = (size_t)w * h * d;
    uint32_t* pb[2] = {static_cast<uint32_t*>(temp), static_cast<uint32_t*>(temp) + cells};
    unsigned* words = reinterpret_cast<unsigned*>(static_cast<char*>(temp) + half);   // the second buffer's start
    int* odd = checked ? nullptr : reinterpret_cast<int*>(words);
    JfaSteps js;
    js.n = np;
    for (int i = 0; i < np; i++) js.s[i] = steps[i];
    int per_sm = 0;
    if (!checked) {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_jfa3_general, 256, 0) != cudaSuccess || per_sm < 1)
            return false;
        cudaMemsetAsync(odd, 0, 2 * sizeof(unsigned), st);
    }
    const int warps = h * d;
    k_jfa3_pack<<<min((warps + 7) / 8, g_num_sms * 16), 256, 0, st>>>(static_cast<const int16_t*>(deltas), pb[0], w, h, d,
                                                                     cw, odd);
    // cells a thread walks: a chunk of n loads n + 2 slices, but small volumes need
    // the threads (whole calls with 8 | 16 | 32 cells: 64^3 78 | 96 | 116 us, 128^3 247 |
    // 253 | 275, 400 x 300 x 100 2342 | 2309 | 2345, 256^3 1511 | 1442 | 1442)
    const int len = (long long)w * h * d <= (1 << 20) ? 8 : 16;
    for (int i = 0; i < np; i++) {
        ProfScope ps("jumpflood_pass", st);
        const int sv = steps[i], nres = sv < d ? sv : d;
        const int nchunk = ((d + sv - 1) / sv + len - 1) / len;
        const dim3 gz((w + 31) / 32, (h + ry - 1) / ry, (unsigned)(nres * nchunk));
        if (i == np - 1)
            k_jfa3p<true><<<gz, 32 * ry, 0, st>>>(pb[i & 1], deltas, w, h, d, sv, cw, len, nchunk, odd);
        else
            k_jfa3p<false><<<gz, 32 * ry, 0, st>>>(pb[i & 1], pb[(i & 1) ^ 1], w, h, d, sv, cw, len, nchunk, odd);
    }
    if (!checked) {
        // as `len` above (2 | 4 | 8 | 16 | 32 cells: 64^3 129 | 167 | 225 | 322 | 456 us,
        // 128^3 622 | 514 | 578 | 562 | 841, 256^3 4048 | 3354 | 3107 | 2974 | 2918)
        const int glen = cells <= (1 << 19) ? 2 : cells <= (1 << 21) ? 4 : 16;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)min((long long)per_sm * g_num_sms, (long long)(cells + 255) / 256));
        cfg.blockDim = dim3(256);
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        cudaLaunchKernelEx(&cfg, k_jfa3_general, static_cast<int16_t*>(deltas), static_cast<uint2*>(temp), w, h, d, cw, js,
                           glen, (const int*)odd, words + 1, err);
    }
    return true;
}

void launch_jumpflood(int dim, void* deltas, void* temp, int w, int h, int d, int cw, bool initial, int* err,
                      size_t scratch_cap, cudaStream_t st)
{
    int m = w > h ? w : h;
    if (dim == 3 && d > m) m = d;
    // rows per CTA (32 x ry threads): tuned, else 8
    int ry = tune_get(dim == 2 ? kTuneJfa2 : kTuneJfa3, w);
    const bool per_cell = dim == 3 && ry < 0;   // 3D, negative tuned values: one thread per cell (k_jfa3)
    if (per_cell) ry = -ry;
    if (ry != 2 && ry != 4 && ry != 8 && ry != 16) ry = 8;
    // the reference's schedule: steps FloorPow2(m - 1) .. 1 ping-ponging with
    // the caller's buffer, plus one step-1 pass when the result would end in temp
    int steps[40], np = 0;
    for (int s = floor_pow2(m - 1); s > 0; s /= 2) steps[np++] = s;
    if (np & 1) steps[np++] = 1;
    if (dim == 2) {
        void* a = deltas;
        void* b = temp;
        if (tune_get(kTuneJfa2, w) == 0 && (long long)w * h <= kJfaOneLaunch && np > 1 &&
            (!scratch_cap || scratch_cap >= sizeof(unsigned)) &&
            jfa2_one_launch(static_cast<uint32_t*>(deltas), static_cast<uint32_t*>(temp), w, h, cw, steps, np, err, st))
            return;
        const dim3 grid((w + 31) / 32, (h + ry - 1) / ry);
        for (int i = 0; i < np; i++) {
            ProfScope ps("jumpflood_pass", st);
            k_jfa2<<<grid, 32 * ry, 0, st>>>(static_cast<const uint32_t*>(a), static_cast<uint32_t*>(b), w, h, steps[i],
                                             cw);
            void* t = a;
            a = b;
            b = t;
        }
        return;
    }
    const size_t cells = (size_t)w * h * d;
    const size_t half = ((cells * sizeof(uint2)) + 255) & ~(size_t)255;
    // sites in 32 bits: sides within the packed positions' range
    if (!per_cell && np > 0 && (long long)cw * (m - 1) + 2 <= kSiteSpan && ((uintptr_t)temp & 7) == 0 &&
        run_packed(deltas, temp, half, w, h, d, cw, steps, np, ry, initial, err, st))
        return;
    // 3D: the caller's 6-byte cells -> 8-byte ping-pong buffers -> the caller's cells
    uint2* wb[2] = {static_cast<uint2*>(temp),
                    reinterpret_cast<uint2*>(static_cast<char*>(temp) + (((cells * sizeof(uint2)) + 255) & ~(size_t)255))};
    const dim3 grid((w + 31) / 32, (h + ry - 1) / ry, d);
    for (int i = 0; i < np; i++) {
        ProfScope ps("jumpflood_pass", st);
        const bool first = i == 0, last = i == np - 1;
        const void* src = first ? deltas : wb[(i - 1) & 1];
        void* dst = last ? deltas : wb[i & 1];
        const int sv = steps[i];
        if (per_cell) {
            if (first)
                k_jfa3<false, true><<<grid, 32 * ry, 0, st>>>(src, dst, w, h, d, sv, cw);
            else if (last)
                k_jfa3<true, false><<<grid, 32 * ry, 0, st>>>(src, dst, w, h, d, sv, cw);
            else
                k_jfa3<true, true><<<grid, 32 * ry, 0, st>>>(src, dst, w, h, d, sv, cw);
            continue;
        }
        // z walk: residue classes of z mod s, chunks of kJfaChunk cells along each
        const int nres = sv < d ? sv : d;
        const int nchunk = ((d + sv - 1) / sv + kJfaChunk - 1) / kJfaChunk;
        const dim3 gz((w + 31) / 32, (h + ry - 1) / ry, (unsigned)(nres * nchunk));
        if (first)
            k_jfa3z<false, true><<<gz, 32 * ry, 0, st>>>(src, dst, w, h, d, sv, cw, nchunk);
        else if (last)
            k_jfa3z<true, false><<<gz, 32 * ry, 0, st>>>(src, dst, w, h, d, sv, cw, nchunk);
        else
            k_jfa3z<true, true><<<gz, 32 * ry, 0, st>>>(src, dst, w, h, d, sv, cw, nchunk);
    }
}

// ---- deltas -> distances (DistanceOcclusionTool.cpp:46-61, sign :1262/:1392) ----

// Cells in order, four per thread in flight; a thread finds its first cell's row, for
// the sign, by a division and steps from there.  Whole calls without | with signs,
// us: 1501 x 400 x 300 393 | 525 (446 | 694 with a division per cell, 604 | 607 with a
// warp for 256 cells of a row), 1 x 1000 x 1000 16 | 16 (26 | 25, 179 | 180), 257 x 400
// x 300 69 | 99 (87 | 131, 171 | 172).
template <int kDim, bool kHalve, bool kSigned>
__global__ void __launch_bounds__(256) k_deltas_to_dist(const void* __restrict__ deltas, int cw,
                                                        const uint32_t* __restrict__ sign_mask, float* __restrict__ out,
                                                        int w, long long n)
{
    constexpr int kFlight = 4;
    const int ws = words_per_row(w);
    const long long threads = (long long)gridDim.x * blockDim.x, first = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long row_step = kSigned ? threads / w : 0, row0 = kSigned ? first / w : 0;
    const int x_step = kSigned ? (int)(threads - row_step * w) : 0;
    const uint32_t* srow = kSigned ? sign_mask + row0 * ws : nullptr;   // the cell's row of the mask
    int x = kSigned ? (int)(first - row0 * w) : 0;
    for (long long i0 = first; i0 < n; i0 += kFlight * threads) {
        int32_t l[kFlight];
        uint32_t sign[kFlight];
#pragma unroll
        for (int u = 0; u < kFlight; u++) {
            const long long i = i0 + u * threads;
            l[u] = 0;
            sign[u] = 0;
            if (i < n) {
                if (kDim == 2) l[u] = len(unpack2(__ldg(static_cast<const uint32_t*>(deltas) + i)));
                else l[u] = len(load3(static_cast<const int16_t*>(deltas), i));
                if (kSigned) sign[u] = (__ldg(srow + (x >> 5)) >> (x & 31)) << 31;
            }
            if (kSigned) {
                x += x_step;
                srow += row_step * ws;
                if (x >= w) {
                    x -= w;
                    srow += ws;
                }
            }
        }
#pragma unroll
        for (int u = 0; u < kFlight; u++) {
            const long long i = i0 + u * threads;
            float r = sqrtf((float)l[u]);
            // half of a square root of an integer is exact: the division by 2 in one multiplication
            if (kHalve) r = __fmul_rn(r, 0.5f);
            else if (cw != 1) r = __fdiv_rn(r, (float)cw);
            if (i < n) out[i] = __uint_as_float(__float_as_uint(r) ^ sign[u]);
        }
    }
}

// Signed images of wide rows: a warp takes 256 cells of a row, eight at a time per
// lane in flight, the signs of 32 cells being one word (1501 x 4000 13 us, 22 with
// the cells in order).
template <bool kHalve>
__global__ void __launch_bounds__(256) k_deltas_to_dist_rows(const uint32_t* __restrict__ deltas, int cw,
                                                             const uint32_t* __restrict__ sign_mask,
                                                             float* __restrict__ out, int w, long long items, int segs)
{
    const int ws = words_per_row(w), lane = threadIdx.x & 31;
    const long long warps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long it = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; it < items; it += warps) {
        const long long row = items < (1LL << 31) ? (long long)((unsigned)it / (unsigned)segs) : it / segs;
        const int x0 = (int)(it - row * segs) * 256;
        const long long first = row * w + x0;
        int32_t l[8];
        uint32_t sign[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int x = 32 * u + lane;
            l[u] = 0;
            sign[u] = 0;
            if (x0 + x < w) {
                l[u] = len(unpack2(__ldg(deltas + first + x)));
                sign[u] = (__ldg(sign_mask + row * ws + (x0 >> 5) + u) >> lane) << 31;
            }
        }
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int x = 32 * u + lane;
            float r = sqrtf((float)l[u]);
            if (kHalve) r = __fmul_rn(r, 0.5f);
            else if (cw != 1) r = __fdiv_rn(r, (float)cw);
            if (x0 + x < w) out[first + x] = __uint_as_float(__float_as_uint(r) ^ sign[u]);
        }
    }
}

// The same for volumes of rows of whole fours at 8- and 16-byte aligned arrays: a
// lane takes four cells as three 8-byte loads and stores them as one float4
// (256^3 with signs: 79 us a cell at a time, 35 us).
template <bool kHalve>
__global__ void __launch_bounds__(256) k_deltas_to_dist4(const uint2* __restrict__ deltas, int cw,
                                                         const uint32_t* __restrict__ sign_mask,
                                                         float4* __restrict__ out, int w4, long long n4)
{
    const int ws = words_per_row(4 * w4);
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (long long)gridDim.x * blockDim.x) {
        const uint2 a = __ldg(deltas + 3 * i), b = __ldg(deltas + 3 * i + 1), c = __ldg(deltas + 3 * i + 2);
        auto lo = [](uint32_t v) { return (int)(int16_t)v; };
        auto hi = [](uint32_t v) { return (int)v >> 16; };
        const int32_t l[4] = {len(C3{lo(a.x), hi(a.x), lo(a.y)}), len(C3{hi(a.y), lo(b.x), hi(b.x)}),
                              len(C3{lo(b.y), hi(b.y), lo(c.x)}), len(C3{hi(c.x), lo(c.y), hi(c.y)})};
        uint32_t sign = 0;
        if (sign_mask) {
            const unsigned row = n4 < (1LL << 31) ? (unsigned)i / (unsigned)w4 : (unsigned)(i / w4);
            const unsigned x = (unsigned)(i - (long long)row * w4) * 4;
            sign = __ldg(sign_mask + (long long)row * ws + (x >> 5)) >> (x & 31);
        }
        float r[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            r[u] = sqrtf((float)l[u]);
            if (kHalve) r[u] = __fmul_rn(r[u], 0.5f);
            else if (cw != 1) r[u] = __fdiv_rn(r[u], (float)cw);
            r[u] = __uint_as_float(__float_as_uint(r[u]) ^ (sign >> u << 31));
        }
        out[i] = make_float4(r[0], r[1], r[2], r[3]);
    }
}

void launch_deltas_to_dist(int dim, const void* deltas, int cw, const uint32_t* sign_mask, float* out, int w, int h,
                           int d, cudaStream_t st)
{
    const long long n = (long long)w * h * (dim == 3 ? d : 1);
    const long long blocks = (n + 255) / 256, cap = (long long)g_num_sms * 32;
    const int grid = (int)(blocks < cap ? blocks : cap);
    ProfScope ps("deltas_to_dist", st);
    if (dim == 3 && w % 4 == 0 && ((uintptr_t)deltas & 7) == 0 && ((uintptr_t)out & 15) == 0) {
        const long long n4 = (long long)(w / 4) * h * d, b4 = (n4 + 255) / 256;
        const int g4 = (int)(b4 < cap ? b4 : cap);
        const uint2* in = static_cast<const uint2*>(deltas);
        float4* o = reinterpret_cast<float4*>(out);
        if (cw == 2) k_deltas_to_dist4<true><<<g4, 256, 0, st>>>(in, cw, sign_mask, o, w / 4, n4);
        else k_deltas_to_dist4<false><<<g4, 256, 0, st>>>(in, cw, sign_mask, o, w / 4, n4);
        return;
    }
    if (dim == 2 && sign_mask && w >= 64) {
        const int segs = (w + 255) / 256;
        const long long items = (long long)h * segs, rb = (items + 7) / 8;
        const int gr = (int)(rb < cap ? rb : cap);
        const uint32_t* in = static_cast<const uint32_t*>(deltas);
        if (cw == 2) k_deltas_to_dist_rows<true><<<gr, 256, 0, st>>>(in, cw, sign_mask, out, w, items, segs);
        else k_deltas_to_dist_rows<false><<<gr, 256, 0, st>>>(in, cw, sign_mask, out, w, items, segs);
        return;
    }
    auto run = [&](auto signed_kern, auto unsigned_kern) {
        if (sign_mask) signed_kern<<<grid, 256, 0, st>>>(deltas, cw, sign_mask, out, w, n);
        else unsigned_kern<<<grid, 256, 0, st>>>(deltas, cw, sign_mask, out, w, n);
    };
    if (dim == 2) {
        if (cw == 2) run(k_deltas_to_dist<2, true, true>, k_deltas_to_dist<2, true, false>);
        else run(k_deltas_to_dist<2, false, true>, k_deltas_to_dist<2, false, false>);
    } else {
        if (cw == 2) run(k_deltas_to_dist<3, true, true>, k_deltas_to_dist<3, true, false>);
        else run(k_deltas_to_dist<3, false, true>, k_deltas_to_dist<3, false, false>);
    }
}

// ---- two-pass signed distance: Dist(exterior) - Dist(interior) ----
// The tool's -S path (GenerateSignedDistance, DistanceOcclusionTool.cpp:1082-1123
// 2D, :1197-1232 3D; Dist :54-61): deltas to set cells and deltas to clear cells,
// each with cw = 1, give sqrtf of each squared length, subtracted in float.
template <int kDim>
__global__ void __launch_bounds__(256) k_two_pass_dist(const void* __restrict__ ext, const void* __restrict__ intr,
                                                       float* __restrict__ out, long long n)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        int32_t a, b;
        if (kDim == 2) {
            a = len(unpack2(__ldg(static_cast<const uint32_t*>(ext) + i)));
            b = len(unpack2(__ldg(static_cast<const uint32_t*>(intr) + i)));
        } else {
            a = len(load3(static_cast<const int16_t*>(ext), i));
            b = len(load3(static_cast<const int16_t*>(intr), i));
        }
        out[i] = __fsub_rn(sqrtf((float)a), sqrtf((float)b));
    }
}

void launch_two_pass_dist(int dim, const void* ext, const void* intr, float* out, long long cells, cudaStream_t st)
{
    long long blocks = (cells + 255) / 256;
    long long cap = (long long)g_num_sms * 32;
    int grid = (int)(blocks < cap ? blocks : cap);
    ProfScope ps("two_pass_dist", st);
    if (dim == 2)
        k_two_pass_dist<2><<<grid, 256, 0, st>>>(ext, intr, out, cells);
    else
        k_two_pass_dist<3><<<grid, 256, 0, st>>>(ext, intr, out, cells);
}

}  // namespace dolk
