// k_felz.cu -- DOL::Felzenszwalb(w, h, float[]) on arbitrary float input.
//
// The reference's 1D lower envelope in its own float operations and order
// (DistanceOcclusionLib.cpp:1026-1062), columns into a transposed scratch
// field, then rows back (:1065-1085).  The envelope's float comparisons decide
// which parabola a cell gets, so a line's stack is built serially; lines are
// independent.
//
// The build is a chain of one division and compare per push or pop, at most
// 2n - 1 of them.  But its outcome is the lower hull of the points
// (q, f(q) + q^2) wherever rounding cannot have turned a decision, and the hull
// can be built in parallel.  So, one warp per line:
//   1. each lane builds the hull of a word of 32 positions (a bit per vertex),
//      and the words' hulls merge pairwise (felz_merge);
//   2. every position is checked against its neighbours on that hull, by the
//      boundaries with them.  e = 2^-24; a boundary computed from heights (a
//      difference and a division, each correctly rounded) is off by at most 2 e
//      of its size, the difference of two, the gap, by 6 e of the larger one's.
//      A vertex whose right boundary is above its left one, or another point
//      with them the other way round, by more than kFelzClear = 128 e of their
//      size is clear (in truth: by 122 e).  If no point is off by more than
//      kFelzOff = 2 e (8 e), and the vertices whose gap is not surely above zero
//      (kFelzSure) are at most kFelzTurns = 4, then along the hull boundaries
//      fall back by at most 4 x 8 e, and a point lies above an edge's line to
//      within 8 e more: from a clear vertex every later point is seen at or above
//      its right boundary, every earlier one at or below its left one, each
//      to within 40 e, so that the two stay 122 - 80 = 42 e apart, and the
//      reference, whose two boundaries are off by 2 e each, decides as on
//      exact numbers.
//      So a clear vertex is never popped, and a clear other point between two
//      clear vertices is popped at the latest by the second.
//   3. what is not clear -- ties of integer fields, now and then a near tie -- is
//      built again by the serial rule in the reference's float operations, from
//      the clear vertex before it to the clear vertex after it: pops stop at the
//      first, and nothing later reaches back over the second;
//   4. boundaries by neighbouring vertices, a binary search per cell.
// A line that step 2 finds worse than that (not finite, say) is built serially as
// a whole; step 1 so needs no bound on its rounding.  (Input that is not finite
// has no defined result: the reference leaves its stack there.  Here the bottom
// of the stack stays, whatever compares.)
//
// What bounds it: latency of the dependent steps of a warp (an SM holds one to
// three warps per scheduler).  1024 x 1024 heights, both passes: 3.47 ms with one
// thread per line and its stack in global memory; 0.26 ms with a serial build in
// shared memory by one lane; 0.11 ms with hulls in parallel.  Small integers
// (many ties) 0.16 ms (3.21); a field of nothing but ties, all serial, 0.61 ms
// (2.12).
#include <float.h>

#include "kernels.h"

namespace dolk {

constexpr int kFelzMaxLines = 8;
constexpr size_t kFelzSmemLimit = 224 * 1024;
constexpr float kFelzClear = 0x1p-17f;
constexpr float kFelzOff = 0x1p-23f;
constexpr float kFelzSure = 0x1p-21f;
constexpr int kFelzTurns = 4;

// Shared memory of a line of n cells: values, heights (value + position^2; a word
// of padding per 32, so that lanes a word apart fall in different banks),
// boundaries, hull and doubt bits, vertex positions.
struct FelzSmem {
    int vstride;   // floats between staged lines: 4 mod 32, so that the staging stores of 8 lines x 4 positions
                   // fall in different banks
    int words;
    size_t line_bytes;
};

static __host__ __device__ FelzSmem felz_smem(int n)
{
    FelzSmem s;
    s.vstride = ((n + 27) / 32) * 32 + 4;
    s.words = (n + 31) / 32;
    s.line_bytes = 4 * ((size_t)s.vstride + 33 * (size_t)s.words + n + 2 * (size_t)s.words + (n + 1) / 2);
    s.line_bytes = (s.line_bytes + 15) & ~(size_t)15;
    return s;
}

struct FelzLine {
    int n, words;
    float* f;
    float* h;       // height q at h[q + q / 32]
    float* z;       // boundary of vertex k with the one before
    uint32_t* on;   // hull vertices
    uint32_t* doubt;
    uint16_t* pos;

    __device__ __forceinline__ float height(int q) const { return h[q + (q >> 5)]; }
    // the last vertex before q at or after word lo (-1: none), the first after q before word hi (n: none)
    __device__ __forceinline__ int prev(const uint32_t* b, int q, int lo) const
    {
        int w = q >> 5;
        uint32_t m = b[w] & ((1u << (q & 31)) - 1u);
        while (!m) {
            if (--w < lo) return -1;
            m = b[w];
        }
        return 32 * w + 31 - __clz(m);
    }
    __device__ __forceinline__ int next(const uint32_t* b, int q, int hi) const
    {
        int w = q >> 5;
        uint32_t m = b[w] & ~((2u << (q & 31)) - 1u);
        while (!m) {
            if (++w >= hi) return n;
            m = b[w];
        }
        return 32 * w + __ffs(m) - 1;
    }
};

// is t on or above the segment from u to q (u < t < q)?  Scaled so that no
// difference of finite heights overflows times a distance.
__device__ __forceinline__ bool felz_over(int u, float hu, int t, float ht, int q, float hq)
{
    const float a = (hq - ht) * 0x1p-16f, b = (ht - hu) * 0x1p-16f;
    return a * (float)(t - u) <= b * (float)(q - t);
}

// the hull of word w
__device__ __forceinline__ void felz_word(const FelzLine& l, int w)
{
    const int q0 = 32 * w, q1 = min(l.n, q0 + 32);
    uint32_t bits = 1u;
    int t = q0, u = -1;
    float ht = l.height(q0), hu = 0.0f;
    for (int q = q0 + 1; q < q1; q++) {
        const float hq = l.height(q);
        while (u >= 0 && felz_over(u, hu, t, ht, q, hq)) {
            bits &= ~(1u << (t - q0));
            t = u;
            ht = hu;
            const uint32_t below = bits & ((1u << (t - q0)) - 1u);
            u = below ? q0 + 31 - __clz(below) : -1;
            if (u >= 0) hu = l.height(u);
        }
        u = t;
        hu = ht;
        t = q;
        ht = hq;
        bits |= 1u << (q - q0);
    }
    l.on[w] = bits;
}

// the hulls of words lo .. mid-1 and mid .. hi-1 into one: from the two facing
// vertices, those that lie on or above the bridge go
__device__ __forceinline__ void felz_merge(const FelzLine& l, int lo, int mid, int hi)
{
    int a = l.prev(l.on, 32 * mid, lo), b = l.next(l.on, 32 * mid - 1, hi);
    float ha = l.height(a), hb = l.height(b);
    int pa = l.prev(l.on, a, lo), nb = l.next(l.on, b, hi);
    float hpa = pa >= 0 ? l.height(pa) : 0.0f, hnb = nb < l.n ? l.height(nb) : 0.0f;
    for (;;) {
        if (pa >= 0 && felz_over(pa, hpa, a, ha, b, hb)) {
            l.on[a >> 5] &= ~(1u << (a & 31));
            a = pa;
            ha = hpa;
            pa = l.prev(l.on, a, lo);
            if (pa >= 0) hpa = l.height(pa);
        } else if (nb < l.n && felz_over(a, ha, b, hb, nb, hnb)) {
            l.on[b >> 5] &= ~(1u << (b & 31));
            b = nb;
            hb = hnb;
            nb = l.next(l.on, b, hi);
            if (nb < l.n) hnb = l.height(nb);
        } else {
            break;
        }
    }
}

// The reference's build over positions v .. e in its float operations, v staying
// at the bottom; sets the vertex bits between them.  The stack is the range's
// part of pos.
__device__ __noinline__ void felz_serial(const FelzLine& l, int v, int e)
{
    uint16_t* st = l.pos + v;
    int k = 0;
    st[0] = (uint16_t)v;
    int p = v;
    float hp = l.height(v), zp = -FLT_MAX;   // the top and its boundary
    for (int q = v + 1; q <= e; q++) {
        const float hq = l.height(q);
        float s;
        for (;;) {
            s = __fdiv_rn(hq - hp, (float)(2 * (q - p)));
            if (s > zp || k == 0) break;   // (the bottom has no boundary that counts)
            l.on[p >> 5] &= ~(1u << (p & 31));
            p = st[--k];
            hp = l.height(p);
            zp = k > 0 ? __fdiv_rn(hp - l.height(st[k - 1]), (float)(2 * (p - st[k - 1]))) : -FLT_MAX;
        }
        st[++k] = (uint16_t)q;
        p = q;
        hp = hq;
        zp = s;
        l.on[q >> 5] |= 1u << (q & 31);
    }
}

// Line l of `lines`: position q at in[q * lines + l], results at out[l * n + q]
// (both passes: columns of the field, then columns of its transpose).  A CTA
// takes L adjacent lines (32-byte runs of the input for L = 8), a warp each.
__global__ void __launch_bounds__(32 * kFelzMaxLines) k_felz_lines(const float* __restrict__ in, float* __restrict__ out,
                                                                 int lines, int n, int L)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const FelzSmem lay = felz_smem(n);
    float* F = reinterpret_cast<float*>(smem);
    const int l0 = blockIdx.x * L, nl = min(L, lines - l0);
    // staging: 8 threads per position (those past the CTA's lines idle), 4 loads in flight each
    {
        const int j = threadIdx.x & 7;
#pragma unroll 4
        for (int q = threadIdx.x >> 3; q < n; q += 4 * kFelzMaxLines)
            if (j < nl) F[j * lay.vstride + q] = in[(long long)q * lines + l0 + j];
    }
    __syncthreads();
    const int j = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (j >= nl) return;
    FelzLine l;
    l.n = n;
    l.words = lay.words;
    l.f = F + j * lay.vstride;
    l.h = reinterpret_cast<float*>(smem + (size_t)L * lay.vstride * 4 + (size_t)j * (lay.line_bytes - (size_t)lay.vstride * 4));
    l.on = reinterpret_cast<uint32_t*>(l.h + 33 * lay.words);
    l.doubt = l.on + lay.words;
    l.z = reinterpret_cast<float*>(l.doubt + lay.words);
    l.pos = reinterpret_cast<uint16_t*>(l.z + n);
    float* o = out + (long long)(l0 + j) * n;
    bool none = true;
    for (int q = lane; q < n; q += 32) {
        const float v = l.f[q];
        none &= v == FLT_MAX;
        l.h[q + (q >> 5)] = v + (float)(q * q);
    }
    if (__all_sync(0xFFFFFFFFu, none)) {   // no site on the line: every cell keeps FLT_MAX
        for (int q = lane; q < n; q += 32) o[q] = FLT_MAX;
        return;
    }
    __syncwarp();
    // 1. the hull
    for (int w = lane; w < l.words; w += 32) {
        l.doubt[w] = 0;
        felz_word(l, w);
    }
    __syncwarp();
    for (int half = 1; half < l.words; half <<= 1) {
        for (int lo = 2 * half * lane; lo + half < l.words; lo += 64 * half)
            felz_merge(l, lo, lo + half, min(lo + 2 * half, l.words));
        __syncwarp();
    }
    // 2. what is in doubt
    bool any = false;
    int bad = 0;
    for (int w = lane; w < l.words; w += 32) {
        const uint32_t bits = l.on[w];
        const int q0 = 32 * w, q1 = min(n, q0 + 32);
        int p = l.prev(l.on, q0, 0);
        const int after = l.next(l.on, q0 + 31, l.words);
        float hp = p >= 0 ? l.height(p) : 0.0f;
        int x = q0 - 1;
        float hx = 0.0f;   // the vertex at or after q + 1 that hx belongs to: x
        uint32_t doubt = 0;
        for (int q = q0; q < q1; q++) {
            const int b = q - q0;
            const bool vertex = (bits >> b) & 1u;
            if (x <= q) {
                const uint32_t rest = bits & ~((2u << b) - 1u);
                x = rest ? q0 + __ffs(rest) - 1 : after;
                if (x < n) hx = l.height(x);
            }
            const float hq = l.height(q);
            if (q > 0 && q < n - 1) {   // the ends are vertices of any build
                const float s1 = __fdiv_rn(hq - hp, (float)(2 * (q - p)));
                const float s2 = __fdiv_rn(hx - hq, (float)(2 * (x - q)));
                const float gap = vertex ? s2 - s1 : s1 - s2;
                const float size = fmaxf(fabsf(s1), fabsf(s2));
                if (!(gap > __fmaf_rn(kFelzClear, size, FLT_MIN))) {
                    doubt |= 1u << b;
                    if (!(gap >= -kFelzOff * size)) bad += kFelzTurns + 1;
                    if (vertex && !(gap > kFelzSure * size)) bad++;
                }
            }
            if (vertex) {
                p = q;
                hp = hq;
            }
        }
        l.doubt[w] = doubt;
        any |= doubt != 0;
    }
    __syncwarp();
    bad = __reduce_add_sync(0xFFFFFFFFu, min(bad, kFelzTurns + 1));
    // 3. the serial rule between clear vertices
    if (__any_sync(0xFFFFFFFFu, any)) {
        if (lane == 0) {
            auto clear_vertex = [&](int q) {
                return (l.on[q >> 5] >> (q & 31) & 1u) && !(l.doubt[q >> 5] >> (q & 31) & 1u);
            };
            int q = l.next(l.doubt, 0, l.words);   // (0 is never in doubt)
            if (bad > kFelzTurns) {
                felz_serial(l, 0, n - 1);
                q = n;
            }
            while (q < n) {
                int v = l.prev(l.on, q, 0), e = l.next(l.on, q, l.words);
                while (!clear_vertex(v)) v = l.prev(l.on, v, 0);
                while (!clear_vertex(e)) e = l.next(l.on, e, l.words);
                felz_serial(l, v, e);
                q = l.next(l.doubt, e, l.words);
            }
        }
        __syncwarp();
    }
    // 4. vertices in order, their boundaries
    int k = 0;
    for (int w0 = 0; w0 < l.words; w0 += 32) {
        const int w = w0 + lane;
        uint32_t bits = w < l.words ? l.on[w] : 0u;
        int c = __popc(bits), sum = c;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int v = __shfl_up_sync(0xFFFFFFFFu, sum, d);
            if (lane >= d) sum += v;
        }
        int at = k + sum - c;
        while (bits) {
            l.pos[at++] = (uint16_t)(32 * w + __ffs(bits) - 1);
            bits &= bits - 1;
        }
        k += __shfl_sync(0xFFFFFFFFu, sum, 31);
    }
    k--;   // the last vertex's number
    __syncwarp();
    for (int e = 1 + lane; e <= k; e += 32) {
        const int p = l.pos[e], b = l.pos[e - 1];
        l.z[e] = __fdiv_rn(l.height(p) - l.height(b), (float)(2 * (p - b)));
    }
    __syncwarp();
    // cell q belongs to the last vertex whose boundary lies below q; four cells
    // per lane and trip keep four searches in flight
    int top = 1;
    while (top <= k) top <<= 1;
    for (int q0 = lane; q0 < n; q0 += 128) {
        int e[4] = {0, 0, 0, 0};
        for (int step = top >> 1; step > 0; step >>= 1)
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int c = e[u] + step;
                if (c <= k && l.z[c] < (float)(q0 + 32 * u)) e[u] = c;
            }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int q = q0 + 32 * u;
            if (q < n) {
                const int p = l.pos[e[u]];
                o[q] = __fadd_rn((float)((q - p) * (q - p)), l.f[p]);
            }
        }
    }
}

// Lines too long for shared memory: one thread per line, the stack in global
// memory, interleaved by line for coalescing.
__device__ void felz_line_dev(int n, const float* f, long long fstride, float* out, long long ostride, int* v, float* z,
                              long long sstride)
{
    int k = 0;
    v[0] = 0;
    z[0] = -FLT_MAX;
    z[sstride] = FLT_MAX;
    for (int q = 1; q < n; q++) {
        float hq = f[q * fstride] + (float)(q * q);
        float s;
        for (;;) {
            int p = v[k * sstride];
            float hp = f[p * fstride] + (float)(p * p);
            s = __fdiv_rn(hq - hp, (float)(2 * (q - p)));
            if (s > z[k * sstride] || k == 0) break;   // (k == 0: only input that is not finite)
            k--;
        }
        k++;
        v[k * sstride] = q;
        z[k * sstride] = s;
        z[(k + 1) * sstride] = FLT_MAX;
    }
    k = 0;
    for (int q = 0; q < n; q++) {
        while (z[(k + 1) * sstride] < (float)q) k++;
        int p = v[k * sstride];
        out[q * ostride] = __fadd_rn((float)((q - p) * (q - p)), f[p * fstride]);
    }
}

__global__ void k_felz_long(const float* __restrict__ in, float* __restrict__ out, int lines, int n, int* v, float* z)
{
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= lines) return;
    felz_line_dev(n, in + l, lines, out + (long long)l * n, 1, v + l, z + l, lines);
}

size_t felz_float_workspace_bytes(int w, int h)
{
    size_t n = (size_t)(w > h ? w : h);
    size_t lines = (size_t)(w > h ? w : h);
    size_t td = ((size_t)w * h * sizeof(float) + 255) & ~(size_t)255;
    size_t vb = (n * lines * sizeof(int) + 255) & ~(size_t)255;
    size_t zb = (n + 1) * lines * sizeof(float);
    return td + vb + zb;
}

static void felz_pass(const float* in, float* out, int lines, int n, int* v, float* z, cudaStream_t st)
{
    const FelzSmem lay = felz_smem(n);
    // as many adjacent lines per CTA as keep every SM busy, at most 8 (32-byte
    // runs) and what fits in shared memory
    int L = (lines + g_num_sms - 1) / g_num_sms;
    if (L > kFelzMaxLines) L = kFelzMaxLines;
    if ((size_t)L * lay.line_bytes > kFelzSmemLimit) L = (int)(kFelzSmemLimit / lay.line_bytes);
    if (L < 1) {
        k_felz_long<<<(lines + 127) / 128, 128, 0, st>>>(in, out, lines, n, v, z);
        return;
    }
    const size_t bytes = (size_t)L * lay.line_bytes;
    cudaFuncSetAttribute(k_felz_lines, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFelzSmemLimit);
    k_felz_lines<<<(lines + L - 1) / L, 32 * kFelzMaxLines, bytes, st>>>(in, out, lines, n, L);
}

void launch_felz_float_2d(float* dist, int w, int h, void* ws, cudaStream_t st)
{
    size_t n = (size_t)(w > h ? w : h);
    char* p = static_cast<char*>(ws);
    float* td = reinterpret_cast<float*>(p);
    p += ((size_t)w * h * sizeof(float) + 255) & ~(size_t)255;
    int* v = reinterpret_cast<int*>(p);
    p += (n * n * sizeof(int) + 255) & ~(size_t)255;
    float* z = reinterpret_cast<float*>(p);
    ProfScope ps("felzenszwalb_2d", st);
    felz_pass(dist, td, w, h, v, z, st);   // columns -> td[x * h + q]
    felz_pass(td, dist, h, w, v, z, st);   // rows (columns of td) back
}

}  // namespace dolk
