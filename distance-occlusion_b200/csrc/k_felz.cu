// k_felz.cu -- DOL::Felzenszwalb(w, h, float[]) on arbitrary float input.
//
// The reference's 1D lower envelope in its own float operations and order
// (DistanceOcclusionLib.cpp:1026-1062), columns into a transposed scratch
// field, then rows back (:1065-1085).  The envelope's float comparisons decide
// which parabola a cell gets, so a line's stack is built serially; lines are
// independent.
//
// What bounds it: the build, one decision per push or pop (at most 2n - 1 of
// them), each needing the one before.  The reference decides by a quotient
// s = (hq - hp) / (2 (q - p)) against the top entry's own quotient; dividing
// puts ~100 cycles into every link of the chain.  Here the two quotients are
// compared by cross products (felz_above), which settles all but near ties in
// a subtraction, a fused multiply-add and a compare; near ties divide.  The
// boundaries themselves follow from neighbouring entries of the finished
// stack, so all lanes divide for them at the end.  The stack lives in shared
// memory beside the line, its top entry in registers.  One warp per line: lane 0 builds, then all lanes look their cells up
// (binary search over the boundaries, which ascend by construction).
// 1024 x 1024 heights, both passes: 3.47 ms with one thread per line and its
// stack in global memory; 0.33 ms with this layout and a division per
// decision; 0.26 ms with cross products.
#include <float.h>

#include "kernels.h"

namespace dolk {

// Line l of `lines`: position q at in[q * lines + l], results at out[l * n + q]
// (both passes: columns of the field, then columns of its transpose).  A CTA
// takes L adjacent lines (32-byte runs of the input for L = 8).
struct FelzSmem {
    int stride;   // floats between staged lines: n rounded up to 4 mod 32, so that the staging stores of
                  // 8 lines x 4 positions fall in different banks
    size_t line_bytes;
};

static __host__ __device__ FelzSmem felz_smem(int n)
{
    FelzSmem s;
    s.stride = ((n + 27) / 32) * 32 + 4;
    s.line_bytes = (size_t)s.stride * 4 + (size_t)n * 16;   // values, stack entries
    return s;
}

constexpr int kFelzMaxLines = 8;
constexpr size_t kFelzSmemLimit = 224 * 1024;

// A stack entry: parabola at position pos2 / 2 of height h (value + position^2);
// num / den is its boundary with the entry below before rounding.
struct FelzEntry {
    float h, num, den, pos2;
};

// The reference's test "s > z" for s = num / den and z = e.num / e.den, both
// rounded to nearest (den, e.den > 0).  With u = e.num * den rounded and
// t = num * e.den - u (one rounding): t < 0 by more than the error of u means
// s <= z; t > 0 by more than 2^-21 |u| puts the quotients at least 2^-22 of
// their size apart, so they round to different floats.  In between (and for
// anything that overflows or is not finite) the quotients themselves decide.
// 1: above, -1: not above, 0: the quotients have to decide.
__device__ __forceinline__ int felz_above(float num, float den, const FelzEntry& e)
{
    const float u = __fmul_rn(e.num, den);
    const float t = __fmaf_rn(num, e.den, -u);
    const float m = __fmaf_rn(fabsf(u), 0x1p-21f, 0x1p-100f);
    return t > m ? 1 : (t < -m ? -1 : 0);
}

__device__ __noinline__ bool felz_above_divided(float num, float den, float enum_, float eden)
{
    return __fdiv_rn(num, den) > __fdiv_rn(enum_, eden);
}

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
            if (j < nl) F[j * lay.stride + q] = in[(long long)q * lines + l0 + j];
    }
    __syncthreads();
    const int j = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (j >= nl) return;
    const float* f = F + j * lay.stride;
    float4* st = reinterpret_cast<float4*>(smem + (size_t)L * lay.stride * 4) + (size_t)j * n;
    int k = 0;
    if (lane == 0) {
        // the first entry has no boundary below it: one far to the left stands
        // in, and a test that still comes out "not above" leaves it in place
        FelzEntry e{f[0], -1e30f, 1.0f, 0.0f};
        float4* top = st;
        *top = make_float4(e.h, e.num, e.den, e.pos2);
        float fq = n > 1 ? f[1] : 0.0f, q2 = 2.0f;
#pragma unroll 1
        for (int q = 1; q < n; q++, q2 += 2.0f) {
            const float hq = fq + (float)(q * q);
            fq = f[q + 1 < n ? q + 1 : q];
            float num, den;
#pragma unroll 1
            for (;;) {
                num = hq - e.h;
                den = q2 - e.pos2;
                const int a = felz_above(num, den, e);
                if (a > 0) break;
                if (a == 0 && felz_above_divided(num, den, e.num, e.den)) break;
                if (top == st) break;
                const float4 v = *--top;
                e = FelzEntry{v.x, v.y, v.z, v.w};
            }
            e = FelzEntry{hq, num, den, q2};
            *++top = make_float4(hq, num, den, q2);
        }
        k = (int)(top - st);
    }
    __syncwarp();
    k = __shfl_sync(0xFFFFFFFFu, k, 0);
    for (int e = 1 + lane; e <= k; e += 32) st[e].y = __fdiv_rn(st[e].y, st[e].z);
    __syncwarp();
    // cell q belongs to the last entry whose boundary lies below q; four cells
    // per lane and trip keep four searches in flight
    float* o = out + (long long)(l0 + j) * n;
    int top = 1;
    while (top <= k) top <<= 1;
    for (int q0 = lane; q0 < n; q0 += 128) {
        int e[4] = {0, 0, 0, 0};
        for (int step = top >> 1; step > 0; step >>= 1)
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int c = e[u] + step;
                if (c <= k && st[c].y < (float)(q0 + 32 * u)) e[u] = c;
            }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int q = q0 + 32 * u;
            if (q < n) {
                const int p = (int)st[e[u]].w >> 1;
                o[q] = __fadd_rn((float)((q - p) * (q - p)), f[p]);
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
