// grid_barrier.cuh -- a bounded grid-wide barrier for cooperative launches.
#pragma once

namespace dolk {

constexpr unsigned long long kGridWaitNs = 20ull * 1000 * 1000 * 1000;   // 20 s per wait

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Grid barrier for a cooperative launch (all CTAs resident): `count` counts
// arrivals over the whole launch (zero at its start), `passed` the barriers
// that this CTA has been through (kept by the caller, the same in all
// threads).  The wait gives up after kGridWaitNs, sets *err and returns false in
// every thread of the CTA.
__device__ __forceinline__ bool grid_barrier(unsigned* count, unsigned& passed, int* err)
{
    passed++;
    __syncthreads();
    int ok = 1;
    if (threadIdx.x == 0) {
        const unsigned target = passed * gridDim.x;
        __threadfence();
        atomicAdd(count, 1u);
        const unsigned long long t0 = global_ns();
        for (unsigned polls = 1;; polls++) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
            if ((int)(v - target) >= 0) break;
            if (polls % 64 == 0 && global_ns() - t0 > kGridWaitNs) {
                atomicExch(err, 2);
                ok = 0;
                break;
            }
        }
        __threadfence();
    }
    return __syncthreads_and(ok);
}

}  // namespace dolk
