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

// Grid barrier for a cooperative launch (all CTAs resident).  The wait gives
// up after `limit_ns`, sets *err and returns false in every thread of the CTA.
__device__ __forceinline__ bool grid_barrier(unsigned* count, unsigned* gen, int* err, unsigned long long limit_ns)
{
    __syncthreads();
    int ok = 1;
    if (threadIdx.x == 0) {
        volatile unsigned* vg = gen;
        const unsigned g = *vg;
        __threadfence();
        if (atomicAdd(count, 1u) == gridDim.x - 1) {
            atomicExch(count, 0u);
            __threadfence();
            atomicAdd(gen, 1u);
        } else {
            const unsigned long long t0 = global_ns();
            while (*vg == g) {
                __nanosleep(32);
                if (global_ns() - t0 > limit_ns) {
                    atomicExch(err, 2);
                    ok = 0;
                    break;
                }
            }
        }
        __threadfence();
    }
    return __syncthreads_and(ok);
}

}  // namespace dolk
