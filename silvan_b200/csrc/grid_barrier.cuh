// A bounded barrier over all CTAs of a cooperative launch.
#pragma once
#include <cstdint>

namespace silvan {

__device__ __forceinline__ uint32_t ld_acquire(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(uint32_t *p, uint32_t v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Over bar[0] (arrivals) and bar[1] (generation); false when this CTA gave up
// waiting after `polls` looks.  Warps come as they are: lanes that a loop left
// apart are joined first.
__device__ __forceinline__ bool grid_barrier(uint32_t *bar, uint32_t polls) {
    __syncwarp();
    __syncthreads();
    int ok = 1;
    if (threadIdx.x == 0) {
        const uint32_t gen = ld_acquire(&bar[1]);
        __threadfence();
        if (atomicAdd(&bar[0], 1u) == gridDim.x - 1) {
            bar[0] = 0u;
            __threadfence();
            st_release(&bar[1], gen + 1u);
        } else {
            uint32_t i = 0;
            while (ld_acquire(&bar[1]) == gen) {
                if (++i > polls) {
                    ok = 0;
                    break;
                }
                __nanosleep(32);
            }
        }
    }
    __syncwarp();
    return __syncthreads_and(ok) != 0;
}

// The same over one counter that starts at zero and only grows: the barrier is
// passed when it reaches `target`, the CTAs times the barriers so far.  An
// arrival without an answer and a poll of the counter itself, where the one
// above waits for two atomics' answers and two fences: for launches whose
// counter is zeroed before each (102 barriers between levels of a few
// microseconds: 731 -> 638 us).
__device__ __forceinline__ bool grid_barrier_to(uint32_t *ctr, uint32_t target, uint32_t polls) {
    __syncwarp();
    __syncthreads();
    int ok = 1;
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
        uint32_t i = 0;
        while ((int32_t)(ld_acquire(ctr) - target) < 0) {
            if (++i > polls) {
                ok = 0;
                break;
            }
            if (i > 64) __nanosleep(32);
        }
    }
    __syncwarp();
    return __syncthreads_and(ok) != 0;
}

}  // namespace silvan
