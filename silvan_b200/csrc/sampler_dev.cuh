// Device helpers shared by the two samplers (sampler.cu, warp_sampler.cu).
#pragma once
#include <cstdint>

#include "sampler.cuh"

namespace silvan {

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

__device__ __forceinline__ uint32_t draw32(uint64_t seed, uint32_t sample, uint32_t d) {
    return philox_lo32(seed, sample, kStreamSampler, d);
}

// x mod m for a 32-bit x and a non-zero 64-bit m: x itself when m >= 2^32.
__device__ __forceinline__ uint32_t mod_u64(uint32_t x, unsigned long long m) {
    return (m >> 32) ? x : x % (uint32_t)m;
}

// A whole record in one 32-byte store.
__device__ __forceinline__ void rec_store(void *r, uint4 lo, uint4 hi) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(r), "r"(lo.x),
                 "r"(lo.y), "r"(lo.z), "r"(lo.w), "r"(hi.x), "r"(hi.y), "r"(hi.z), "r"(hi.w)
                 : "memory");
}

// A whole record in one 32-byte load through L2 (the slot is written by this
// CTA and, for shared levels, by others): words 0-3 and 4-7.
__device__ __forceinline__ void rec_load(const void *r, uint4 &lo, uint4 &hi) {
    asm volatile("ld.global.cg.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(lo.x), "=r"(lo.y), "=r"(lo.z), "=r"(lo.w), "=r"(hi.x), "=r"(hi.y),
                   "=r"(hi.z), "=r"(hi.w)
                 : "l"(r)
                 : "memory");
}

// Segment owning work index w: the last segment whose base is <= w.
__device__ __forceinline__ uint32_t segment_of(const SegDesc *segs, uint32_t nsegs, uint32_t w) {
    uint32_t l = 0, h = nsegs;
    while (h - l > 1) {
        const uint32_t mid = (l + h) >> 1;
        if (segs[mid].base <= w) l = mid;
        else h = mid;
    }
    return l;
}

__device__ __forceinline__ uint32_t ld_acquire_u32(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

}  // namespace silvan
