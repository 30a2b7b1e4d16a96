// The samples of a round drawn one warp each.  The launch draws every sample
// whose two searches stay small (its visited nodes fit a hash table in shared
// memory) and lists the others for the CTA sampler (sampler.cuh), which draws
// them afterwards; both give the same samples bit for bit.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "common.cuh"
#include "sampler.cuh"

namespace silvan {

constexpr uint32_t kWarpLevels = 4096;  // levels per side of a search
constexpr uint32_t kWarpMeets = 4096;   // meeting edges of a sample

// A visited node, at its queue position.
struct __align__(32) BallRec {
    uint32_t st;            // side << 30 | distance from its root
    uint32_t cnt;           // predecessors
    uint64_t sigma;         // shortest paths from the root, wrapping
    uint32_t first, last;   // queue positions of the first and last predecessor
    uint32_t node;
    uint32_t hit;           // paths of the sample through the node
};
static_assert(sizeof(BallRec) == 32, "BallRec must be one sector");

// Per warp: cap visited nodes, kWarpMeets meeting edges, the queue bounds of
// 2 x kWarpLevels levels.
struct WarpSlots {
    BallRec *ball;
    uint2 *rows;        // the visited nodes' rows in the direction of their side
    uint32_t *touched;  // positions on the sample's paths
    uint2 *meet;
    uint64_t *mpre;
    uint2 *lvl;
    uint32_t cap;
};

struct WarpLaunch {
    WarpSlots slots;
    RoundHeader *hdr;
    const SegDesc *segs;
    uint32_t *list;  // work indices left to the CTA sampler, list_cap per class
    uint32_t list_cap;
};

cudaError_t warp_sampler_launch(const WarpLaunch &L, uint32_t grid, cudaStream_t stream);
int warp_sampler_per_sm();  // resident warps per SM

}  // namespace silvan
