// Device-side CSR preparation (see graph_dev.cuh).
#include "graph_dev.cuh"

namespace silvan {

namespace {

// Offsets above the entry count are clamped to it and flagged, so that no
// later kernel reads past the adjacency array.
__global__ void narrow_offsets_kernel(const uint64_t *in, uint32_t *out, uint32_t count,
                                      uint64_t limit, uint32_t *bad) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count;
         i += gridDim.x * blockDim.x) {
        const uint64_t v = in[i];
        if (v > limit) atomicOr(bad, 1u);
        out[i] = (uint32_t)(v > limit ? limit : v);
    }
}

// 64-bit finaliser (Steele, Lea, Flood, "Fast splittable pseudorandom number
// generators", OOPSLA 2014).
__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}

// The rows' invariants, and sums over all entries that tell whether two directions
// hold the same edges.  sums[0..1] += the entries (v, y) under two mixes (fwd),
// sums[2..3] the entries the other way round, (y, v) (bwd): two lists of entries
// give the same sums when they hold the same entries, and different ones, but for
// a chance of 2^-128, when they do not.  One pass over the adjacency for both (16 M
// entries: the upload of R-MAT 19 took 3 % longer with a pass of its own for the
// sums).  One warp per row; rows of more than kLongRow entries wait for the whole
// CTA (with one warp for a hub's row the upload of undirected R-MAT 17 took 1.44 ms
// instead of 1.33).
constexpr uint32_t kLongRow = 512, kLongRows = 256;  // and how many a CTA keeps

__global__ void validate_rows_kernel(const uint32_t *off, const uint32_t *adj, uint32_t n,
                                     uint32_t *bad, int fwd, int bwd, unsigned long long *sums) {
    __shared__ uint32_t later[kLongRows], n_later;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    unsigned long long a[4] = {0, 0, 0, 0};
    bool ok = true;
    if (threadIdx.x == 0) n_later = 0u;
    __syncthreads();
    const auto look = [&](uint32_t v, uint32_t b, uint32_t k) {
        const uint32_t y = adj[k];
        if (y >= n || (k > b && adj[k - 1] >= y)) ok = false;
        const unsigned long long f = (unsigned long long)v << 32 | y;
        const unsigned long long r = (unsigned long long)y << 32 | v;
        if (fwd) {
            a[0] += mix64(f + 0x9e3779b97f4a7c15ull);
            a[1] += mix64(f ^ 0xd1b54a32d192ed03ull);
        }
        if (bwd) {
            a[2] += mix64(r + 0x9e3779b97f4a7c15ull);
            a[3] += mix64(r ^ 0xd1b54a32d192ed03ull);
        }
    };
    for (uint32_t v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < n; v += nw) {
        const uint32_t b = off[v], e = off[v + 1];
        if (e < b) ok = false;
        if (e > b && e - b > kLongRow) {
            uint32_t at = 0;
            if (lane == 0) at = atomicAdd(&n_later, 1u);
            at = __shfl_sync(0xffffffffu, at, 0);
            if (at < kLongRows) {
                if (lane == 0) later[at] = v;
                continue;
            }
        }
        for (uint32_t k = b + lane; k < e; k += 32) look(v, b, k);
        __syncwarp();
    }
    __syncwarp();
    __syncthreads();
    const uint32_t m = min(n_later, kLongRows);
    for (uint32_t j = 0; j < m; j++) {
        const uint32_t v = later[j], b = off[v], e = off[v + 1];
        for (uint32_t k = b + threadIdx.x; k < e; k += blockDim.x) look(v, b, k);
    }
    __syncwarp();
    if (__any_sync(0xffffffffu, !ok) && lane == 0) atomicOr(bad, 1u);
    for (int i = 0; i < 4; i++) {
        for (int o = 16; o > 0; o >>= 1) a[i] += __shfl_xor_sync(0xffffffffu, a[i], o);
        if (lane == 0 && a[i]) atomicAdd(&sums[i], a[i]);
    }
}

__global__ void make_rows_kernel(const uint32_t *off, uint2 *rows, uint32_t n) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
        rows[v] = make_uint2(off[v], off[v + 1]);
}

}  // namespace

cudaError_t make_rows(const uint32_t *off, uint2 *rows, uint32_t n, cudaStream_t s) {
    make_rows_kernel<<<592, 256, 0, s>>>(off, rows, n);
    return cudaGetLastError();
}

cudaError_t narrow_offsets(const uint64_t *in, uint32_t *out, uint32_t count, uint64_t limit,
                           uint32_t *bad, cudaStream_t s) {
    narrow_offsets_kernel<<<592, 256, 0, s>>>(in, out, count, limit, bad);
    return cudaGetLastError();
}

cudaError_t validate_rows(const uint32_t *off, const uint32_t *adj, uint32_t n, uint32_t *bad,
                          bool fwd, bool bwd, unsigned long long *sums, cudaStream_t s) {
    validate_rows_kernel<<<1184, 256, 0, s>>>(off, adj, n, bad, fwd ? 1 : 0, bwd ? 1 : 0, sums);
    return cudaGetLastError();
}

}  // namespace silvan
