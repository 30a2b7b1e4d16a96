// Components and the diameter bound of an undirected graph on the device,
// identical to the reference's compute_cc + estimate_diameter
// (silvan/src/Graph.cpp:109-316) for undirected graphs:
//   * Tarjan's iterative DFS starts from the roots in ascending id order and
//     an undirected component is one strongly connected component, numbered
//     when its DFS finishes, so component c is the one whose smallest node id
//     is the c-th smallest of all components' smallest ids;
//   * the pivot of a component is its node of largest degree sum, the lowest
//     id on ties (compute_pivot, :204-214);
//   * no edge joins two components, so the AllCCUpperBound recursion reduces
//     to max over components of ecc_f(pivot) + ecc_b(pivot) = 2 ecc(pivot),
//     the eccentricity being the distance of the last node of the BFS from
//     the pivot (compute_ecc_in_scc, :238-270).
// Components: every node starts under its smallest neighbour and the trees are
// flattened; a lock-free union-find over the edges then links what is left,
// always the larger root under the smaller one (so every root is its
// component's smallest id); then every node's root and a prefix count of the
// roots.
// Eccentricities: one breadth-first search from all pivots at once (the
// components are disjoint), all levels in one launch.
//
// Directed graphs: their component numbers are the completion order of the
// reference's sequential DFS (the void test of the sampler compares them, so
// the numbering must be that DFS's, and a depth-first order is inherently
// sequential); the host computes them, and device_directed_bound computes
// the pivots, the eccentricities and the AllCCUpperBound recursion from them
// on the device.
#include <cub/cub.cuh>

#include <vector>

#include "components.h"
#include "grid_barrier.cuh"

namespace silvan {

namespace {

#define CC_CK(x)                                                                    \
    do {                                                                            \
        cudaError_t e_ = (x);                                                       \
        if (e_ != cudaSuccess) return cuda_status(e_, "device components");         \
    } while (0)
#define CC_RK(x)                                                                    \
    do {                                                                            \
        int r_ = (x);                                                               \
        if (r_ != SILVAN_OK) return r_;                                             \
    } while (0)

__device__ __forceinline__ uint32_t find_root(uint32_t *parent, uint32_t x) {
    uint32_t p = __ldcg(&parent[x]);
    while (p != x) {
        const uint32_t gp = __ldcg(&parent[p]);
        if (gp != p) parent[x] = gp;  // path halving; a stale value is still an ancestor
        x = p;
        p = gp;
    }
    return x;
}

// A node's smallest neighbour, if that is smaller, is its parent: a forest that
// needs no links.
__global__ void cc_init_kernel(const uint32_t *off, const uint32_t *adj, uint32_t *parent,
                               uint32_t n) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n;
         v += gridDim.x * blockDim.x) {
        const uint32_t b = off[v], e = off[v + 1];
        parent[v] = b < e ? min(v, adj[b]) : v;
    }
}

// Pointer jumping: every thread moves its node's parent to the grandparent until
// that is a root, and as the others do the same each step doubles the way.  No
// links are made meanwhile, so every root found is the tree's.
__global__ void cc_flatten_kernel(uint32_t *parent, uint32_t n) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n;
         v += gridDim.x * blockDim.x) {
        uint32_t p = __ldcg(&parent[v]);
        for (uint32_t gp; (gp = __ldcg(&parent[p])) != p; p = gp) parent[v] = gp;
    }
}

// The last row that starts at or before entry k (it holds the entry): a 32-way
// search by the whole warp.
__device__ __forceinline__ uint32_t row_of_entry(const uint32_t *off, uint32_t n, uint32_t k) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t l = 0, h = n;  // off[l] <= k, and off[h] > k or h == n
    while (h - l > 1) {
        const uint32_t step = (h - l + 31u) / 32u;
        const uint32_t i = l + lane * step;
        const uint32_t c = (uint32_t)__popc(
            __ballot_sync(0xffffffffu, i < h && off[i] <= k));  // lane 0 always counts
        h = min(h, l + c * step);
        l = l + (c - 1u) * step;
    }
    return l;
}

// Every edge (u, w) unites the two sets.  A warp takes a chunk of entries wherever
// they lie, so that rows of 2 and of 100,000 entries keep all lanes busy (with a
// warp per row the 490,000 rows of a lattice took 356 us; now 58, after 43 for
// the sample), and knows their rows from the ends of 32 rows, one in each lane.
__global__ void cc_union_kernel(const uint32_t *off, const uint32_t *adj, uint32_t n, uint32_t m,
                                uint32_t *parent) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t chunk = min(32u, m / (32u * warps) + 1u) * 32u;  // 32 to 1,024 entries
    const uint32_t chunks = m / chunk + (m % chunk ? 1u : 0u);
    for (uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < chunks; c += warps) {
        uint32_t pos = c * chunk;
        const uint32_t k1 = min(m - pos, chunk) + pos;
        uint32_t r = row_of_entry(off, n, pos);
        uint32_t end = off[min(r + 1u + lane, n)];  // where row r + lane ends
        while (pos < k1) {
            uint32_t wend = __shfl_sync(0xffffffffu, end, 31);
            if (wend <= pos) {
                r += 32u;
                end = off[min(r + 1u + lane, n)];
                wend = __shfl_sync(0xffffffffu, end, 31);
                if (wend <= pos) {  // many empty rows
                    r = row_of_entry(off, n, pos);
                    end = off[min(r + 1u + lane, n)];
                    wend = __shfl_sync(0xffffffffu, end, 31);
                }
            }
            const uint32_t lim = min(k1, wend), k = pos + lane;
            uint32_t row = 0;  // rows of the window that end at or before k
#pragma unroll
            for (uint32_t s = 16; s > 0; s >>= 1)
                if (__shfl_sync(0xffffffffu, end, row + s - 1u) <= k) row += s;
            if (lane < lim - pos) {
                const uint32_t u = r + row, w = adj[k];
                if (w < u) {  // each undirected edge once
                    uint32_t a = find_root(parent, u), b = find_root(parent, w);
                    while (a != b) {
                        if (a > b) {
                            const uint32_t t = a;
                            a = b;
                            b = t;
                        }
                        // link the larger root b under the smaller a, if b is still a root
                        const uint32_t old = atomicCAS(&parent[b], b, a);
                        if (old == b) break;
                        a = find_root(parent, a);
                        b = find_root(parent, old);
                    }
                }
            }
            __syncwarp();
            pos = lim - pos > 32u ? pos + 32u : lim;
        }
    }
}

// After the unions: every node's root, read-only (a compressing find here
// could overwrite another thread's final answer with an older ancestor).
__global__ void cc_compress_kernel(const uint32_t *parent, uint32_t n, uint32_t *root,
                                   uint32_t *is_root) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        uint32_t x = v, p = parent[v];
        while (p != x) {
            x = p;
            p = parent[x];
        }
        root[v] = x;
        is_root[v] = x == v ? 1u : 0u;
    }
}

// The largest key of each component, from one (component, key) a lane (of the
// warp's active lanes, all 32 or the first few): one atomic for a warp whose
// lanes lie in one component, and only where the key exceeds what is there.
// 490,000 atomics on the one address of a giant component took 320 us.
__device__ __forceinline__ void component_max(unsigned long long *best, uint32_t c,
                                              unsigned long long key) {
    const uint32_t act = __activemask();
    bool first = true;
    if (act == 0xffffffffu && __match_any_sync(0xffffffffu, c) == 0xffffffffu) {
        const uint32_t hi = __reduce_max_sync(0xffffffffu, (uint32_t)(key >> 32));
        const uint32_t lo = __reduce_max_sync(
            0xffffffffu, (uint32_t)(key >> 32) == hi ? (uint32_t)key : 0u);
        key = (unsigned long long)hi << 32 | lo;
        first = (threadIdx.x & 31) == 0;
    }
    if (first && key > __ldcg(&best[c])) atomicMax(&best[c], key);
}

// cc[v] = number of roots below v's root; the pivot key of each component:
// degree sum (2 x degree) in the high word, the inverted id in the low word.
__global__ void cc_number_kernel(const uint32_t *root, const uint32_t *rank, const uint32_t *off,
                                 uint32_t n, uint32_t *cc, unsigned long long *pivot_key) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const uint32_t c = rank[root[v]];
        cc[v] = c;
        const unsigned long long deg2 = 2ull * (off[v + 1] - off[v]);
        component_max(pivot_key, c, (deg2 << 32) | (0xffffffffull - v));
    }
}

__global__ void bfs_seed_kernel(const unsigned long long *pivot_key, uint32_t ncomp,
                                uint32_t *seen, uint32_t *queue) {
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < ncomp;
         c += gridDim.x * blockDim.x) {
        const uint32_t p = 0xffffffffu - (uint32_t)(pivot_key[c] & 0xffffffffull);
        seen[p] = 1;
        queue[c] = p;
    }
}

// The breadth-first searches from all pivots at once, each inside its component
// (the components are disjoint; where edges lead out of a component, cc keeps
// the search inside), in one cooperative launch: a lattice has a hundred levels
// of a few hundred nodes, and a launch, a copy of the count and a wait for it
// took 25 us for each where a level in here takes 5 (one CTA of 512 threads an
// SM: 492 us for all of 490,000 nodes; of 1,024: 620, of 128: 581).
//
// queue holds the pivots and gets every node once; a level is the part that the
// level before appended.  A warp takes a few nodes of the level, as many as
// leave no warp without work (at most 32), and goes through their entries 32 at
// a time; rows of more than kLongRow entries are left to all warps together
// after the others.  Counts are kept three levels apart, so that the one being
// zeroed is not read any more and not yet appended to.
//
// ctl: [0..2] nodes appended, [3..5] long rows, [6] the barrier, [8] the
// deepest level, [9] set when a wait gave up.  ecc (where given) gets each
// component's eccentricity.
constexpr int kBfsThreads = 512;
constexpr uint32_t kLongRow = 2048;
constexpr uint32_t kBfsCtl = 10;
constexpr uint32_t kBfsPolls = 1u << 26;  // a minute: a level may hold all of a large graph

struct BfsArgs {
    const uint32_t *off, *adj;
    const uint32_t *cc;  // null: no edge leaves a component
    uint32_t *queue, *seen, *long_rows, *ctl;
    int32_t *ecc;  // null: not wanted
    uint32_t ncomp;
};

// One entry a lane: nodes not seen yet join the next level.
// `look` spares the atomic where a look shows the node was seen; on a narrow
// level the look is one more wait in a chain of waits.
__device__ __forceinline__ void bfs_visit(const BfsArgs &a, bool act, uint32_t k, uint32_t cu,
                                          int32_t level, bool look, uint32_t *next,
                                          uint32_t *next_count) {
    bool join = false;
    uint32_t w = 0;
    if (act) {
        w = a.adj[k];
        join = (!a.cc || a.cc[w] == cu) && (!look || __ldcg(&a.seen[w]) == 0u) &&
               atomicExch(&a.seen[w], 1u) == 0u;
    }
    const uint32_t mask = __ballot_sync(0xffffffffu, join);
    if (!mask) return;
    const uint32_t lane = threadIdx.x & 31;
    uint32_t at = 0;
    if (lane == 0) at = atomicAdd(next_count, (uint32_t)__popc(mask));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (join) {
        next[at + (uint32_t)__popc(mask & ((1u << lane) - 1u))] = w;
        if (a.ecc) a.ecc[cu] = level + 1;  // levels rise: the last one written stays
    }
}

__global__ void __launch_bounds__(kBfsThreads, 1) bfs_kernel(const BfsArgs a) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    uint32_t count = a.ncomp, lo = 0, passed = 0;
    int32_t level = 0;
    for (;; level++) {
        const uint32_t now = (uint32_t)level % 3u, nxt = (now + 1u) % 3u, old = (now + 2u) % 3u;
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            a.ctl[old] = 0u;
            a.ctl[3u + nxt] = 0u;
        }
        uint32_t *next = a.queue + lo + count, *next_count = &a.ctl[nxt];
        const uint32_t group = min(32u, count / warps + (count % warps ? 1u : 0u));
        for (uint32_t i0 = warp * group; i0 < count; i0 += warps * group) {
            uint32_t b = 0, len = 0, cu = 0;
            if (lane < group && i0 + lane < count) {
                const uint32_t u = __ldcg(&a.queue[lo + i0 + lane]);
                b = a.off[u];
                len = a.off[u + 1] - b;
                if (a.cc) cu = a.cc[u];
                if (len > kLongRow) {
                    a.long_rows[atomicAdd(&a.ctl[3u + now], 1u)] = u;
                    len = 0;
                }
            }
            uint32_t ends = len;  // inclusive prefix
#pragma unroll
            for (uint32_t o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, ends, o);
                if (lane >= o) ends += y;
            }
            const uint32_t total = __shfl_sync(0xffffffffu, ends, 31);
            for (uint32_t it = 0; it < total; it += 32u) {
                const uint32_t item = it + lane;
                uint32_t row = 0;
#pragma unroll
                for (uint32_t s = 16; s > 0; s >>= 1)
                    if (__shfl_sync(0xffffffffu, ends, row + s - 1u) <= item) row += s;
                const uint32_t k = __shfl_sync(0xffffffffu, b + len - ends, row) + item;
                const uint32_t c = __shfl_sync(0xffffffffu, cu, row);
                bfs_visit(a, item < total, k, c, level, group > 8u, next, next_count);
            }
        }
        if (!grid_barrier_to(a.ctl + 6, passed += gridDim.x, kBfsPolls)) break;
        const uint32_t nl = __ldcg(&a.ctl[3u + now]);
        if (nl) {
            for (uint32_t j = 0; j < nl; j++) {
                const uint32_t u = __ldcg(&a.long_rows[j]);
                const uint32_t b = a.off[u], len = a.off[u + 1] - b;
                const uint32_t c = a.cc ? a.cc[u] : 0u;
                for (uint32_t i = warp * 32u; i < len; i += warps * 32u)
                    bfs_visit(a, i + lane < len, b + i + lane, c, level, true, next, next_count);
            }
            if (!grid_barrier_to(a.ctl + 6, passed += gridDim.x, kBfsPolls)) break;
        }
        lo += count;
        count = __ldcg(next_count);
        if (count == 0u) {
            if (blockIdx.x == 0 && threadIdx.x == 0) a.ctl[8] = (uint32_t)level;
            return;
        }
    }
    if (threadIdx.x == 0) atomicExch(&a.ctl[9], 1u);
}

// Queues the search from the ncomp seeded pivots.
cudaError_t launch_bfs(const BfsArgs &a, cudaStream_t st) {
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaMemsetAsync(a.ctl, 0, 4 * kBfsCtl, st);
    if (e != cudaSuccess) return e;
    BfsArgs args = a;
    void *params[] = {&args};
    return cudaLaunchCooperativeKernel((const void *)bfs_kernel, dim3((unsigned)sms),
                                       dim3(kBfsThreads), params, 0, st);
}

// ---- directed graphs: the diameter bound over given component ids --------

// Pivot key of every component: out + in degree in the high word, the
// inverted id in the low word (largest degree sum, lowest id on ties).
__global__ void dir_pivot_kernel(const uint32_t *oo, const uint32_t *io, const uint32_t *cc,
                                 uint32_t n, unsigned long long *pivot_key) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const unsigned long long d = (unsigned long long)(oo[v + 1] - oo[v]) + (io[v + 1] - io[v]);
        component_max(pivot_key, cc[v], (d << 32) | (0xffffffffull - v));
    }
}

// Edges between different components, as (source component, target
// component); every one goes to a smaller id (Tarjan numbers a component
// after every component it reaches).
__global__ void dir_inter_kernel(const uint32_t *off, const uint32_t *adj, const uint32_t *cc,
                                 uint32_t n, uint2 *inter, unsigned long long *n_inter,
                                 unsigned long long cap, uint32_t *bad) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < n; u += warps) {
        const uint32_t cu = cc[u];
        for (uint32_t k = off[u] + lane; k < off[u + 1]; k += 32) {
            const uint32_t cw = cc[adj[k]];
            if (cw == cu) continue;
            if (cw > cu) atomicExch(bad, 1u);
            const unsigned long long i = atomicAdd(n_inter, 1ull);
            if (i < cap) inter[i] = make_uint2(cu, cw);
        }
    }
}

// One pass of the AllCCUpperBound recursion (silvan/src/Graph.cpp:298-306)
// as a fixpoint: fp[c] = max(ecc_f[c], ecc_f[c] + 1 + ecc_b[d] + fp[d]) over
// the edges c -> d.  Passes repeat until nothing grows; the result is the
// recursion's, which the reference evaluates in ascending component order.
__global__ void dir_dp_kernel(const uint2 *inter, unsigned long long m, const int32_t *ecc_f,
                              const int32_t *ecc_b, int32_t *fp, uint32_t *changed) {
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < m;
         i += (unsigned long long)gridDim.x * blockDim.x) {
        const uint2 e = inter[i];
        const int32_t cand = ecc_f[e.x] + 1 + ecc_b[e.y] + __ldcg(&fp[e.y]);
        if (cand > __ldcg(&fp[e.x]) && atomicMax(&fp[e.x], cand) < cand) *changed = 1u;
    }
}

__global__ void dir_diam_kernel(const int32_t *fp, const int32_t *ecc_b, uint32_t ncomp,
                                unsigned int *diam) {
    uint32_t mx = 0;
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < ncomp;
         c += gridDim.x * blockDim.x)
        mx = max(mx, (uint32_t)(fp[c] + ecc_b[c]));
    for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) atomicMax(diam, mx);
}

}  // namespace

int device_directed_bound(DeviceGraph &G, cudaStream_t st) {
    const uint32_t n = G.n, ncomp = G.ncomp;
    std::vector<void *> bufs;
    struct Free {
        std::vector<void *> &b;
        ~Free() {
            for (void *p : b) device_free(p);
        }
    } fr{bufs};
    auto get = [&](void **p, size_t bytes) -> int {
        int rc = device_alloc(p, bytes);
        if (rc == SILVAN_OK) bufs.push_back(*p);
        return rc;
    };
    uint32_t *queue = nullptr, *seen = nullptr, *long_rows = nullptr, *ctl = nullptr,
             *flag = nullptr;
    int32_t *ecc_f = nullptr, *ecc_b = nullptr, *fp = nullptr;
    unsigned long long *pivot_key = nullptr, *n_inter = nullptr;
    unsigned int *d_diam = nullptr;
    CC_RK(get((void **)&queue, 4ull * n));
    CC_RK(get((void **)&seen, 4ull * n));
    CC_RK(get((void **)&long_rows, 4ull * (std::max(G.m, G.m_in) / kLongRow + 1)));
    CC_RK(get((void **)&ctl, 4ull * 2 * kBfsCtl));
    CC_RK(get((void **)&flag, 16));
    CC_RK(get((void **)&n_inter, 8));
    CC_RK(get((void **)&d_diam, 4));
    CC_RK(get((void **)&pivot_key, 8ull * ncomp));
    CC_RK(get((void **)&ecc_f, 4ull * ncomp));
    CC_RK(get((void **)&ecc_b, 4ull * ncomp));
    CC_RK(get((void **)&fp, 4ull * ncomp));
    CC_CK(cudaMemsetAsync(pivot_key, 0, 8ull * ncomp, st));
    CC_CK(cudaMemsetAsync(ecc_f, 0, 4ull * ncomp, st));
    CC_CK(cudaMemsetAsync(ecc_b, 0, 4ull * ncomp, st));
    CC_CK(cudaMemsetAsync(d_diam, 0, 4, st));
    CC_CK(cudaMemsetAsync(n_inter, 0, 8, st));
    CC_CK(cudaMemsetAsync(flag, 0, 16, st));
    dir_pivot_kernel<<<592, 256, 0, st>>>(G.d_out_off, G.d_in_off, G.d_cc, n, pivot_key);
    CC_CK(cudaGetLastError());
    // eccentricity of every pivot inside its component, forward then backward
    // (compute_ecc_in_scc, silvan/src/Graph.cpp:238-270)
    for (int dir = 0; dir < 2; dir++) {
        CC_CK(cudaMemsetAsync(seen, 0, 4ull * n, st));
        bfs_seed_kernel<<<64, 256, 0, st>>>(pivot_key, ncomp, seen, queue);
        CC_CK(cudaGetLastError());
        CC_CK(launch_bfs(BfsArgs{dir == 0 ? G.d_out_off : G.d_in_off,
                                 dir == 0 ? G.d_out_adj : G.d_in_adj, G.d_cc, queue, seen,
                                 long_rows, ctl + dir * kBfsCtl, dir == 0 ? ecc_f : ecc_b, ncomp},
                         st));
    }
    // the recursion over the condensation
    const uint64_t m = G.m;
    uint2 *inter = nullptr;
    CC_RK(get((void **)&inter, 8ull * std::max<uint64_t>(m, 1)));
    dir_inter_kernel<<<1184, 256, 0, st>>>(G.d_out_off, G.d_out_adj, G.d_cc, n, inter, n_inter, m,
                                           flag + 1);
    CC_CK(cudaMemcpyAsync(fp, ecc_f, 4ull * ncomp, cudaMemcpyDeviceToDevice, st));
    unsigned long long mi = 0;
    uint32_t badf = 0, bfs[2 * kBfsCtl];
    CC_CK(cudaMemcpyAsync(bfs, ctl, sizeof(bfs), cudaMemcpyDeviceToHost, st));
    CC_CK(cudaMemcpyAsync(&mi, n_inter, 8, cudaMemcpyDeviceToHost, st));
    CC_CK(cudaMemcpyAsync(&badf, flag + 1, 4, cudaMemcpyDeviceToHost, st));
    CC_CK(cudaStreamSynchronize(st));
    if (bfs[9] || bfs[kBfsCtl + 9]) {
        set_error("the breadth-first searches of the diameter bound did not end");
        return SILVAN_E_TIMEOUT;
    }
    if (badf || mi > m) {
        set_error("component ids are not in the reference's completion order");
        return SILVAN_E_STATE;
    }
    // Pass p settles every component whose longest chain of descendants has
    // p edges, so shallow condensations (small-world graphs) take a few
    // passes; a deep one (a long chain of components) is finished by the
    // recursion in ascending order on the host copy, which directed graphs
    // keep for the component numbering.
    constexpr uint32_t kMaxPasses = 64;
    for (uint32_t pass = 0;; pass++) {
        uint32_t changed = 0;
        CC_CK(cudaMemsetAsync(flag, 0, 4, st));
        if (mi) dir_dp_kernel<<<1184, 256, 0, st>>>(inter, mi, ecc_f, ecc_b, fp, flag);
        CC_CK(cudaGetLastError());
        CC_CK(cudaMemcpyAsync(&changed, flag, 4, cudaMemcpyDeviceToHost, st));
        CC_CK(cudaStreamSynchronize(st));
        if (!changed) break;
        if (pass + 1 >= kMaxPasses) {
            if (!G.has_host || G.cc.size() != n) {
                set_error("diameter recursion needs the host copy of a deep condensation");
                return SILVAN_E_STATE;
            }
            std::vector<uint32_t> ef(ncomp), eb(ncomp);
            CC_CK(cudaMemcpyAsync(ef.data(), ecc_f, 4ull * ncomp, cudaMemcpyDeviceToHost, st));
            CC_CK(cudaMemcpyAsync(eb.data(), ecc_b, 4ull * ncomp, cudaMemcpyDeviceToHost, st));
            CC_CK(cudaStreamSynchronize(st));
            G.diameter = diameter_recursion(G.host, G.cc, ncomp, ef, eb);
            return SILVAN_OK;
        }
    }
    dir_diam_kernel<<<64, 256, 0, st>>>(fp, ecc_b, ncomp, d_diam);
    CC_CK(cudaGetLastError());
    unsigned int diam = 0;
    CC_CK(cudaMemcpyAsync(&diam, d_diam, 4, cudaMemcpyDeviceToHost, st));
    CC_CK(cudaStreamSynchronize(st));
    G.diameter = diam;
    return SILVAN_OK;
}

int device_undirected_components(DeviceGraph &G, cudaStream_t st) {
    const uint32_t n = G.n;
    std::vector<void *> bufs;
    struct Free {
        std::vector<void *> &b;
        ~Free() {
            for (void *p : b) device_free(p);
        }
    } fr{bufs};
    auto get = [&](void **p, size_t bytes) -> int {
        int rc = device_alloc(p, bytes);
        if (rc == SILVAN_OK) bufs.push_back(*p);
        return rc;
    };
    uint32_t *parent = nullptr, *root = nullptr, *is_root = nullptr, *rank = nullptr,
             *queue = nullptr, *seen = nullptr, *long_rows = nullptr, *ctl = nullptr;
    unsigned long long *pivot_key = nullptr;
    CC_RK(get((void **)&parent, 4ull * n));
    CC_RK(get((void **)&root, 4ull * n));
    CC_RK(get((void **)&is_root, 4ull * n));
    CC_RK(get((void **)&rank, 4ull * (n + 1)));
    CC_RK(get((void **)&queue, 4ull * n));
    CC_RK(get((void **)&seen, 4ull * n));
    CC_RK(get((void **)&long_rows, 4ull * (G.m / kLongRow + 1)));
    CC_RK(get((void **)&ctl, 4ull * kBfsCtl));
    uint32_t *d_cc = nullptr;
    CC_RK(device_alloc((void **)&d_cc, 4ull * n));  // owned by the graph
    G.d_cc = d_cc;

    cc_init_kernel<<<1184, 256, 0, st>>>(G.d_out_off, G.d_out_adj, parent, n);
    cc_flatten_kernel<<<1184, 256, 0, st>>>(parent, n);
    // A 32nd of the entries first: with all of them at once, hundreds of thousands
    // of lanes would find the same few roots apart and fight over the links
    // (the lattice of 490,000 nodes: 338 us in one go, 43 + 9 + 58 this way).
    const uint32_t m = (uint32_t)G.m;
    if (m / 32) {
        cc_union_kernel<<<1184, 256, 0, st>>>(G.d_out_off, G.d_out_adj, n, m / 32, parent);
        cc_flatten_kernel<<<1184, 256, 0, st>>>(parent, n);
    }
    if (m) cc_union_kernel<<<1184, 256, 0, st>>>(G.d_out_off, G.d_out_adj, n, m, parent);
    cc_compress_kernel<<<592, 256, 0, st>>>(parent, n, root, is_root);
    CC_CK(cudaGetLastError());
    size_t tb = 0;
    CC_CK(cub::DeviceScan::ExclusiveSum(nullptr, tb, is_root, rank, n, st));
    void *tmp = nullptr;
    CC_RK(get(&tmp, tb));
    CC_CK(cub::DeviceScan::ExclusiveSum(tmp, tb, is_root, rank, n, st));
    uint32_t last_rank = 0, last_root = 0;
    CC_CK(cudaMemcpyAsync(&last_rank, rank + n - 1, 4, cudaMemcpyDeviceToHost, st));
    CC_CK(cudaMemcpyAsync(&last_root, is_root + n - 1, 4, cudaMemcpyDeviceToHost, st));
    CC_CK(cudaStreamSynchronize(st));
    const uint32_t ncomp = last_rank + last_root;
    CC_RK(get((void **)&pivot_key, 8ull * ncomp));
    CC_CK(cudaMemsetAsync(pivot_key, 0, 8ull * ncomp, st));
    CC_CK(cudaMemsetAsync(seen, 0, 4ull * n, st));
    cc_number_kernel<<<592, 256, 0, st>>>(root, rank, G.d_out_off, n, d_cc, pivot_key);
    bfs_seed_kernel<<<64, 256, 0, st>>>(pivot_key, ncomp, seen, queue);
    CC_CK(cudaGetLastError());
    CC_CK(launch_bfs(BfsArgs{G.d_out_off, G.d_out_adj, nullptr, queue, seen, long_rows, ctl,
                             nullptr, ncomp},
                     st));
    uint32_t bfs[kBfsCtl];
    CC_CK(cudaMemcpyAsync(bfs, ctl, sizeof(bfs), cudaMemcpyDeviceToHost, st));
    CC_CK(cudaStreamSynchronize(st));
    if (bfs[9]) {
        set_error("the breadth-first searches of the diameter bound did not end");
        return SILVAN_E_TIMEOUT;
    }
    // max over components of 2 ecc(pivot): the searches run side by side, so the
    // deepest level is the largest eccentricity
    const unsigned int diam = 2u * bfs[8];
    G.ncomp = ncomp;
    G.diameter = diam;
    return SILVAN_OK;
}

}  // namespace silvan
