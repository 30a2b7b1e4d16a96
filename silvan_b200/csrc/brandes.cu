// Exact betweenness on the device (Brandes, "A faster algorithm for
// betweenness centrality", J. Math. Sociol. 2001), normalised the way SILVAN
// estimates it: the sum over ordered pairs (s, t), s != t, of
// sigma_st(v) / sigma_st, divided by n (n - 1).  It is the ground truth for
// checking the (eps, delta) guarantee on graphs too large for the CPU
// restatement; the reference has no exact algorithm of its own.
//
// One CTA per source at a time (persistent; slot b takes the sources b,
// b + slots, ..., so that the result does not depend on scheduling).
// Forward: level-synchronous BFS.  A node is claimed by atomicOr on a bitmap;
// its path count is the sum over its neighbours on the level before, pulled
// while its own row is scanned for the next level (undirected graphs; directed
// ones pull it from the reverse row).  Backward: with
// g(w) = (1 + delta(w)) / sigma(w), delta(v) = sigma(v) x the sum of g over v's
// successors on the next level; g(v) then takes sigma(v)'s place.  Every sum
// runs in the row's order over fixed lanes, so the value does not depend on
// scheduling, except that rows which do not match (kForward) add their path
// counts in the order of arrival: exact up to 2^53, rounded beyond.  A count
// beyond the doubles' range is infinite: the pairs that end in such a node add
// nothing, and a node with one whose successors have one too gets NaN.
//
// What bounds it: two scans of all rows per source, each entry a probe of the
// neighbour's level.  Up to 19,164 nodes, the levels, the queue, the path
// counts and (up to 11,546 nodes) the running sums lie in shared memory, so
// only the rows come from L2; larger graphs keep them per slot in global
// memory.  A row is scanned by as many lanes as the mean degree asks for, a
// long one by its whole warp.  Barabasi-Albert graph of 10,000 nodes, 5 edges
// per new node, one B200: 14.1 ms (with all of it in global memory and one thread a
// node in the backward pass: 50.5 ms); issue slots 55 % busy.
#include "brandes.h"

#include <algorithm>
#include <cfloat>
#include <vector>

namespace silvan {

namespace {

#define BK(x)                                                                       \
    do {                                                                            \
        cudaError_t e_ = (x);                                                       \
        if (e_ != cudaSuccess) return cuda_status(e_, "exact betweenness");         \
    } while (0)
#define BR(x)                                                                       \
    do {                                                                            \
        int r_ = (x);                                                               \
        if (r_ != SILVAN_OK) return r_;                                             \
    } while (0)

struct BrandesArgs {
    const uint32_t *out_off, *out_adj, *in_off, *in_adj;  // in_* alias out_* when undirected
    uint32_t n;
    uint32_t group_log;  // log2 of the lanes that scan a row
    uint32_t *levels;    // slot-major, n + 2 per slot: queue index where each level starts
    double *partial;     // slot-major, n per slot
    // graphs beyond shared memory, slot-major
    uint32_t *dist;      // kUnseen between sources
    uint32_t *queue;
    double *val;
    uint32_t *seen;      // bitmap, zero between sources
};

// Bytes of shared memory per node: path count, level, queue entry and bitmap
// bit; with the running sums.
constexpr size_t near_bytes(uint32_t n, bool sums) {
    return (size_t)n * (sums ? 20 : 12) + 4 * (((size_t)n + 31) / 32) + 16;
}
constexpr size_t kSharedMax = 227 * 1024 - 64;  // less the static part

// How a node's path count is found: from its own row (undirected), from its
// reverse row (directed), or, for uploaded rows whose two directions do not
// match, added by the nodes before it as their forward rows are scanned (sums
// of integers: exact in any order).
constexpr int kSymmetric = 0, kDirected = 1, kForward = 2;

// Where a source's state lies.
template <bool kNear>
struct State {
    typedef uint16_t Id;
    static constexpr uint32_t kUnseen = 0xffffu;
};
template <>
struct State<false> {
    typedef uint32_t Id;
    static constexpr uint32_t kUnseen = 0xffffffffu;
};

// Sums f(entry) over the rows (off, adj) of the queue's nodes [lo, hi) and
// hands each node and its sum to done.  f(ok, x, v) is called by whole warps (ok:
// the lane has an entry x, of the row of v).
template <typename Id, typename F, typename D>
__device__ __forceinline__ void scan_rows(const uint32_t *off, const uint32_t *adj,
                                          const Id *queue, uint32_t lo, uint32_t hi,
                                          uint32_t group_log, F f, D done) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const uint32_t G = 1u << group_log, gl = lane & (G - 1u), gi = lane >> group_log;
    const uint32_t per = 32u >> group_log;
    for (uint32_t i0 = lo + warp * per; i0 < hi; i0 += nwarps * per) {
        const bool has = i0 + gi < hi;
        uint32_t v = 0, b = 0, e = 0;
        if (has) {
            v = queue[i0 + gi];
            b = __ldg(&off[v]);
            e = __ldg(&off[v + 1]);
        }
        // rows of more than eight steps are left to the whole warp
        const bool far = e - b > 8u * G;
        uint32_t far_rows = __ballot_sync(0xffffffffu, far && gl == 0u);
        const uint32_t steps =
            __reduce_max_sync(0xffffffffu, far ? 0u : (e - b + G - 1u) >> group_log);
        // the next entry is loaded while the current one is looked at
        double acc = 0.0;
        const uint32_t end = far ? b : e;
        uint32_t k = b + gl;
        uint32_t x = k < end ? __ldg(&adj[k]) : 0u;
        for (uint32_t t = 0; t < steps; t++) {
            const bool ok = k < end;
            const uint32_t cur = x;
            k += G;
            if (k < end) x = __ldg(&adj[k]);
            acc += f(ok, cur, v);
        }
        for (uint32_t o = G >> 1; o > 0u; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        while (far_rows) {
            const int src = __ffs(far_rows) - 1;
            far_rows &= far_rows - 1u;
            const uint32_t rb = __shfl_sync(0xffffffffu, b, src);
            const uint32_t re = __shfl_sync(0xffffffffu, e, src);
            const uint32_t rv = __shfl_sync(0xffffffffu, v, src);
            double a = 0.0;
            for (uint32_t k0 = rb; k0 < re; k0 += 32u) {
                const bool ok = k0 + lane < re;
                a += f(ok, ok ? __ldg(&adj[k0 + lane]) : 0u, rv);
            }
            for (uint32_t o = 16; o > 0u; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
            if ((int)lane == src) acc = a;
        }
        if (has && gl == 0u) done(v, acc);
        __syncwarp();
    }
}

template <int BLOCK, bool kNear, bool kSums, int kMode>
__global__ void __launch_bounds__(BLOCK, 1024 / BLOCK) brandes_kernel(BrandesArgs A) {
    typedef typename State<kNear>::Id Id;
    constexpr uint32_t kUnseen = State<kNear>::kUnseen;
    extern __shared__ __align__(16) unsigned char brandes_smem[];
    __shared__ uint32_t s_tail;
    const uint32_t n = A.n, lane = threadIdx.x & 31;
    const uint64_t slot = (uint64_t)blockIdx.x * n;
    const uint32_t words = (n + 31u) / 32u;
    double *part = A.partial + slot;
    uint32_t *lvl = A.levels + (uint64_t)blockIdx.x * (n + 2);
    double *val, *sum = part;
    Id *dist, *queue;
    uint32_t *seen;
    if constexpr (kNear) {
        val = reinterpret_cast<double *>(brandes_smem);
        unsigned char *p = brandes_smem + 8 * (size_t)n;
        if constexpr (kSums) {
            sum = reinterpret_cast<double *>(p);
            p += 8 * (size_t)n;
        }
        seen = reinterpret_cast<uint32_t *>(p);
        dist = reinterpret_cast<Id *>(p + 4 * (size_t)words);
        queue = dist + n;
        if constexpr (kSums)
            for (uint32_t i = threadIdx.x; i < n; i += BLOCK) sum[i] = 0.0;
    } else {
        val = A.val + slot;
        dist = A.dist + slot;
        queue = A.queue + slot;
        seen = A.seen + (uint64_t)blockIdx.x * words;
    }
    for (uint32_t s = blockIdx.x; s < n; s += gridDim.x) {
        if constexpr (kNear) {
            for (uint32_t i = threadIdx.x; i < n; i += BLOCK) {
                dist[i] = (Id)kUnseen;
                if constexpr (kMode == kForward) val[i] = 0.0;
            }
            for (uint32_t i = threadIdx.x; i < words; i += BLOCK) seen[i] = 0u;
            __syncthreads();
        }
        if (threadIdx.x == 0) {
            dist[s] = 0;
            seen[s >> 5] = 1u << (s & 31);
            val[s] = 1.0;
            queue[0] = (Id)s;
            s_tail = 1;
            lvl[0] = 0;
            lvl[1] = 1;
        }
        __syncthreads();
        // forward, one level at a time (a level is a queue segment)
        uint32_t lev = 0, lo = 0, hi = 1;
        for (;; lev++) {
            const auto visit = [&](bool ok, uint32_t x, uint32_t v) -> double {
                const uint32_t d = ok ? (uint32_t)dist[x] : 0u;
                bool first = false;
                if (ok && d == kUnseen) {
                    const uint32_t bit = 1u << (x & 31);
                    first = (atomicOr(&seen[x >> 5], bit) & bit) == 0u;
                    if (first) dist[x] = (Id)(lev + 1u);
                }
                const uint32_t m = __ballot_sync(0xffffffffu, first);
                if (m) {
                    uint32_t at = 0;
                    if (lane == 0) at = atomicAdd(&s_tail, (uint32_t)__popc(m));
                    at = __shfl_sync(0xffffffffu, at, 0);
                    if (first) queue[at + __popc(m & ((1u << lane) - 1u))] = (Id)x;
                }
                if constexpr (kMode == kForward) {
                    if (ok && (d == kUnseen || d == lev + 1u)) atomicAdd(&val[x], val[v]);
                }
                return kMode == kSymmetric && ok && lev > 0u && d == lev - 1u ? val[x] : 0.0;
            };
            scan_rows(A.out_off, A.out_adj, queue, lo, hi, A.group_log, visit,
                      [&](uint32_t v, double a) {
                          if (lev > 0u && kMode == kSymmetric) val[v] = a;
                      });
            __syncthreads();
            lo = hi;
            hi = s_tail;
            if (threadIdx.x == 0) lvl[lev + 2u] = hi;
            if (lo == hi) break;
            if constexpr (kMode == kDirected) {
                scan_rows(A.in_off, A.in_adj, queue, lo, hi, A.group_log,
                          [&](bool ok, uint32_t x, uint32_t) {
                              return ok && (uint32_t)dist[x] == lev ? val[x] : 0.0;
                          },
                          [&](uint32_t v, double a) { val[v] = a; });
            }
            __syncthreads();
        }
        __syncthreads();
        // backward: the levels lev, lev - 1, ..., 0
        for (int32_t l = (int32_t)lev; l >= 0; l--) {
            const uint32_t b = __ldcg(&lvl[l]), e = __ldcg(&lvl[l + 1]);
            scan_rows(A.out_off, A.out_adj, queue, b, e, A.group_log,
                      [&](bool ok, uint32_t x, uint32_t) {
                          return ok && (uint32_t)dist[x] == (uint32_t)l + 1u ? val[x] : 0.0;
                      },
                      [&](uint32_t v, double a) {
                          const double sg = val[v];
                          double delta = sg * a;
                          if (sg > DBL_MAX) {  // infinity times nothing is nothing
                              const uint32_t e = A.out_off[v + 1];
                              uint32_t k = A.out_off[v];
                              while (k < e && (uint32_t)dist[A.out_adj[k]] != (uint32_t)l + 1u) k++;
                              if (k == e) delta = 0.0;
                          }
                          if (v != s) sum[v] += delta;
                          val[v] = (1.0 + delta) / sg;
                      });
            __syncthreads();
        }
        if constexpr (!kNear) {  // restore the visited nodes
            const uint32_t tail = s_tail;
            for (uint32_t i = threadIdx.x; i < tail; i += BLOCK) {
                const uint32_t v = queue[i];
                dist[v] = kUnseen;
                seen[v >> 5] = 0u;
                if constexpr (kMode == kForward) val[v] = 0.0;
            }
            __syncthreads();
        }
    }
    if constexpr (kNear && kSums)
        for (uint32_t i = threadIdx.x; i < n; i += BLOCK) part[i] = sum[i];
}

__global__ void brandes_init_kernel(uint32_t *dist, double *val, double *partial, uint64_t total,
                                    uint32_t *seen, uint64_t words) {
    const uint64_t t0 = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = t0; i < total; i += nth) {
        if (dist) {
            dist[i] = 0xffffffffu;
            val[i] = 0.0;
        }
        partial[i] = 0.0;
    }
    if (seen)
        for (uint64_t i = t0; i < words; i += nth) seen[i] = 0u;
}

__global__ void brandes_sum_kernel(const double *partial, uint32_t n, uint32_t slots,
                                   double norm, double *out) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        double acc = 0.0;
#pragma unroll 8
        for (uint32_t s = 0; s < slots; s++) acc += partial[(uint64_t)s * n + v];
        out[v] = acc / norm;
    }
}

struct BrandesKernel {
    const void *fn = nullptr;
    int block = 0;
    size_t smem = 0;
    bool near = false;
};

// The kernel for a graph of n nodes.  One CTA per SM takes 1024 threads, up
// to three 512 each, more 256: about as many threads as an SM's registers
// hold at 64 each.
template <int kMode>
BrandesKernel pick_kernel(uint32_t n) {
    const bool sums = near_bytes(n, true) <= kSharedMax;
    if (!sums && near_bytes(n, false) > kSharedMax)
        return {(const void *)brandes_kernel<512, false, false, kMode>, 512, 0, false};
    const size_t smem = near_bytes(n, sums);
    const size_t ctas = kSharedMax / (smem + 1024);
    if (!sums) return {(const void *)brandes_kernel<1024, true, false, kMode>, 1024, smem, true};
    if (ctas <= 1) return {(const void *)brandes_kernel<1024, true, true, kMode>, 1024, smem, true};
    if (ctas <= 3) return {(const void *)brandes_kernel<512, true, true, kMode>, 512, smem, true};
    return {(const void *)brandes_kernel<256, true, true, kMode>, 256, smem, true};
}

}  // namespace

int exact_betweenness(const DeviceGraph &G, double *out_host) {
    const uint32_t n = G.n;
    int dev = 0, sms = 0, per_sm = 0;
    BK(cudaGetDevice(&dev));
    BK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const BrandesKernel K = !G.rows_match  ? pick_kernel<kForward>(n)
                            : G.directed ? pick_kernel<kDirected>(n)
                                         : pick_kernel<kSymmetric>(n);
    if (K.smem)
        BK(cudaFuncSetAttribute(K.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)K.smem));
    BK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, K.fn, K.block, K.smem));
    // slots: the resident CTAs, bounded by a quarter of the free memory
    size_t fr = 0, tot = 0;
    BK(cudaMemGetInfo(&fr, &tot));
    const uint64_t words = ((uint64_t)n + 31) / 32;
    const uint64_t per_slot = (uint64_t)n * (4 + 8) + 8 + (K.near ? 0 : (uint64_t)n * 16 + 4 * words);
    uint64_t slots = std::min<uint64_t>((uint64_t)sms * std::max(per_sm, 1),
                                        std::max<uint64_t>(1, fr / 4 / per_slot));
    slots = std::min<uint64_t>(slots, n);
    BrandesArgs A{};
    A.out_off = G.d_out_off;
    A.out_adj = G.d_out_adj;
    A.in_off = G.d_in_off;
    A.in_adj = G.d_in_adj;
    A.n = n;
    // about the mean degree in lanes per row, at least four
    const uint64_t degree = G.m / n;
    A.group_log = degree <= 5 ? 2 : degree <= 12 ? 3 : degree <= 24 ? 4 : 5;
    void *p = nullptr;
    struct Bufs {
        std::vector<void *> v;
        ~Bufs() {
            for (void *b : v) device_free(b);
        }
    } bufs;
    auto get = [&](void **q, size_t bytes) -> int {
        int rc = device_alloc(q, bytes);
        if (rc == SILVAN_OK) bufs.v.push_back(*q);
        return rc;
    };
    const uint64_t tot_nodes = slots * n;
    BR(get(&p, 4 * slots * ((uint64_t)n + 2)));
    A.levels = (uint32_t *)p;
    BR(get(&p, 8 * tot_nodes));
    A.partial = (double *)p;
    if (!K.near) {
        BR(get(&p, 4 * tot_nodes));
        A.dist = (uint32_t *)p;
        BR(get(&p, 4 * tot_nodes));
        A.queue = (uint32_t *)p;
        BR(get(&p, 8 * tot_nodes));
        A.val = (double *)p;
        BR(get(&p, 4 * slots * words));
        A.seen = (uint32_t *)p;
    }
    double *d_out = nullptr;
    BR(get(&p, 8 * (uint64_t)n));
    d_out = (double *)p;
    brandes_init_kernel<<<1184, 256>>>(A.dist, A.val, A.partial, tot_nodes, A.seen, slots * words);
    BK(cudaGetLastError());
    void *args[] = {&A};
    BK(cudaLaunchKernel(K.fn, dim3((uint32_t)slots), dim3(K.block), args, K.smem, 0));
    brandes_sum_kernel<<<(n + 63) / 64, 64>>>(A.partial, n, (uint32_t)slots,
                                              (double)n * (double)(n - 1), d_out);
    BK(cudaGetLastError());
    BK(cudaMemcpy(out_host, d_out, sizeof(double) * n, cudaMemcpyDeviceToHost));
    return SILVAN_OK;
}

}  // namespace silvan
