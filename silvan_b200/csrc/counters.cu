// Ordered commit of sample contributions (see counters.cuh).
//
// The reference adds every sample's path map to the per-node counters inside
// one critical section, in sample order (silvan/src/Probabilistic.cpp:479-544):
//   x = count * (1 / num_paths)
//   approx[u] += x;  emp_wimpy_vars[u] += x * x;
//   mcrade[u][j] = (int64)((double)mcrade[u][j] + sign_j * x)   (truncation)
// With num_paths > 1 the additions are not associative, so a node's updates
// must be applied in sample order.  A draw's records are grouped by node once
// (count, bucket space, scatter) and each node's group put in sample order (by
// rank: compares for groups of <= 32, a bitmap of the draw's samples
// otherwise).  A commit round then folds each group's entries of its sample
// range sequentially, one warp a node: lanes 0..24 each carry one Monte Carlo
// trial, lane 25 approx, lane 26 the wimpy variance.  Different nodes are
// independent, so the only serial work is per node.
#include <algorithm>
#include <cstddef>
#include <cfloat>
#include <climits>
#include <cstring>
#include <vector>

#include "counters.cuh"
#include "grid_barrier.cuh"

namespace silvan {

namespace {

// ---------------------------------------------------------------------------
// A draw's records by node as a single cooperative kernel.  Its phases are
// separated by grid-wide barriers (every CTA is resident: cooperative launch):
//   A  per sample the Rademacher signs and 1 / num_paths; records counted per
//      node and the touched nodes listed
//   B  bucket space of every touched node taken from a cursor (warp
//      aggregated), the scatter cursors, the list of buckets of more than
//      32 entries
//   C  records scattered into their nodes' buckets
//   D  each bucket put in sample order, its entries with their factor and
//      signs: the huge buckets by whole CTAs (claimed from a cursor), then the
//      others one warp each (fixed assignment); cursors zeroed
// Each barrier is bounded: a CTA that waits longer than ApplyArgs::polls polls
// records SILVAN_E_TIMEOUT in the job's error word and leaves the kernel.  Such a
// draw is published with no touched node, so that the commit rounds queued behind
// it read none of the buckets, and a later draw of the job (its error is only
// seen at the next check) ends at once: the counts it would start from are not
// zero.
//
// Once per draw, not per commit round: an estimation commits a draw in about
// ten rounds, and the three barriers and their phases were more than half of
// each (R-MAT 20, a million nodes: 14 of 31-35 us; a round is now 20 and the draw 66 once).
// ---------------------------------------------------------------------------
constexpr int kCommitThreads = 1024;

__device__ __forceinline__ uint32_t round_records(const RoundBuffers &rb, const ApplyArgs &a) {
    return (uint32_t)min((uint64_t)a.n_records, rb.rec_cap);
}

__device__ void bucket_count(const RoundBuffers &rb, const ApplyArgs &a) {
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
    const uint32_t lane = threadIdx.x & 31;
    // per sample, one warp: the Rademacher signs (read in pass 2; lane j draws
    // trial j, as rademacher_mask does) and 1 / num_paths, the factor every
    // record of the sample is multiplied by (Probabilistic.cpp:502)
    for (uint32_t s = tid >> 5; s < a.count; s += nth >> 5) {
        bool plus = false;
        if (lane < (uint32_t)kTrials)
            plus = philox_lo32(a.seed, a.first_sample + s, kStreamRademacher, lane) %
                       100000000u >= 50000000u;
        const uint32_t m = __ballot_sync(0xffffffffu, plus);
        if (lane == 0) rb.signs[s] = m;
        if (lane == 31) rb.inv_np[s] = __ddiv_rn(1.0, (double)rb.np[s]);
    }
    const uint32_t R = round_records(rb, a);
    // warp-uniform loop: the first record of a node is appended to the
    // touched list with one counter increment per warp (a single counter
    // that every warp hits would serialise the whole phase)
    for (uint32_t i0 = tid - lane; i0 < R; i0 += nth) {
        const uint32_t i = i0 + lane;
        bool first = false;
        uint32_t node = 0;
        if (i < R) {
            const PathRec r = rb.recs[i];
            node = r.node;
            first = atomicAdd(&rb.node_cnt[r.node], 1u) == 0u;
        }
        const uint32_t m = __ballot_sync(0xffffffffu, first);
        if (m) {
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(rb.n_touched, (uint32_t)__popc(m));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (first) rb.touched[base + __popc(m & ((1u << lane) - 1u))] = node;
        }
    }
}

// Bucket space of every touched node, taken from a cursor (the buckets need
// no order among themselves): one atomic per warp for the warp's nodes, the
// lanes' offsets by a warp scan.  The node's count becomes its scatter
// cursor; buckets of more than 32 entries are listed for fold_large, of more than
// kHugeBucket for order_huge.
__device__ void bucket_alloc(const RoundBuffers &rb, uint32_t T) {
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t t0 = tid - lane; t0 < T; t0 += nth) {
        const uint32_t t = t0 + lane;
        uint32_t node = 0, b = 0;
        if (t < T) {
            node = rb.touched[t];
            b = rb.node_cnt[node];
        }
        uint32_t incl = b;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        uint32_t base = 0;
        if (lane == 31 && incl) base = atomicAdd(rb.n_touched + 4, incl);
        base = __shfl_sync(0xffffffffu, base, 31);
        const bool large = b > 32;
        const uint32_t lm = __ballot_sync(0xffffffffu, large);
        uint32_t lbase = 0;
        if (lm && lane == 0) lbase = atomicAdd(rb.n_large, (uint32_t)__popc(lm));
        lbase = __shfl_sync(0xffffffffu, lbase, 0);
        if (t < T) {
            const uint32_t off = base + incl - b;
            rb.bucket_off[t] = off;
            rb.bucket_len[t] = b;
            rb.node_cnt[node] = off;  // becomes the scatter cursor
            if (large) rb.large[lbase + __popc(lm & ((1u << lane) - 1u))] = t;
            if (b > kHugeBucket) rb.huge[atomicAdd(rb.n_touched + 7, 1u)] = t;
        }
    }
}

__device__ void bucket_scatter(const RoundBuffers &rb, const ApplyArgs &a) {
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
    const uint32_t R = round_records(rb, a);
    for (uint32_t i = tid; i < R; i += nth) {
        PathRec r = rb.recs[i];
        uint32_t pos = atomicAdd(&rb.node_cnt[r.node], 1u);
        rb.entries[pos] = ((unsigned long long)r.sample << 32) | r.count;
    }
}

// An entry of a bucket as the rounds read it.  inv_np and signs were written by
// other CTAs before the last grid barrier.
__device__ __forceinline__ DrawEntry draw_entry(const RoundBuffers &rb, unsigned long long e) {
    const uint32_t sl = (uint32_t)(e >> 32);
    DrawEntry d;
    d.x = __dmul_rn((double)(uint32_t)e, __ldcg(&rb.inv_np[sl]));
    d.signs = __ldcg(&rb.signs[sl]);
    d.sample = sl;
    return d;
}

// In sample order at `pos`: x where the records were (read for the last time
// before the barrier), sample and signs in the place of an entry (of the same
// bucket, whose entries the caller has read).  20 bytes a record in all.
__device__ __forceinline__ void entry_store(const RoundBuffers &rb, uint32_t pos,
                                            const DrawEntry &d) {
    rb.x[pos] = d.x;
    rb.entries[pos] = (unsigned long long)d.sample << 32 | d.signs;
}

// Shared memory of phase D: the samples of the CTA's huge bucket and the set
// bits before each word; then each warp's bucket.
struct OrderSmem {
    union {
        struct {
            uint32_t bits[kDrawSamples / 32];
            uint32_t wpre[kDrawSamples / 32];
        } h;
        uint32_t sample[kCommitThreads / 32][kHugeBucket];
    };
    uint32_t scan[33];
    uint32_t li;
};
static_assert(sizeof(OrderSmem) <= 48 * 1024, "static shared memory");

// Buckets of more than kHugeBucket entries, by whole CTAs.  The entries of a
// bucket are distinct samples of the draw (a node is on a sample's path map
// once), so their order is the rank of each sample in a bitmap of the draw:
// set one bit per entry, prefix-count the bits per word, and each entry goes
// to its rank (linear in the bucket; no comparison sort).  (One warp a bucket
// took 400 us for a hub's 60,000 entries.)
__device__ void order_huge(const RoundBuffers &rb, const JobCounters &jc, uint32_t S,
                           OrderSmem &sm) {
    constexpr uint32_t kWords = kDrawSamples / 32, kPer = kWords / kCommitThreads;
    const uint32_t lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const uint32_t NH = __ldcg(rb.n_touched + 7);
    for (;;) {
        if (threadIdx.x == 0) sm.li = atomicAdd(rb.n_touched + 5, 1u);
        for (uint32_t w = threadIdx.x; w < kWords; w += kCommitThreads) sm.h.bits[w] = 0u;
        __syncthreads();
        const uint32_t li = sm.li;
        if (li >= NH) break;
        const uint32_t t = __ldcg(&rb.huge[li]);
        const uint32_t b0 = __ldcg(&rb.bucket_off[t]), b = __ldcg(&rb.bucket_len[t]);
        if (b > S) {  // more entries than samples: not a bucket of distinct samples
            if (threadIdx.x == 0) {
                atomicCAS(&jc.sc->error, 0, SILVAN_E_STATE);
                rb.bucket_span[t] = make_ushort2(0, 0);
            }
            __syncthreads();
            continue;
        }
        for (uint32_t i = threadIdx.x; i < b; i += kCommitThreads) {
            const uint32_t sidx = (uint32_t)(__ldcg(&rb.entries[b0 + i]) >> 32);
            if (sidx < S) atomicOr(&sm.h.bits[sidx >> 5], 1u << (sidx & 31));
            else atomicCAS(&jc.sc->error, 0, SILVAN_E_STATE);
        }
        __syncwarp();
        __syncthreads();
        // exclusive prefix of the words' bit counts (thread L owns words
        // [L kPer, (L + 1) kPer))
        uint32_t c = 0;
#pragma unroll
        for (uint32_t w = 0; w < kPer; w++) c += __popc(sm.h.bits[threadIdx.x * kPer + w]);
        uint32_t incl = c;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
            if ((int)lane >= o) incl += u;
        }
        if (lane == 31) sm.scan[wib] = incl;
        __syncthreads();
        uint32_t ws = sm.scan[lane];
        const uint32_t own = ws;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, ws, o);
            if ((int)lane >= o) ws += u;
        }
        uint32_t run = __shfl_sync(0xffffffffu, ws - own, (int)wib) + incl - c;
#pragma unroll
        for (uint32_t w = 0; w < kPer; w++) {
            sm.h.wpre[threadIdx.x * kPer + w] = run;
            run += __popc(sm.h.bits[threadIdx.x * kPer + w]);
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < b; i += kCommitThreads) {
            const unsigned long long e = __ldcg(&rb.entries[b0 + i]);
            const uint32_t sidx = (uint32_t)(e >> 32);
            if (sidx >= S) continue;
            const uint32_t w = sidx >> 5;
            const uint32_t r = sm.h.wpre[w] + __popc(sm.h.bits[w] & ((1u << (sidx & 31)) - 1u));
            rb.x[b0 + r] = draw_entry(rb, e).x;
            rb.order[b0 + r] = sidx;
            uint16_t *span = reinterpret_cast<uint16_t *>(&rb.bucket_span[t]);
            if (r == 0u) span[0] = (uint16_t)sidx;
            if (r == b - 1u) span[1] = (uint16_t)sidx;
        }
        __syncwarp();
        __syncthreads();
        // all entries are read: samples and signs take their places
        for (uint32_t i = threadIdx.x; i < b; i += kCommitThreads) {
            const uint32_t sidx = __ldcg(&rb.order[b0 + i]);
            if (sidx < S)
                rb.entries[b0 + i] = (unsigned long long)sidx << 32 | __ldcg(&rb.signs[sidx]);
        }
    }
    __syncthreads();
}

// The other buckets, touched node t on warp t mod (warps of the grid), no
// cursor.  A bucket holds distinct samples, so each entry's position in sample
// order is the number of entries with a smaller sample: compares across the
// warp up to 32 entries, over a copy in shared memory up to kHugeBucket.
__device__ void order_others(const RoundBuffers &rb, uint32_t T, OrderSmem &sm) {
    constexpr uint32_t kKeys = kHugeBucket / 32;
    const uint32_t lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const uint32_t stride = gridDim.x * (kCommitThreads / 32);
    uint32_t *mine = sm.sample[wib];
    for (uint32_t t = blockIdx.x * (kCommitThreads / 32) + wib; t < T; t += stride) {
        const uint32_t b = __ldcg(&rb.bucket_len[t]);
        if (b > kHugeBucket) continue;
        const uint32_t off = __ldcg(&rb.bucket_off[t]);
        uint16_t *span = reinterpret_cast<uint16_t *>(&rb.bucket_span[t]);
        if (b <= 32u) {
            const unsigned long long key = lane < b ? __ldcg(&rb.entries[off + lane]) : ~0ull;
            uint32_t rank = 0;
            for (uint32_t j = 0; j < b; j++)
                rank += __shfl_sync(0xffffffffu, key, (int)j) < key;
            if (lane < b) {
                entry_store(rb, off + rank, draw_entry(rb, key));
                if (rank == 0u) span[0] = (uint16_t)(key >> 32);
                if (rank == b - 1u) span[1] = (uint16_t)(key >> 32);
            }
        } else {
            unsigned long long key[kKeys];
            uint32_t rank[kKeys];
#pragma unroll
            for (uint32_t r = 0; r < kKeys; r++) {
                const uint32_t i = r * 32u + lane;
                key[r] = i < b ? __ldcg(&rb.entries[off + i]) : ~0ull;
                mine[i] = (uint32_t)(key[r] >> 32);
                rank[r] = 0u;
            }
            __syncwarp();
            for (uint32_t j = 0; j < b; j++) {
                const uint32_t o = mine[j];
#pragma unroll
                for (uint32_t r = 0; r < kKeys; r++) rank[r] += o < (uint32_t)(key[r] >> 32);
            }
#pragma unroll
            for (uint32_t r = 0; r < kKeys; r++) {
                if (r * 32u + lane >= b) continue;
                entry_store(rb, off + rank[r], draw_entry(rb, key[r]));
                if (rank[r] == 0u) span[0] = (uint16_t)(key[r] >> 32);
                if (rank[r] == b - 1u) span[1] = (uint16_t)(key[r] >> 32);
            }
        }
        __syncwarp();
    }
}

// The last CTA out keeps the draw's counts (zeros when a CTA did not reach the
// end) and zeroes the control words.
__device__ void prepare_exit(const RoundBuffers &rb, bool complete) {
    __syncthreads();
    if (threadIdx.x == 0) {
        if (!complete) atomicExch(rb.n_touched + 10, 1u);
        __threadfence();
        if (atomicAdd(rb.n_touched + 6, 1u) == gridDim.x - 1) {
            const bool all = __ldcg(&rb.n_touched[10]) == 0u;
            rb.n_touched[8] = all ? __ldcg(&rb.n_touched[0]) : 0u;
            rb.n_touched[9] = all ? __ldcg(&rb.n_touched[1]) : 0u;
            rb.n_touched[10] = 0u;
            rb.n_touched[0] = 0u;
            rb.n_touched[1] = 0u;
            rb.n_touched[2] = 0u;  // arrivals at a barrier that was given up
            rb.n_touched[4] = 0u;
            rb.n_touched[5] = 0u;
            rb.n_touched[6] = 0u;
            rb.n_touched[7] = 0u;
            __threadfence();
        }
    }
}

// ---------------------------------------------------------------------------
// A commit round.  The kernel that groups a draw commits a small one's first
// part itself, after one more barrier: the plain form draws eleven samples at a
// time and commits them at once, and with a second kernel for that, both of all
// SMs, 10,000 nodes of Barabasi-Albert took 52 ms instead of 47.
// ---------------------------------------------------------------------------

// Sequential fold of one node's contributions in sample order.  Every lane
// runs the same instruction stream and carries one chain: lane j < 25 trial j
// of mcrade, lane 25 approx (and the top-k crossing), lane 26 the wimpy
// variance; lanes 27..31 repeat lane 25's chain and store nothing.  The entries
// are staged 32 at a time in the warp's scratch: x = count * (1 / num_paths),
// the sample's signs and its round-local index.  A hub's chain bounds a round:
// the sums advance one dependent addition (8 cycles) per entry; the trials,
// whose chain (add, truncate) takes 24, advance four entries a step where 32
// are there (fold_full): R-MAT 14, 60,000 entries of one node: 740 -> 540 us.
struct alignas(16) FoldScratch {
    double x[32];
    uint32_t signs[32];
    uint32_t sample[32];
    uint32_t upd[32];  // nodes updated for the first time, not yet on upd_list
    uint32_t nupd;
    double sup_a, sup_w;  // the warp's maxima of approx and emp_wimpy_vars
};

// Per-warp folding state: reset before a warp's first fold, flushed after its
// last (fold_flush), so that the job-wide maxima and the update list take one
// global atomic per warp rather than one per node.
__device__ __forceinline__ void fold_begin(FoldScratch &fs) {
    if ((threadIdx.x & 31) == 0) {
        fs.nupd = 0;
        fs.sup_a = 0.0;
        fs.sup_w = 0.0;
    }
    __syncwarp();
}

__device__ __forceinline__ void upd_flush(const JobCounters &jc, FoldScratch &fs) {
    const uint32_t lane = threadIdx.x & 31;
    __syncwarp();
    const uint32_t k = fs.nupd;
    if (k) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(&jc.sc->n_upd, k);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (lane < k) jc.upd_list[base + lane] = fs.upd[lane];
        __syncwarp();
        if (lane == 0) fs.nupd = 0;
    }
    __syncwarp();
}

__device__ __forceinline__ void atomic_max_nonneg_double(unsigned long long *p, double v) {
    atomicMax(p, (unsigned long long)__double_as_longlong(v));
}

__device__ __forceinline__ void fold_flush(const JobCounters &jc, FoldScratch &fs) {
    upd_flush(jc, fs);
    if ((threadIdx.x & 31) == 0) {
        if (fs.sup_a > 0.) atomic_max_nonneg_double(&jc.sc->sup_approx_bits, fs.sup_a);
        if (fs.sup_w > 0.) atomic_max_nonneg_double(&jc.sc->sup_wimpy_bits, fs.sup_w);
    }
    __syncwarp();
}

// A node's counters as its fold starts.
struct NodeState {
    double v;         // this lane's chain
    uint32_t lu0;     // last_upd before the round
    uint32_t lu;      // and after the entries so far (0: no addition)
    bool crossed;     // lane 25: approx reached 3 in an earlier round (top-k pass 1)
};

__device__ __forceinline__ NodeState fold_load(const JobCounters &jc, const ApplyArgs &a,
                                               uint32_t node) {
    const int lane = threadIdx.x & 31;
    NodeState s{0.0, 0u, 0u, true};
    if (lane < kTrials) {
        if (a.pass == 2) s.v = (double)jc.mcrade[(uint64_t)node * kTrials + lane];
    } else if (lane == 26) {
        s.v = jc.wimpy[node];
    } else {
        s.v = jc.approx[node];
        if (lane == 25) {
            s.lu0 = jc.last_upd[node];
            if (a.track_cross) s.crossed = jc.cross_flag[node] != 0;
        }
    }
    return s;
}

// A journaled round saves them at the node's touched position t.
__device__ __forceinline__ void fold_journal(const RoundJournal &jr, const ApplyArgs &a,
                                             uint32_t t, const NodeState &s) {
    const int lane = threadIdx.x & 31;
    if (lane < kTrials) {
        if (a.pass == 2) jr.mcrade[(uint64_t)t * kTrials + lane] = (long long)s.v;
    } else if (lane == 25) {
        jr.approx[t] = s.v;
        jr.last_upd[t] = s.lu0;
    } else if (lane == 26) {
        jr.wimpy[t] = s.v;
    }
}

// One entry of a trial: m + s x for an integer m, truncated towards zero, where
// x is 1 (c) or far enough from 0 and 1 that m + s x is no integer after
// rounding.  With x == 1 the entry moves m by its sign.  With 0 < x < 1, m + x
// is m for m >= 0 and m + 1 for m < 0, and m - x is m for m <= 0 and m - 1 for
// m > 0: a step towards zero or none.
__host__ __device__ constexpr int32_t trial_step(int32_t m, bool plus, bool c) {
    if (plus) return c || m < 0 ? m + 1 : m;
    return c || m > 0 ? m - 1 : m;
}

// Four entries at once: what they add to m depends on their c and plus bits and
// on m only from -4 to 4 (further out no step reaches zero before the last),
// so the additions for these nine m are four bits each of one word.
struct TrialSteps {
    unsigned long long v[256];  // c bits << 4 | plus bits
};
constexpr TrialSteps make_trial_steps() {
    TrialSteps t{};
    for (int i = 0; i < 256; i++) {
        unsigned long long w = 0;
        for (int s = -4; s <= 4; s++) {
            int32_t m = s;
            for (int k = 0; k < 4; k++) m = trial_step(m, (i >> k) & 1, (i >> (4 + k)) & 1);
            w |= (unsigned long long)((m - s) & 15) << (4 * (s + 4));
        }
        t.v[i] = w;
    }
    return t;
}
__device__ const TrialSteps g_trial_steps = make_trial_steps();

// Folds 32 staged entries, each x either 1 (its bit in c) or at least 2^-25 away
// from 0 and 1, with fewer than 2^26 samples so far: m + s x then lies at least
// 2^-26 from an integer, more than it can be rounded by, and trial_step holds.
// All loads come before the two chains, which every lane runs side by side:
// 32 additions of 8 cycles, 8 steps of the trials of about 30.
__device__ __forceinline__ void fold_full(const JobCounters &jc, const ApplyArgs &a,
                                          uint32_t node, uint32_t c, NodeState &st,
                                          const FoldScratch &fs) {
    const int lane = threadIdx.x & 31;
    const bool mc = lane < kTrials, wv = lane == 26;
    st.lu = a.first_sample + fs.sample[31] + 1u;
    int32_t m = 0;
    if (a.pass == 2) {
        unsigned long long w[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint4 g = *reinterpret_cast<const uint4 *>(&fs.signs[4 * i]);
            const uint32_t plus = ((g.x >> lane) & 1u) | ((g.y >> lane) & 1u) << 1 |
                                  ((g.z >> lane) & 1u) << 2 | ((g.w >> lane) & 1u) << 3;
            w[i] = __ldg(&g_trial_steps.v[((c >> (4 * i)) & 15u) << 4 | plus]);
        }
        m = mc ? (int32_t)st.v : 0;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int32_t near = max(-4, min(4, m));
            m += (int32_t)((uint32_t)(w[i] >> (4 * (near + 4))) << 28) >> 28;
        }
    }
    double v = st.v;
#pragma unroll
    for (int k = 0; k < 32; k += 2) {
        const double2 x = *reinterpret_cast<const double2 *>(&fs.x[k]);
        v = __dadd_rn(v, wv ? __dmul_rn(x.x, x.x) : x.x);
        v = __dadd_rn(v, wv ? __dmul_rn(x.y, x.y) : x.y);
    }
    if (lane == 25 && !st.crossed && v >= 3.0) {  // approx reached 3 at entry k
        double t = st.v;
        int k = 0;
        while ((t = __dadd_rn(t, fs.x[k])) < 3.0) k++;
        st.crossed = true;
        jc.cross_flag[node] = 1;
        const uint32_t q = atomicAdd(&jc.sc->n_cross, 1u);
        jc.cross_sample[q] = a.first_sample + fs.sample[k];
    }
    if (!mc)
        st.v = v;
    else if (a.pass == 2)
        st.v = (double)m;
    __syncwarp();
}

// Folds the kmax entries staged in the scratch.
__device__ __forceinline__ void fold_entries(const JobCounters &jc, const ApplyArgs &a,
                                             uint32_t node, uint32_t kmax, NodeState &st,
                                             const FoldScratch &fs) {
    const int lane = threadIdx.x & 31;
    const bool mc = lane < kTrials, wv = lane == 26;
    const bool in = (uint32_t)lane < kmax;
    const uint32_t pm = __ballot_sync(0xffffffffu, in && fs.x[lane] > 0.);
    // 1 + global index of the last sample that adds to approx
    if (pm) st.lu = a.first_sample + fs.sample[31 - __clz(pm)] + 1u;
    int kc = -1;
    double v = st.v;
#pragma unroll 4
    for (uint32_t k = 0; k < kmax; k++) {
        const double x = fs.x[k];
        const bool plus = (fs.signs[k] >> lane) & 1u;
        // mcrade: (int64)((double)m + s x), m kept as an integer-valued
        // double (|m| is at most the sample count, far below 2^53, so the
        // conversions are exact and truncating in double is the same);
        // approx and the wimpy variance add x and x * x when x > 0
        const double add = x > 0. ? (wv ? __dmul_rn(x, x) : x) : 0.0;
        const double y = mc ? (plus ? x : -x) : add;
        const double t = __dadd_rn(v, y);
        if (!st.crossed && kc < 0 && t >= 3.0) kc = (int)k;
        v = mc ? trunc(t) : t;
    }
    st.v = v;
    if (kc >= 0) {  // lane 25 only: approx reached 3 at entry kc
        st.crossed = true;
        jc.cross_flag[node] = 1;
        const uint32_t q = atomicAdd(&jc.sc->n_cross, 1u);
        jc.cross_sample[q] = a.first_sample + fs.sample[kc];
    }
    __syncwarp();
}

__device__ __forceinline__ void fold_store(const JobCounters &jc, const ApplyArgs &a,
                                           uint32_t node, const NodeState &st, FoldScratch &fs) {
    const int lane = threadIdx.x & 31;
    if (lane < kTrials) {
        if (a.pass == 2) jc.mcrade[(uint64_t)node * kTrials + lane] = (long long)st.v;
    } else if (lane == 25) {
        jc.approx[node] = st.v;
        if (st.lu) {
            if (st.lu0 == 0) fs.upd[fs.nupd++] = node;
            jc.last_upd[node] = st.lu;
        }
        fs.sup_a = fmax(fs.sup_a, st.v);
    } else if (lane == 26) {
        jc.wimpy[node] = st.v;
        fs.sup_w = fmax(fs.sup_w, st.v);
    }
    __syncwarp();
    if (fs.nupd == 32) upd_flush(jc, fs);
}

__device__ __forceinline__ void fold_stage(FoldScratch &fs, uint32_t i, const DrawEntry &e) {
    fs.x[i] = e.x;
    fs.signs[i] = e.signs;
    fs.sample[i] = e.sample;
}

__device__ __forceinline__ DrawEntry entry_load(const RoundBuffers &rb, uint32_t pos) {
    const unsigned long long m = __ldcg(&rb.entries[pos]);
    DrawEntry e;
    e.x = __ldcg(&rb.x[pos]);
    e.signs = (uint32_t)m;
    e.sample = (uint32_t)(m >> 32);
    return e;
}

constexpr int kRoundThreads = 512;
constexpr int kRoundCtas = 2;     // per SM
constexpr uint32_t kAhead = 3;    // sets of 32 entries on their way in a large bucket
constexpr uint32_t kBatch = 8;    // small buckets a warp looks at together

// Buckets of more than 32 entries, one warp each: the first entry of the round
// by a 32-way search, then 32 entries at a time, the next sets on their
// way while one is folded.
__device__ void fold_large(const RoundBuffers &rb, const JobCounters &jc, const RoundJournal &jr,
                           const ApplyArgs &a, uint32_t NL, uint32_t w, uint32_t nw,
                           FoldScratch &fs) {
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t li = w; li < NL; li += nw) {
        const uint32_t t = __ldcg(&rb.large[li]);
        const uint32_t off = __ldcg(&rb.bucket_off[t]), b = __ldcg(&rb.bucket_len[t]);
        const ushort2 span = __ldcg(&rb.bucket_span[t]);
        const uint32_t node = __ldcg(&rb.touched[t]);
        if (span.x >= a.hi || span.y < a.lo) continue;
        NodeState st = fold_load(jc, a, node);
        // the samples are the entries' high words
        const uint32_t *sample = reinterpret_cast<const uint32_t *>(rb.entries + off) + 1;
        uint32_t l = 0, h = span.x >= a.lo ? 0u : b;  // first entry at or beyond lo in [l, h]
        while (h > l) {
            const uint32_t step = (h - l + 31u) / 32u;
            const uint32_t i = l + lane * step;
            const bool below = i < h && __ldcg(&sample[2u * i]) < a.lo;
            const uint32_t k = (uint32_t)__popc(__ballot_sync(0xffffffffu, below));
            if (k == 0u) break;
            h = min(h, l + k * step);
            l = l + (k - 1u) * step + 1u;
        }
        DrawEntry e{0.0, 0u, 0xffffffffu}, next[kAhead];
#pragma unroll
        for (uint32_t p = 0; p < kAhead; p++)
            if (l + p * 32u + lane < b) next[p] = entry_load(rb, off + l + p * 32u + lane);
        const bool few = (uint64_t)a.first_sample + a.hi < (1ull << 26);
        bool first = true;
        for (uint32_t i = l;; i += 32u) {
            e = next[0];
#pragma unroll
            for (uint32_t p = 0; p + 1 < kAhead; p++) next[p] = next[p + 1];
            const uint32_t k =
                (uint32_t)__popc(__ballot_sync(0xffffffffu, i + lane < b && e.sample < a.hi));
            if (k == 0u) break;
            if (first && a.journal) fold_journal(jr, a, t, st);
            first = false;
            if (lane < k) fold_stage(fs, lane, e);
            const uint32_t far = i + kAhead * 32u + lane;
            if (far < b) next[kAhead - 1] = entry_load(rb, off + far);
            __syncwarp();
            const bool one = e.x == 1.0;
            const bool plain = one || (e.x >= 0x1p-25 && e.x <= 1.0 - 0x1p-25);
            if (k == 32u && few && __all_sync(0xffffffffu, plain))
                fold_full(jc, a, node, __ballot_sync(0xffffffffu, one), st, fs);
            else
                fold_entries(jc, a, node, k, st, fs);
            if (k < 32u) break;
        }
        if (!first) fold_store(jc, a, node, st, fs);
    }
}

// Buckets of at most 32 entries: a warp looks at up to kBatch of them (one where
// there are as many warps), leaves out those without samples of the round by their span, and folds the others one
// after another, the next one's entries and counters loaded meanwhile.
__device__ void fold_small(const RoundBuffers &rb, const JobCounters &jc, const RoundJournal &jr,
                           const ApplyArgs &a, uint32_t T, uint32_t w, uint32_t nw,
                           FoldScratch &fs) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t batch = min(kBatch, (T + nw - 1u) / nw);
    for (uint32_t t0 = w * batch; t0 < T; t0 += nw * batch) {
        const uint32_t t = t0 + lane;
        uint32_t off = 0, len = 33, node = 0;
        ushort2 span = make_ushort2(0, 0);
        if (lane < batch && t < T) {
            off = __ldcg(&rb.bucket_off[t]);
            len = __ldcg(&rb.bucket_len[t]);
            span = __ldcg(&rb.bucket_span[t]);
            node = __ldcg(&rb.touched[t]);
        }
        uint32_t m = __ballot_sync(0xffffffffu, len <= 32u && span.x < a.hi && span.y >= a.lo);
        int i = m ? __ffs(m) - 1 : 0;
        uint32_t o_n = __shfl_sync(0xffffffffu, off, i), l_n = __shfl_sync(0xffffffffu, len, i);
        uint32_t v_n = __shfl_sync(0xffffffffu, node, i);
        DrawEntry e_n{0.0, 0u, 0xffffffffu};
        NodeState s_n{0.0, 0u, 0u, true};
        if (m) {
            if (lane < l_n) e_n = entry_load(rb, o_n + lane);
            s_n = fold_load(jc, a, v_n);
        }
        while (m) {
            const uint32_t at = t0 + (uint32_t)i, v = v_n, l = l_n;
            const DrawEntry e = e_n;
            NodeState st = s_n;
            m &= m - 1u;
            if (m) {
                i = __ffs(m) - 1;
                o_n = __shfl_sync(0xffffffffu, off, i);
                l_n = __shfl_sync(0xffffffffu, len, i);
                v_n = __shfl_sync(0xffffffffu, node, i);
                e_n.sample = 0xffffffffu;
                if (lane < l_n) e_n = entry_load(rb, o_n + lane);
                s_n = fold_load(jc, a, v_n);
            }
            const bool in = lane < l && e.sample >= a.lo && e.sample < a.hi;
            const uint32_t im = __ballot_sync(0xffffffffu, in);
            if (!im) continue;
            if (a.journal) fold_journal(jr, a, at, st);
            if (in) fold_stage(fs, (uint32_t)__popc(im & ((1u << lane) - 1u)), e);
            __syncwarp();
            fold_entries(jc, a, v, (uint32_t)__popc(im), st, fs);
            fold_store(jc, a, v, st, fs);
        }
    }
}

__device__ void commit_sums(const RoundBuffers &rb, const JobCounters &jc, const ApplyArgs &a) {
    unsigned long long vis = 0, cnt = 0, vd = 0, paths = 0, ball = 0, pred = 0;
    for (uint32_t s = a.lo + blockIdx.x * blockDim.x + threadIdx.x; s < a.hi;
         s += gridDim.x * blockDim.x) {
        const int32_t st = rb.status[s];
        if (st != 0) atomicCAS(&jc.sc->error, 0, st);
        vis += rb.vis[s];
        ball += rb.ball[s];
        pred += rb.pred[s];
        const int32_t pl = rb.pl[s];
        if (pl > 0) {
            if ((uint32_t)pl <= a.D) atomicAdd((unsigned long long *)&jc.sp_lengths[pl], 1ull);
            else atomicCAS(&jc.sc->error, 0, SILVAN_E_STATE);
            cnt++;
            paths += (unsigned long long)rb.np[s];
        } else {
            vd++;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        vis += __shfl_xor_sync(0xffffffffu, vis, o);
        cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
        vd += __shfl_xor_sync(0xffffffffu, vd, o);
        paths += __shfl_xor_sync(0xffffffffu, paths, o);
        ball += __shfl_xor_sync(0xffffffffu, ball, o);
        pred += __shfl_xor_sync(0xffffffffu, pred, o);
    }
    // per CTA in shared memory, then one global add per CTA and sum
    __shared__ unsigned long long cs[6];
    if (threadIdx.x < 6) cs[threadIdx.x] = 0ull;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        if (vis) atomicAdd(&cs[0], vis);
        if (cnt) atomicAdd(&cs[1], cnt);
        if (vd) atomicAdd(&cs[2], vd);
        if (paths) atomicAdd(&cs[3], paths);
        if (ball) atomicAdd(&cs[4], ball);
        if (pred) atomicAdd(&cs[5], pred);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (cs[0]) atomicAdd(&jc.sc->vis_edges, cs[0]);
        if (cs[1]) atomicAdd(&jc.sc->counted_samples, cs[1]);
        if (cs[2]) atomicAdd(&jc.sc->void_samples, cs[2]);
        if (cs[3]) atomicAdd(&jc.sc->paths, cs[3]);
        if (cs[4]) atomicAdd(&jc.sc->ball_nodes, cs[4]);
        if (cs[5]) atomicAdd(&jc.sc->pred_entries, cs[5]);
    }
}


// Commits the samples [lo, hi) of the grouped draw, WARPS warps a CTA.
template <uint32_t WARPS>
__device__ __forceinline__ void commit_part(const ApplyState &st, uint32_t touched,
                                            uint32_t large, FoldScratch *fsc) {
    const uint32_t wib = threadIdx.x >> 5, nw = gridDim.x * WARPS;
    FoldScratch &fs = fsc[wib];
    fold_begin(fs);
    // the long buckets first, spread over the CTAs
    fold_large(st.rb, st.jc, st.jr, st.a, large, wib * gridDim.x + blockIdx.x, nw, fs);
    fold_small(st.rb, st.jc, st.jr, st.a, touched, blockIdx.x * WARPS + wib, nw, fs);
    fold_flush(st.jc, fs);
    commit_sums(st.rb, st.jc, st.a);
}

__global__ void __launch_bounds__(kRoundThreads, kRoundCtas) commit_round_kernel(
    const ApplyState st) {
    __shared__ FoldScratch fsc[kRoundThreads / 32];
    commit_part<kRoundThreads / 32>(st, __ldcg(st.rb.n_touched + 8), __ldcg(st.rb.n_touched + 9),
                                    fsc);
}

__global__ void __launch_bounds__(kCommitThreads, 1) prepare_draw_kernel(const ApplyState st) {
    __shared__ union {
        OrderSmem order;
        FoldScratch fold[kCommitThreads / 32];
    } sm;
    const RoundBuffers &rb = st.rb;
    const JobCounters &jc = st.jc;
    const ApplyArgs &a = st.a;
    uint32_t *bar = rb.n_touched + 2;
    if (__ldcg(&jc.sc->error) == SILVAN_E_TIMEOUT) {  // the job has failed
        prepare_exit(rb, false);
        return;
    }
    bucket_count(rb, a);
    if (!grid_barrier(bar, a.polls)) goto timeout;
    {
        const uint32_t T = __ldcg(rb.n_touched);
        bucket_alloc(rb, T);
        if (!grid_barrier(bar, a.polls)) goto timeout;
        bucket_scatter(rb, a);
        if (!grid_barrier(bar, a.polls)) goto timeout;
        order_huge(rb, jc, a.count, sm.order);
        order_others(rb, T, sm.order);
        // the scatter cursors back to zero for the next draw
        for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < T;
             t += gridDim.x * blockDim.x)
            rb.node_cnt[rb.touched[t]] = 0;
        if (a.lo < a.hi) {  // a small draw
            if (!grid_barrier(bar, a.polls)) goto timeout;
            commit_part<kCommitThreads / 32>(st, T, __ldcg(rb.n_touched + 1), sm.fold);
        }
    }
    prepare_exit(rb, true);
    return;
timeout:
    if (threadIdx.x == 0) atomicCAS(&jc.sc->error, 0, SILVAN_E_TIMEOUT);
    prepare_exit(rb, false);
}

int g_commit_grid = 0;  // resident CTAs of prepare_draw_kernel (apply_init)
int g_sms = 0;

}  // namespace

cudaError_t apply_init() {
    int dev = 0, per_sm = 0;
    cudaError_t e;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
        return e;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, prepare_draw_kernel,
                                                      kCommitThreads, 0);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorLaunchOutOfResources;
    g_commit_grid = g_sms;
    return cudaSuccess;
}

// One warp per node of the draw's touched list, lanes as in the fold.  The nodes
// that the round folded (and saved) have a last update at or beyond `from`, the
// round's first sample + 1: every contribution is positive.
__global__ void undo_round_kernel(RoundBuffers rb, JobCounters jc, RoundJournal jr, int pass,
                                  uint32_t D, uint32_t from) {
    const uint32_t T = __ldcg(rb.n_touched + 8);
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < T; t += nw) {
        const uint32_t node = rb.touched[t];
        const bool folded = jc.last_upd[node] >= from;
        __syncwarp();  // every lane has looked before lane 25 writes
        if (!folded) continue;
        if (lane < kTrials) {
            if (pass == 2)
                jc.mcrade[(uint64_t)node * kTrials + lane] = jr.mcrade[(uint64_t)t * kTrials + lane];
        } else if (lane == 25) {
            jc.approx[node] = jr.approx[t];
            jc.last_upd[node] = jr.last_upd[t];
        } else if (lane == 26) {
            jc.wimpy[node] = jr.wimpy[t];
        }
    }
    if (blockIdx.x == 0) {
        const unsigned long long *src = reinterpret_cast<const unsigned long long *>(jr.sc);
        unsigned long long *dst = reinterpret_cast<unsigned long long *>(jc.sc);
        for (uint32_t i = threadIdx.x; i < sizeof(JobScalars) / 8; i += blockDim.x) dst[i] = src[i];
        for (uint32_t i = threadIdx.x; i <= D; i += blockDim.x) jc.sp_lengths[i] = jr.sp_lengths[i];
    }
}

cudaError_t prepare_draw(const ApplyState &st, cudaStream_t stream) {
    if (g_commit_grid <= 0) return cudaErrorNotReady;
    if (st.a.count > kDrawSamples) return cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg{};
    // a warp for every record and every sample is enough
    cfg.gridDim = dim3(
        std::min<uint32_t>(g_commit_grid, std::max(st.a.n_records, st.a.count) / 32 + 1));
    cfg.blockDim = dim3(kCommitThreads);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, prepare_draw_kernel, st);
}

cudaError_t apply_round(const ApplyState &st, cudaStream_t stream) {
    if (g_sms <= 0) return cudaErrorNotReady;
    commit_round_kernel<<<g_sms * kRoundCtas, kRoundThreads, 0, stream>>>(st);
    return cudaGetLastError();
}

namespace {

// Neutral accumulator: every maximum at its identity.
__global__ void stop_init_kernel(StopReduction *acc) {
    for (int i = threadIdx.x; i < kMaxPartitions * kTrials; i += blockDim.x)
        acc->mc_max[i] = LLONG_MIN;
    for (int i = threadIdx.x; i < kMaxPartitions; i += blockDim.x) {
        acc->wimpy_max[i] = 0.0;
        acc->touched[i] = 0;
    }
    if (threadIdx.x == 0) {
        acc->approx_max = 0.0;
        acc->wimpy_all_max = 0.0;
    }
}

// One warp per updated node: lanes 0..24 read the node's 25 trials (one
// 200-byte row), lane 25 approx and wimpy.  Each CTA folds its nodes in
// shared memory and into the device accumulator; the last CTA out writes the
// result, the job's scalars and the path-length counts to the (host-mapped)
// readback and leaves the accumulator neutral for the next check.
__global__ void __launch_bounds__(512) stop_reduce_kernel(JobCounters jc, int nparts, uint32_t D,
                                                          StopReduction *acc, uint32_t *ticket,
                                                          StopReadback rb, RoundJournal jr) {
    __shared__ long long smc[kMaxPartitions * kTrials];
    __shared__ unsigned long long sw[kMaxPartitions];
    __shared__ uint32_t st[kMaxPartitions];
    __shared__ bool last;
    for (int i = threadIdx.x; i < nparts * kTrials; i += blockDim.x) smc[i] = LLONG_MIN;
    for (int i = threadIdx.x; i < nparts; i += blockDim.x) {
        sw[i] = 0ull;
        st[i] = 0;
    }
    __syncthreads();
    const uint32_t T = jc.sc->n_upd;
    const int lane = threadIdx.x & 31;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    unsigned long long amax = 0, wmax = 0;
    // kNodes nodes per warp at a time, their loads in flight together
    constexpr int kNodes = 4;
    for (uint32_t t0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t0 < T; t0 += kNodes * nw) {
        uint32_t v[kNodes];
        int p[kNodes];
        long long m[kNodes];
        unsigned long long wb[kNodes], ab[kNodes];
#pragma unroll
        for (int i = 0; i < kNodes; i++) {
            const uint32_t t = t0 + (uint32_t)i * nw;
            v[i] = t < T ? jc.upd_list[t] : 0xffffffffu;
        }
#pragma unroll
        for (int i = 0; i < kNodes; i++) {
            p[i] = 0;
            m[i] = LLONG_MIN;
            wb[i] = ab[i] = 0ull;
            if (v[i] == 0xffffffffu) continue;
            p[i] = jc.partition[v[i]];
            if (lane < kTrials) {
                m[i] = jc.mcrade[(uint64_t)v[i] * kTrials + lane];
            } else if (lane == kTrials) {
                wb[i] = (unsigned long long)__double_as_longlong(jc.wimpy[v[i]]);
                ab[i] = (unsigned long long)__double_as_longlong(jc.approx[v[i]]);
            }
        }
#pragma unroll
        for (int i = 0; i < kNodes; i++) {
            if (v[i] == 0xffffffffu) continue;
            if (lane < kTrials) {
                if (m[i] > smc[p[i] * kTrials + lane]) atomicMax(&smc[p[i] * kTrials + lane], m[i]);
            } else if (lane == kTrials) {
                if (wb[i] > sw[p[i]]) atomicMax(&sw[p[i]], wb[i]);
                atomicAdd(&st[p[i]], 1u);
                amax = ab[i] > amax ? ab[i] : amax;
                wmax = wb[i] > wmax ? wb[i] : wmax;
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        unsigned long long x = __shfl_xor_sync(0xffffffffu, amax, o);
        unsigned long long y = __shfl_xor_sync(0xffffffffu, wmax, o);
        amax = x > amax ? x : amax;
        wmax = y > wmax ? y : wmax;
    }
    if (lane == 0) {
        if (amax) atomicMax(reinterpret_cast<unsigned long long *>(&acc->approx_max), amax);
        if (wmax) atomicMax(reinterpret_cast<unsigned long long *>(&acc->wimpy_all_max), wmax);
    }
    __syncthreads();
    // every CTA folds the same few hundred words: an atomic only where this
    // CTA's value is above the accumulator's (most are not), so that the
    // CTAs do not queue on the same addresses
    for (int i = threadIdx.x; i < nparts * kTrials; i += blockDim.x)
        if (smc[i] != LLONG_MIN && smc[i] > __ldcg(&acc->mc_max[i]))
            atomicMax(&acc->mc_max[i], smc[i]);
    for (int i = threadIdx.x; i < nparts; i += blockDim.x) {
        unsigned long long *wm = reinterpret_cast<unsigned long long *>(&acc->wimpy_max[i]);
        if (sw[i] && sw[i] > __ldcg(wm)) atomicMax(wm, sw[i]);
        if (st[i]) atomicAdd(&acc->touched[i], st[i]);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int i = threadIdx.x; i < nparts * kTrials; i += blockDim.x) {
        rb.red->mc_max[i] = __ldcg(&acc->mc_max[i]);
        acc->mc_max[i] = LLONG_MIN;
    }
    for (int i = threadIdx.x; i < nparts; i += blockDim.x) {
        rb.red->wimpy_max[i] = __ldcg(&acc->wimpy_max[i]);
        rb.red->touched[i] = __ldcg(&acc->touched[i]);
        acc->wimpy_max[i] = 0.0;
        acc->touched[i] = 0;
    }
    if (threadIdx.x == 0) {
        rb.red->approx_max = __ldcg(&acc->approx_max);
        rb.red->wimpy_all_max = __ldcg(&acc->wimpy_all_max);
        acc->approx_max = 0.0;
        acc->wimpy_all_max = 0.0;
        *ticket = 0u;
    }
    const unsigned long long *src = reinterpret_cast<const unsigned long long *>(jc.sc);
    unsigned long long *dst = reinterpret_cast<unsigned long long *>(rb.sc);
    unsigned long long *keep = reinterpret_cast<unsigned long long *>(jr.sc);
    for (uint32_t i = threadIdx.x; i < sizeof(JobScalars) / 8; i += blockDim.x) {
        const unsigned long long x = __ldcg(&src[i]);
        dst[i] = x;
        if (keep) keep[i] = x;
    }
    for (uint32_t i = threadIdx.x; i <= D; i += blockDim.x) {
        const uint64_t x = __ldcg(&jc.sp_lengths[i]);
        if (rb.sp) rb.sp[i] = x;
        if (jr.sp_lengths) jr.sp_lengths[i] = x;
    }
}

// Peeling index of node v (Probabilistic.cpp:855-862), stored in peel_idx.
// The C library's log may differ from the device's by an ulp; the nodes
// where that could move (int)t are listed so that the host recomputes them.
__device__ __forceinline__ int32_t peel_index_of(const JobCounters &jc, uint32_t v, double m,
                                                 double la, uint32_t *unc, uint32_t *n_unc,
                                                 uint32_t cap) {
    const double ew = jc.wimpy[v] / m;
    const double mi = fmin(1. / ew, m);
    const double t = log(mi) / la + 1;
    const int32_t idx = (int)t;
    jc.peel_idx[v] = idx;
    const double fr = t - floor(t);
    if (fr < 1e-9 || fr > 1.0 - 1e-9) {
        uint32_t k = atomicAdd(n_unc, 1u);
        if (k < cap) unc[k] = v;
    }
    return idx;
}

// The end of pass 1 in one kernel: with peeling (nbins > 0) every node's
// index, the uncertain list and the histogram of the indices over
// [idx_min, idx_min + nbins) (hist and n_unc zeroed before); the last CTA
// out copies the histogram, the uncertain count, the scalars and the
// path-length counts to `out` (host-mapped).
__global__ void __launch_bounds__(512) pass1_readback_kernel(
    JobCounters jc, uint32_t n, double m, double a, int32_t idx_min, int32_t nbins,
    uint32_t *hist, uint32_t *unc, uint32_t *n_unc, uint32_t cap, uint32_t D, uint32_t *ticket,
    Pass1Readback out) {
    extern __shared__ uint32_t sh[];
    __shared__ bool last;
    const bool local = nbins > 0 && nbins <= kPeelLocalBins;
    if (local)
        for (int i = threadIdx.x; i < nbins; i += blockDim.x) sh[i] = 0;
    __syncthreads();
    if (nbins > 0) {
        const double la = log(a);
        for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n;
             v += gridDim.x * blockDim.x) {
            int32_t b = peel_index_of(jc, v, m, la, unc, n_unc, cap) - idx_min;
            b = b < 0 ? 0 : (b >= nbins ? nbins - 1 : b);
            atomicAdd(local ? &sh[b] : &hist[b], 1u);
        }
    }
    __syncthreads();
    if (local)
        for (int i = threadIdx.x; i < nbins; i += blockDim.x)
            if (sh[i]) atomicAdd(&hist[i], sh[i]);
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int i = threadIdx.x; i < nbins; i += blockDim.x) out.hist[i] = __ldcg(&hist[i]);
    if (threadIdx.x == 0) {
        *out.n_unc = __ldcg(n_unc);
        *ticket = 0u;
    }
    const unsigned long long *src = reinterpret_cast<const unsigned long long *>(jc.sc);
    unsigned long long *dst = reinterpret_cast<unsigned long long *>(out.sc);
    for (uint32_t i = threadIdx.x; i < sizeof(JobScalars) / 8; i += blockDim.x) dst[i] = __ldcg(&src[i]);
    for (uint32_t i = threadIdx.x; i <= D; i += blockDim.x) out.sp[i] = __ldcg(&jc.sp_lengths[i]);
}

// Zeroes approx, wimpy and last_upd of the nodes on upd_list (every node
// with a non-zero one): the counters of pass 2 start from zero.
__global__ void reset_updated_kernel(JobCounters jc) {
    const uint32_t T = jc.sc->n_upd;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < T; t += gridDim.x * blockDim.x) {
        const uint32_t v = jc.upd_list[t];
        jc.approx[v] = 0.0;
        jc.wimpy[v] = 0.0;
        jc.last_upd[v] = 0u;
    }
}

// Shared-memory histogram per block (the bins are few: about log(m)/log(a)).
__global__ void peel_hist_kernel(JobCounters jc, uint32_t n, int32_t idx_min, int32_t nbins,
                                 uint32_t *hist) {
    extern __shared__ uint32_t sh[];
    for (int i = threadIdx.x; i < nbins; i += blockDim.x) sh[i] = 0;
    __syncthreads();
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        int32_t b = jc.peel_idx[v] - idx_min;
        b = b < 0 ? 0 : (b >= nbins ? nbins - 1 : b);
        atomicAdd(&sh[b], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nbins; i += blockDim.x)
        if (sh[i]) atomicAdd(&hist[i], sh[i]);
}

__global__ void peel_hist_global_kernel(JobCounters jc, uint32_t n, int32_t idx_min,
                                        int32_t nbins, uint32_t *hist) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        int32_t b = jc.peel_idx[v] - idx_min;
        b = b < 0 ? 0 : (b >= nbins ? nbins - 1 : b);
        atomicAdd(&hist[b], 1u);
    }
}

__global__ void peel_map_kernel(JobCounters jc, uint32_t n, const int32_t *lut, int32_t idx_min,
                                int32_t lut_size) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        int32_t b = jc.peel_idx[v] - idx_min;
        b = b < 0 ? 0 : (b >= lut_size ? lut_size - 1 : b);
        jc.partition[v] = lut[b];
    }
}

}  // namespace

__global__ void divide_kernel(const double *approx, double m, double *out, uint32_t n) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
        out[v] = __ddiv_rn(approx[v], m);
}

cudaError_t undo_round(const RoundBuffers &rb, const JobCounters &jc, const RoundJournal &jr,
                       int pass, uint32_t D, uint32_t from, cudaStream_t stream) {
    undo_round_kernel<<<296, 512, 0, stream>>>(rb, jc, jr, pass, D, from);
    return cudaGetLastError();
}

cudaError_t divide_estimates(const double *approx, double num_samples, double *out, uint32_t n,
                             cudaStream_t stream) {
    divide_kernel<<<592, 256, 0, stream>>>(approx, num_samples, out, n);
    return cudaGetLastError();
}

cudaError_t stop_reduce_init(StopReduction *acc, uint32_t *ticket, cudaStream_t stream) {
    stop_init_kernel<<<1, 256, 0, stream>>>(acc);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return cudaMemsetAsync(ticket, 0, sizeof(uint32_t), stream);
}

cudaError_t stop_reduce(const JobCounters &jc, int nparts, uint32_t D, StopReduction *acc,
                        uint32_t *ticket, const StopReadback &out, const RoundJournal &jr,
                        cudaStream_t stream) {
    stop_reduce_kernel<<<296, 512, 0, stream>>>(jc, nparts, D, acc, ticket, out, jr);
    return cudaGetLastError();
}

cudaError_t pass1_readback(const JobCounters &jc, uint32_t n, double num_samples, double a,
                           int32_t idx_min, int32_t nbins, uint32_t *hist, uint32_t *uncertain,
                           uint32_t *n_uncertain, uint32_t cap, uint32_t D, uint32_t *ticket,
                           const Pass1Readback &out, cudaStream_t stream) {
    cudaError_t e = cudaMemsetAsync(n_uncertain, 0, sizeof(uint32_t), stream);
    if (e == cudaSuccess && nbins > 0)
        e = cudaMemsetAsync(hist, 0, sizeof(uint32_t) * nbins, stream);
    if (e != cudaSuccess) return e;
    const size_t smem = nbins > 0 && nbins <= kPeelLocalBins ? sizeof(uint32_t) * nbins : 0;
    pass1_readback_kernel<<<296, 512, smem, stream>>>(jc, n, num_samples, a, idx_min, nbins, hist,
                                                      uncertain, n_uncertain, cap, D, ticket, out);
    return cudaGetLastError();
}

cudaError_t reset_updated(const JobCounters &jc, cudaStream_t stream) {
    reset_updated_kernel<<<296, 512, 0, stream>>>(jc);
    return cudaGetLastError();
}

cudaError_t peel_hist(const JobCounters &jc, uint32_t n, int32_t idx_min, int32_t nbins,
                      uint32_t *hist, cudaStream_t stream) {
    cudaMemsetAsync(hist, 0, sizeof(uint32_t) * nbins, stream);
    if (nbins <= kPeelLocalBins)
        peel_hist_kernel<<<296, 512, sizeof(uint32_t) * nbins, stream>>>(jc, n, idx_min, nbins,
                                                                          hist);
    else
        peel_hist_global_kernel<<<592, 256, 0, stream>>>(jc, n, idx_min, nbins, hist);
    return cudaGetLastError();
}

cudaError_t peel_map(const JobCounters &jc, uint32_t n, const int32_t *lut, int32_t idx_min,
                     int32_t lut_size, uint32_t *hist, cudaStream_t stream) {
    (void)hist;
    peel_map_kernel<<<592, 256, 0, stream>>>(jc, n, lut, idx_min, lut_size);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Top-K selection of the ranking (see counters.cuh).  A node's key is the
// 128-bit (approx bits, last update << 32 | node), compared as an unsigned
// number: approx is non-negative, so its bit pattern orders like its value,
// and node ids make every key distinct.  Digit i (i = 0 the most
// significant) is 16 bits of it.
// ---------------------------------------------------------------------------
namespace {

constexpr uint32_t kTopkSortCap = 8192;  // candidates one CTA sorts in shared memory

struct Key128 {
    unsigned long long hi, lo;
};

__device__ __forceinline__ Key128 node_key(const JobCounters &jc, uint32_t v) {
    Key128 k;
    k.hi = (unsigned long long)__double_as_longlong(jc.approx[v]);
    k.lo = ((unsigned long long)jc.last_upd[v] << 32) | v;
    return k;
}

// word w (0 most significant) of the key
__device__ __forceinline__ uint32_t key_word(const Key128 &k, int w) {
    const unsigned long long x = w < 2 ? k.hi : k.lo;
    return (w & 1) ? (uint32_t)x : (uint32_t)(x >> 32);
}

__device__ __forceinline__ uint32_t key_digit(const Key128 &k, uint32_t i) {
    return (key_word(k, (int)(i >> 1)) >> ((i & 1) ? 0 : 16)) & 0xffffu;
}

// -1, 0, 1: the key's first L digits against the prefix's (4 words).
__device__ __forceinline__ int cmp_prefix(const Key128 &k, const uint32_t *pre, uint32_t L) {
    for (uint32_t w = 0; w < 4 && 2 * w < L; w++) {
        const uint32_t mask = (2 * w + 1 < L) ? 0xffffffffu : 0xffff0000u;
        const uint32_t a = key_word(k, (int)w) & mask, b = pre[w] & mask;
        if (a != b) return a < b ? -1 : 1;
    }
    return 0;
}

// state: [0] digits fixed (L), [1..4] prefix words, [5] nodes known to be
// above the prefix's group, [6] size of the group, [7] candidates
__global__ void topk_hist_kernel(JobCounters jc, uint32_t n_upd, const uint32_t *state,
                                 uint32_t *hist) {
    const uint32_t L = state[0];
    uint32_t pre[4] = {state[1], state[2], state[3], state[4]};
    const int lane = threadIdx.x & 31;
    for (uint32_t t0 = blockIdx.x * blockDim.x; t0 < n_upd; t0 += gridDim.x * blockDim.x) {
        const uint32_t t = t0 + threadIdx.x;
        bool in = false;
        uint32_t d = 0;
        if (t < n_upd) {
            const Key128 k = node_key(jc, jc.upd_list[t]);
            in = cmp_prefix(k, pre, L) == 0;
            d = key_digit(k, L);
        }
        // one atomic per distinct digit of the warp
        const uint32_t act = __ballot_sync(0xffffffffu, in);
        if (in) {
            const uint32_t peers = __match_any_sync(act, d);
            if ((peers & ((1u << lane) - 1u)) == 0u) atomicAdd(&hist[d], (uint32_t)__popc(peers));
        }
    }
}

// One CTA of 1024 threads: the digit d of level L at which the K-th key lies
// (counting from the largest), the count above it, and the state of the
// next level (its prefix extended by d).
__global__ void __launch_bounds__(1024) topk_pick_kernel(const uint32_t *hist, uint32_t *state,
                                                         uint32_t K) {
    __shared__ uint32_t ws[32];
    __shared__ uint32_t found;
    const uint32_t L = state[0], above = state[5];
    const uint32_t t = threadIdx.x;
    const int lane = t & 31, warp = t >> 5;
    // thread t owns digits [hi - 63, hi], hi = 65535 - 64 t (descending)
    const uint32_t top = 65535u - 64u * t;
    uint32_t sum = 0;
    for (int j = 0; j < 64; j++) sum += hist[top - j];
    uint32_t incl = sum;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += x;
    }
    if (lane == 31) ws[warp] = incl;
    if (t == 0) found = 0;
    __syncthreads();
    if (warp == 0) {
        const uint32_t w = ws[lane];
        uint32_t wi = w;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += x;
        }
        ws[lane] = wi - w;
    }
    __syncthreads();
    uint32_t before = above + ws[warp] + incl - sum;  // keys above this thread's digits
    if (before < K && before + sum >= K) {
        for (int j = 0; j < 64; j++) {
            const uint32_t h = hist[top - j];
            if (before + h >= K) {
                const uint32_t d = top - j;
                const uint32_t w = L >> 1;
                state[1 + w] |= (L & 1) ? d : (d << 16);
                state[0] = L + 1;
                state[5] = before;
                state[6] = h;
                found = 1;
                break;
            }
            before += h;
        }
    }
    __syncthreads();
    if (t == 0 && !found) state[0] = 0xffffffffu;  // fewer than K keys: cannot happen
}

// Every updated node whose first L digits are at least the prefix's.
__global__ void topk_collect_kernel(JobCounters jc, uint32_t n_upd, uint32_t *state,
                                    unsigned long long *cand, uint32_t cap) {
    const uint32_t L = state[0];
    uint32_t pre[4] = {state[1], state[2], state[3], state[4]};
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n_upd;
         t += gridDim.x * blockDim.x) {
        const Key128 k = node_key(jc, jc.upd_list[t]);
        if (cmp_prefix(k, pre, L) >= 0) {
            const uint32_t i = atomicAdd(&state[7], 1u);
            if (i < cap) {
                cand[2 * i] = k.hi;
                cand[2 * i + 1] = k.lo;
            }
        }
    }
}

// One CTA: bitonic sort of the n <= kTopkSortCap candidates, largest first,
// in shared memory; the sorted keys go back to cand.
__global__ void __launch_bounds__(1024) topk_sort_kernel(unsigned long long *cand,
                                                         const uint32_t *state) {
    extern __shared__ unsigned long long kv[];  // 2 x P words
    const uint32_t n = state[7];
    uint32_t P = 64;
    while (P < n) P <<= 1;
    for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) {
        kv[2 * i] = i < n ? cand[2 * i] : 0ull;
        kv[2 * i + 1] = i < n ? cand[2 * i + 1] : 0ull;
    }
    __syncthreads();
    for (uint32_t k = 2; k <= P; k <<= 1) {
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) {
                const uint32_t l = i ^ j;
                if (l > i) {
                    const unsigned long long ah = kv[2 * i], al = kv[2 * i + 1];
                    const unsigned long long bh = kv[2 * l], bl = kv[2 * l + 1];
                    const bool a_less = ah < bh || (ah == bh && al < bl);
                    const bool desc = (i & k) == 0;
                    if (desc ? a_less : !a_less) {
                        kv[2 * i] = bh;
                        kv[2 * i + 1] = bl;
                        kv[2 * l] = ah;
                        kv[2 * l + 1] = al;
                    }
                }
            }
            __syncthreads();
        }
    }
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        cand[2 * i] = kv[2 * i];
        cand[2 * i + 1] = kv[2 * i + 1];
    }
}

}  // namespace

uint32_t topk_capacity(uint32_t K) { return std::max<uint32_t>(kTopkSortCap, 2u * K); }

int topk_select(const JobCounters &jc, uint32_t n_upd, uint32_t K, const TopkBuffers &tb,
                cudaStream_t stream, uint32_t *nodes, double *values, uint32_t *count) {
    *count = 0;
    if (n_upd == 0 || K == 0) return SILVAN_OK;
    if (tb.cap < topk_capacity(K)) return SILVAN_E_BADARG;
    static bool attr_set = false;  // the sort kernel's shared memory (once per process)
    if (!attr_set) {
        if (cudaFuncSetAttribute(topk_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(2 * kTopkSortCap * sizeof(unsigned long long))) !=
            cudaSuccess)
            return SILVAN_E_CUDA;
        attr_set = true;
    }
    uint32_t *hs = tb.h_state;
    for (int i = 0; i < 8; i++) hs[i] = 0;
    if (cudaMemcpyAsync(tb.state, hs, 8 * sizeof(uint32_t), cudaMemcpyHostToDevice, stream) !=
        cudaSuccess)
        return SILVAN_E_CUDA;
    // refine while the candidates (keys at or above the prefix) would not fit
    uint32_t ncand = n_upd;
    while (ncand > tb.cap) {
        if (cudaMemsetAsync(tb.hist, 0, 65536 * sizeof(uint32_t), stream) != cudaSuccess)
            return SILVAN_E_CUDA;
        topk_hist_kernel<<<592, 256, 0, stream>>>(jc, n_upd, tb.state, tb.hist);
        topk_pick_kernel<<<1, 1024, 0, stream>>>(tb.hist, tb.state, K);
        if (cudaMemcpyAsync(hs, tb.state, 8 * sizeof(uint32_t), cudaMemcpyDeviceToHost,
                            stream) != cudaSuccess ||
            cudaStreamSynchronize(stream) != cudaSuccess)
            return SILVAN_E_CUDA;
        if (hs[0] > 8) return SILVAN_E_STATE;
        ncand = hs[5] + hs[6];
        if (hs[0] == 8 && ncand > tb.cap) return SILVAN_E_STATE;  // keys are distinct
    }
    topk_collect_kernel<<<592, 256, 0, stream>>>(jc, n_upd, tb.state, tb.cand, tb.cap);
    if (cudaMemcpyAsync(hs, tb.state, 8 * sizeof(uint32_t), cudaMemcpyDeviceToHost, stream) !=
            cudaSuccess ||
        cudaStreamSynchronize(stream) != cudaSuccess)
        return SILVAN_E_CUDA;
    const uint32_t n = hs[7];
    if (n > tb.cap || n < std::min(K, n_upd)) return SILVAN_E_STATE;
    const uint32_t take = std::min(K, n);
    if (n <= kTopkSortCap) {
        topk_sort_kernel<<<1, 1024, 2 * kTopkSortCap * sizeof(unsigned long long), stream>>>(
            tb.cand, tb.state);
        if (cudaMemcpyAsync(tb.h_cand, tb.cand, 2 * sizeof(unsigned long long) * take,
                            cudaMemcpyDeviceToHost, stream) != cudaSuccess ||
            cudaStreamSynchronize(stream) != cudaSuccess)
            return SILVAN_E_CUDA;
    } else {
        // more than one CTA sorts: the (at most 2K) candidates are ordered on
        // the host, still without any n-sized transfer
        if (cudaMemcpyAsync(tb.h_cand, tb.cand, 2 * sizeof(unsigned long long) * n,
                            cudaMemcpyDeviceToHost, stream) != cudaSuccess ||
            cudaStreamSynchronize(stream) != cudaSuccess)
            return SILVAN_E_CUDA;
        std::vector<uint32_t> ord(n);
        for (uint32_t i = 0; i < n; i++) ord[i] = i;
        const unsigned long long *c = tb.h_cand;
        std::partial_sort(ord.begin(), ord.begin() + take, ord.end(), [&](uint32_t x, uint32_t y) {
            return c[2 * x] != c[2 * y] ? c[2 * x] > c[2 * y] : c[2 * x + 1] > c[2 * y + 1];
        });
        std::vector<unsigned long long> tmp(2 * (size_t)take);
        for (uint32_t i = 0; i < take; i++) {
            tmp[2 * i] = c[2 * ord[i]];
            tmp[2 * i + 1] = c[2 * ord[i] + 1];
        }
        std::copy(tmp.begin(), tmp.end(), tb.h_cand);
    }
    for (uint32_t i = 0; i < take; i++) {
        nodes[i] = (uint32_t)tb.h_cand[2 * i + 1];
        std::memcpy(&values[i], &tb.h_cand[2 * i], sizeof(double));
    }
    *count = take;
    return SILVAN_OK;
}

}  // namespace silvan
