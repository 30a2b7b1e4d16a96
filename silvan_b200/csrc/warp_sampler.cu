// The samples of a round, one warp each (see warp_sampler.cuh).
//
// What the search keeps.  A visited node leaves one 32-byte record (BallRec)
// at its queue position in the warp's part of global memory, and an entry in
// a hash table in shared memory (node -> side and queue position).  Nothing
// is indexed by node and nothing is restored after the sample.
//
// A level is scanned in the reference's order (silvan/src/Sp_sampler.cpp:
// 116-140): the frontier 32 nodes at a time, their adjacency entries 32 at a
// time, one per lane.  The entries of one node come before the next one's and
// a row holds a node once, so within a round the lowest lane that reaches a
// node not in the table joins it, and a later round can only add hits:
//   joining hit  table entry and record written, queue position by its rank
//                among the round's joins;
//   other hits   on a node of the level in progress (its queue position is at
//                or beyond the level's start): count, sigma and last
//                predecessor added to its record;
//   meeting edge an entry of the other side: appended in order.
// There is no second pass and no barrier but the warp's own.
//
// On an undirected graph a neighbour of a frontier node lies on the
// frontier's level or an adjacent one of its own side, or on the other side's
// frontier (an older node of the other side would have joined it to that side
// before), so the table may forget older levels: it is rebuilt from the last
// two levels of either side when it fills up.  A directed search keeps its
// whole ball.
//
// Why one warp.  The CTA sampler pays about 25 us for a sample of a hundred
// entries (8 CTAs of 128 threads an SM): five barriers and as many dependent
// trips to L2 a level, most of its warps waiting.  Here a level costs two
// trips (rows, adjacency) and no barrier, and 21 samples run on an SM.  One
// B200, sampler time of a run with 21 warps an SM against the CTA sampler alone:
// 2.3 k samples on a Barabasi-Albert graph of 600 nodes 0.06 ms, before 0.11;
// 14 k on one of 10 k nodes 0.43 ms, before 0.82; 263 k on R-MAT 14 9.6 ms,
// before 10.3.  It is bound by instruction issue and latency, not by bandwidth: with
// samples for all warps 0.54 instructions a cycle and scheduler, five warps on each,
// an instruction waiting as long for the one before as for memory; DRAM 14 %
// (R-MAT 16).
// A CTA of four warps around the same table was slower than the general
// search: its fixed cost per level is paid by every warp.
#include <algorithm>
#include <cstddef>

#include "sampler_dev.cuh"
#include "warp_sampler.cuh"

namespace silvan {

namespace {

// Table entries of a warp: the resident warps of an SM share its shared memory.
// 1024 entries (10 KB, 21 warps an SM) draw R-MAT 14 samples faster than 2048
// (18 KB, 12 warps, 5 % longer, sampler time of a top-10 run) and 4096 (7 %).
constexpr uint32_t kWarpTable = 1024;
// The warps of an SM that the registers allow for; shared memory holds 21 of them.
constexpr int kWarpsPerSm = 22;
constexpr int kMaxProbe = 32;  // buckets looked at for one node
constexpr uint32_t kNoKey = 0xffffffffu;
// A table value: kSettled | (side V ? kSettledV : 0) | queue position; below
// kSettled a node that the round in progress reached first.
constexpr uint32_t kSettled = 0x80000000u, kSettledV = 0x40000000u, kFresh = 0x3fffffffu;
constexpr uint32_t kPosMask = 0x3fffffffu;
constexpr uint32_t kFull = 0xffffffffu;  // all lanes
constexpr uint32_t kNearMeets = 64;   // meeting edges kept in shared memory
constexpr uint32_t kNearTouched = 128;  // path-map positions kept in shared memory
constexpr uint32_t kWarpPaths = 2048;  // paths of a sample drawn here
constexpr uint32_t kScreenMax = 32;   // samples screened at once, one lane each

constexpr uint32_t kBuckets = kWarpTable / 4;       // of four keys (one 16-byte load)
constexpr uint32_t kTableLimit = kWarpTable * 3 / 4;  // entries in use
// A frontier of more adjacency entries than this is left to the CTA sampler at
// once: its nodes would not fit the table.
constexpr uint32_t kFrontierItems = 4 * kWarpTable;

struct WarpSmem {
    uint4 key[kBuckets];
    uint32_t val[kWarpTable];
    unsigned long long mpre[kNearMeets];
    uint2 meet[kNearMeets];
    uint32_t touched[kNearTouched];
    uint32_t perm[32];
};

// Reads in shared memory that other lanes write to between barriers of the
// warp.
__device__ __forceinline__ uint4 bucket_load(const uint4 *p) {
    uint4 k;
    asm volatile("ld.volatile.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(k.x), "=r"(k.y), "=r"(k.z), "=r"(k.w)
                 : "r"((uint32_t)__cvta_generic_to_shared(p)));
    return k;
}
__device__ __forceinline__ uint32_t value_load(const uint32_t *p) {
    return *reinterpret_cast<const volatile uint32_t *>(p);
}

// This warp's part of the slot arrays.
struct View {
    BallRec *ball;
    uint2 *rows;
    uint32_t *touched;
    uint2 *meet;
    uint64_t *mpre;
    uint2 *lvl;
    uint32_t cap;
};

// The table slots of the lanes' nodes y (where `act`), inserted when absent
// (`won`: by this lane, with value kFresh).  The whole warp goes from bucket to
// bucket together, without branches on single lanes: false when some lane has
// not found its place after kMaxProbe looks.  The values are read after the
// warp has come together again.
__device__ __forceinline__ bool table_slots(WarpSmem &s, uint32_t y, bool act, uint32_t &h,
                                            bool &won) {
    constexpr int kShift = 24;
    static_assert((1u << (32 - kShift)) == kBuckets, "table size");
    uint32_t b = (y * 2654435769u) >> kShift;
    uint32_t *keys = reinterpret_cast<uint32_t *>(s.key);
    won = false;
    h = 0u;
    for (int i = 0; i < kMaxProbe; i++) {
        const uint4 k = bucket_load(&s.key[b]);
        const uint32_t at = k.x == y ? 0u : k.y == y ? 1u : k.z == y ? 2u : k.w == y ? 3u : 4u;
        // a bucket fills from its first key
        const uint32_t used =
            k.x == kNoKey ? 0u : k.y == kNoKey ? 1u : k.z == kNoKey ? 2u : k.w == kNoKey ? 3u : 4u;
        const uint32_t to = min(at, used);  // at > used never names a key
        const bool add = act && at == 4u && used < 4u;
        uint32_t o = y;
        if (add) o = atomicCAS(&keys[4u * b + used], kNoKey, y);
        const bool mine = add && o == kNoKey;
        if (mine) s.val[4u * b + used] = kFresh;
        won = won || mine;
        const bool there = act && to < 4u && (at < 4u || o == kNoKey || o == y);
        if (there) h = 4u * b + to;
        if (to == 4u) b = (b + 1u) & (kBuckets - 1u);
        act = act && !there;
        if (!__any_sync(kFull, act)) return true;
    }
    return false;
}

__device__ __forceinline__ void table_clear(WarpSmem &s) {
    const uint4 e = make_uint4(kNoKey, kNoKey, kNoKey, kNoKey);
#pragma unroll 4
    for (uint32_t i = threadIdx.x & 31; i < kBuckets; i += 32) s.key[i] = e;
}

template <typename T>
__device__ __forceinline__ T warp_inclusive(T v) {
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const T t = __shfl_up_sync(kFull, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// The search's outcome.
struct Found {
    uint32_t nmeet;   // meeting edges (0: the ends are not connected)
    uint32_t end;     // visited nodes
    uint32_t hits;    // predecessor entries
    uint32_t vis;     // adjacency entries scanned (below 2^32: kFrontierItems a level)
    uint32_t depth;   // level of the first end of a meeting edge
    uint32_t wide;    // adjacency entries of the larger frontier, when it does not fit
    bool fits;        // false: the CTA sampler has to draw this sample
};

// The balanced bidirectional BFS (silvan/src/Sp_sampler.cpp:89-144) between
// u and v, whose rows (out of u, into v) are row_u and row_v.
__device__ __forceinline__ Found search(const SegDesc &A, WarpSmem &s, const View &W,
                                        uint32_t u, uint32_t v, uint2 row_u, uint2 row_v) {
    const uint32_t lane = threadIdx.x & 31;
    const uint2 *rows_u = A.out_rows, *rows_v = A.in_rows;
    const uint32_t *adj_u = A.out_adj, *adj_v = A.in_adj;
    const bool window = (A.compact & kCompactWindow) != 0u;
    Found f{0u, 2u, 0u, 0u, 0u, 0u, true};
    table_clear(s);
    __syncwarp();
    bool won;
    uint32_t h;
    table_slots(s, lane ? v : u, lane < 2u, h, won);
    if (lane < 2) {
        const uint32_t x = lane ? v : u;
        rec_store(&W.ball[lane], make_uint4(st_make(lane ? kSideV : kSideU, 0), 0u, 1u, 0u),
                  make_uint4(0u, 0u, x, 0u));
        W.rows[lane] = lane ? row_v : row_u;
        W.lvl[lane * kWarpLevels] = make_uint2(lane, lane + 1u);
        s.val[h] = kSettled | (lane ? kSettledV | 1u : 0u);
    }
    __syncwarp();
    uint32_t keys = 2, end = 2;
    uint32_t lo_u = 0, hi_u = 1, lo_v = 1, hi_v = 2;   // frontiers
    uint32_t sum_u = 0, sum_v = 0, depth_u = 0, depth_v = 0;
    for (;;) {
        const bool side_u = sum_u <= sum_v;
        const uint32_t lo = side_u ? lo_u : lo_v, hi = side_u ? hi_u : hi_v;
        const uint32_t depth = side_u ? depth_u : depth_v;
        const uint2 *rows = side_u ? rows_u : rows_v;
        const uint32_t *adj = side_u ? adj_u : adj_v;
        const uint32_t items =
            depth ? (side_u ? sum_u : sum_v)
                  : (side_u ? row_u.y - row_u.x : row_v.y - row_v.x);
        f.wide = max(max(sum_u, sum_v), items);
        if (items > kFrontierItems || depth + 2u >= kWarpLevels) {
            f.fits = false;
            return f;
        }
        if (window && keys > kWarpTable / 2u) {
            // forget all but the last two levels of either side
            uint2 prev = make_uint2(0u, 0u);
            const uint32_t pd = lane ? depth_v : depth_u;
            if (lane < 2 && pd) prev = __ldcg(&W.lvl[lane * kWarpLevels + pd - 1u]);
            const uint32_t pu0 = __shfl_sync(kFull, prev.x, 0), pu1 = __shfl_sync(kFull, prev.y, 0);
            const uint32_t pv0 = __shfl_sync(kFull, prev.x, 1), pv1 = __shfl_sync(kFull, prev.y, 1);
            const uint32_t live = (hi_u - lo_u) + (hi_v - lo_v) + (pu1 - pu0) + (pv1 - pv0);
            if (live <= kWarpTable / 2u) {
                keys = live;
                table_clear(s);
                __syncwarp();
                for (int i = 0; i < 4; i++) {
                    const uint32_t a = i == 0 ? lo_u : i == 1 ? lo_v : i == 2 ? pu0 : pv0;
                    const uint32_t b = i == 0 ? hi_u : i == 1 ? hi_v : i == 2 ? pu1 : pv1;
                    for (uint32_t q0 = a; q0 < b; q0 += 32) {
                        const uint32_t q = q0 + lane;
                        const uint32_t y = q < b ? __ldcg(&W.ball[q].node) : 0u;
                        if (!table_slots(s, y, q < b, h, won)) {
                            f.fits = false;
                            return f;
                        }
                        if (q < b) s.val[h] = kSettled | ((i & 1) ? kSettledV : 0u) | q;
                    }
                }
                __syncwarp();
            }
        }
        const uint32_t q0 = end;
        uint32_t nmeet = 0, degsum = 0;
        uint2 jrow = make_uint2(0u, 0u);  // a joined node's row, stored a round later
        uint32_t jpos = kNoKey;
        // the frontier, 32 nodes at a time; the next chunk is loaded meanwhile
        uint2 nrow = make_uint2(0u, 0u);
        unsigned long long nsig = 0ull;
        if (lo + lane < hi) {
            nrow = __ldcg(&W.rows[lo + lane]);
            nsig = __ldcg(&W.ball[lo + lane].sigma);
        }
        for (uint32_t c = lo; c < hi; c += 32) {
            uint2 row = nrow;
            unsigned long long sig = nsig;
            uint32_t qx = c + lane;
            nrow = make_uint2(0u, 0u);
            nsig = 0ull;
            if (c + 32u + lane < hi) {
                nrow = __ldcg(&W.rows[c + 32u + lane]);
                nsig = __ldcg(&W.ball[c + 32u + lane].sigma);
            }
            uint32_t deg = row.y - row.x;
            // nodes without entries leave the chunk, the others close up
            const uint32_t nz = __ballot_sync(kFull, deg != 0u);
            if (nz == 0u) continue;
            if (nz & (nz + 1u)) {
                if (deg) s.perm[__popc(nz & lanemask_lt())] = lane;
                __syncwarp();
                const uint32_t k = __popc(nz);
                const int src = lane < k ? (int)s.perm[lane] : (int)lane;
                row.x = __shfl_sync(kFull, row.x, src);
                deg = __shfl_sync(kFull, deg, src);
                sig = __shfl_sync(kFull, sig, src);
                qx = __shfl_sync(kFull, qx, src);
                if (lane >= k) deg = 0u;
                __syncwarp();
            }
            const uint32_t incl = warp_inclusive(deg), excl = incl - deg;
            const uint32_t tot = __shfl_sync(kFull, incl, 31);
            const uint32_t start = row.x - excl;  // + item: its adjacency entry
            f.vis += tot;
            // item base + lane: its frontier node (lane p of the chunk) and its
            // neighbour
            auto item = [&](uint32_t base, uint32_t &p, uint32_t &y) {
                const bool in = incl > base && excl < base + 32u && deg != 0u;
                const uint32_t m =
                    __reduce_or_sync(kFull, in ? 1u << (max(excl, base) - base) : 0u);
                const uint32_t first = __popc(__ballot_sync(kFull, incl <= base));
                p = (first + __popc(m & (lanemask_lt() * 2u + 1u)) - 1u) & 31u;
                const uint32_t at = __shfl_sync(kFull, start, p) + base + lane;
                y = 0u;
                if (base + lane < tot) y = __ldg(&adj[at]);
            };
            uint32_t np, ny;
            item(0u, np, ny);
            for (uint32_t base = 0; base < tot; base += 32) {
                const uint32_t p = np, y = ny;
                if (base + 32u < tot) item(base + 32u, np, ny);
                const bool valid = base + lane < tot;
                const bool placed = table_slots(s, y, valid, h, won);
                __syncwarp();
                uint32_t val = valid ? value_load(&s.val[h]) : 0u;
                const bool fresh = val == kFresh;
                const uint32_t wm = __ballot_sync(kFull, won);
                const uint32_t fm = __ballot_sync(kFull, fresh);
                bool join = won;
                uint32_t jm = wm;
                if (fm != wm) {  // several lanes reached one new node: the lowest joins it
                    if (fresh) atomicMin(&s.val[h], lane);
                    __syncwarp();
                    join = fresh && value_load(&s.val[h]) == lane;
                    jm = __ballot_sync(kFull, join);
                }
                const uint32_t J = __popc(jm);
                keys += J;
                if (!placed || keys > kTableLimit || end + J > W.cap) {
                    f.fits = false;
                    return f;
                }
                // the rows of the round before have arrived
                if (jpos != kNoKey) {
                    W.rows[jpos] = jrow;
                    degsum += jrow.y - jrow.x;
                    jpos = kNoKey;
                }
                const uint32_t px = __shfl_sync(kFull, qx, p);
                const unsigned long long sx = __shfl_sync(kFull, sig, p);
                if (join) {
                    const uint32_t q = end + __popc(jm & lanemask_lt());
                    s.val[h] = kSettled | (side_u ? 0u : kSettledV) | q;
                    rec_store(&W.ball[q],
                              make_uint4(st_make(side_u ? kSideU : kSideV, depth + 1u), 1u,
                                         (uint32_t)sx, (uint32_t)(sx >> 32)),
                              make_uint4(px, px, y, 0u));
                    jrow = __ldg(&rows[y]);
                    jpos = q;
                }
                if (fm != wm) {
                    __syncwarp();
                    if (fresh && !join) val = value_load(&s.val[h]);
                }
                // the other hits on nodes of the level in progress
                const bool old = (val & kSettled) != 0u;
                const bool mine = ((val & kSettledV) == 0u) == side_u;
                const bool more = old && mine && (val & kPosMask) >= q0;
                const uint32_t om = __ballot_sync(kFull, more);
                if (om) {
                    if (more) {
                        BallRec *r = &W.ball[val & kPosMask];
                        atomicAdd(&r->cnt, 1u);
                        atomicMax(&r->last, px);
                        atomicAdd(reinterpret_cast<unsigned long long *>(&r->sigma), sx);
                    }
                }
                f.hits += J + __popc(om);
                const uint32_t mm = __ballot_sync(kFull, old && !mine);
                if (mm) {
                    const uint32_t i = nmeet + __popc(mm & lanemask_lt());
                    if (old && !mine) {
                        const uint2 e = make_uint2(px, val & kPosMask);
                        if (i < kNearMeets) s.meet[i] = e;
                        else if (i < kWarpMeets) W.meet[i] = e;
                    }
                    nmeet += __popc(mm);
                }
                end += J;
                __syncwarp();
            }
        }
        if (jpos != kNoKey) {
            W.rows[jpos] = jrow;
            degsum += jrow.y - jrow.x;
        }
        degsum = __reduce_add_sync(kFull, degsum);
        if (lane == 0) W.lvl[(side_u ? 0u : kWarpLevels) + depth + 1u] = make_uint2(q0, end);
        __syncwarp();
        f.end = end;
        f.depth = depth;
        f.nmeet = nmeet;
        if (nmeet > kWarpMeets) f.fits = false;
        if (nmeet || degsum == 0u) return f;
        if (side_u) {
            lo_u = q0;
            hi_u = end;
            sum_u = degsum;
            depth_u = depth + 1u;
        } else {
            lo_v = q0;
            hi_v = end;
            sum_v = degsum;
            depth_v = depth + 1u;
        }
    }
}

// Predecessor of the node `a` (visited at depth >= 1 of its side), found by
// the whole warp: the level above is walked in queue order, and the nodes on
// a's reverse row are its predecessors.  Plain rule: the one of rank t.
// Weighted rule: the first whose running sum of sigma exceeds t (the last one
// when none does).  Returns its queue position; kNoKey when there is none.
__device__ uint32_t ranked_pred(const SegDesc &A, const View &W, uint32_t a, uint32_t st_a,
                                uint32_t t, bool weighted) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t side = st_side(st_a), d = st_dist(st_a) - 1u;
    const uint2 rr = __ldg(&(side == kSideU ? A.in_rows : A.out_rows)[a]);
    const uint32_t *radj = side == kSideU ? A.in_adj : A.out_adj;
    const uint2 lv = __ldcg(&W.lvl[(side == kSideU ? 0u : kWarpLevels) + d]);
    uint32_t seen = 0, last = kNoKey;
    unsigned long long acc = 0;
    for (uint32_t i0 = lv.x; i0 < lv.y; i0 += 32) {
        const uint32_t i = i0 + lane;
        bool member = false;
        if (i < lv.y) {
            const uint32_t x = __ldcg(&W.ball[i].node);
            uint32_t l = rr.x, h = rr.y;
            while (l < h) {  // first entry >= x
                const uint32_t mid = (l + h) >> 1;
                if (__ldg(&radj[mid]) < x) l = mid + 1;
                else h = mid;
            }
            member = l < rr.y && __ldg(&radj[l]) == x;
        }
        __syncwarp();
        const uint32_t m = __ballot_sync(kFull, member);
        if (!m) continue;
        if (!weighted) {
            const uint32_t k = (uint32_t)__popc(m);
            if (seen + k > t) {
                const bool mine = member && seen + __popc(m & lanemask_lt()) == t;
                return i0 + (uint32_t)__ffs(__ballot_sync(kFull, mine)) - 1u;
            }
            seen += k;
        } else {
            const unsigned long long g =
                warp_inclusive<unsigned long long>(member ? __ldcg(&W.ball[i].sigma) : 0ull);
            const uint32_t over = __ballot_sync(kFull, member && acc + g > t);
            if (over) return i0 + (uint32_t)__ffs(over) - 1u;
            acc += __shfl_sync(kFull, g, 31);
            last = i0 + 31u - (uint32_t)__clz(m);
        }
    }
    return last;
}

// Draws one sample and writes its outputs; false: left to the CTA sampler,
// with nothing written.
__device__ __forceinline__ bool draw_sample(const SegDesc &A, WarpSmem &s, const View &W,
                                            uint32_t sl, uint32_t u, uint32_t v,
                                            uint32_t draw_base, uint2 row_u, uint2 row_v,
                                            uint32_t &wide) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t gidx = A.first_sample + sl;
    const uint64_t seed = A.seed;
    const Found f = search(A, s, W, u, v, row_u, row_v);
    wide = f.wide;
    if (!f.fits) return false;
    const uint32_t nm = f.nmeet;
    int32_t np = 0, pl = 0;
    int32_t status = 0;
    uint32_t nt = 0;
    if (nm) {
        // inclusive prefix of sigma(x) * sigma(y), wrapping; non-decreasing
        // exactly when the 64-bit sum never wrapped (Sp_sampler.cpp:159-170)
        unsigned long long sum = 0ull;
        bool mono = true;
        for (uint32_t i0 = 0; i0 < nm; i0 += 32) {
            const uint32_t i = i0 + lane;
            unsigned long long p = 0ull;
            if (i < nm) {
                const uint2 e = i < kNearMeets ? s.meet[i] : __ldcg(&W.meet[i]);
                p = (unsigned long long)__ldcg(&W.ball[e.x].sigma) *
                    (unsigned long long)__ldcg(&W.ball[e.y].sigma);
            }
            __syncwarp();
            const unsigned long long incl = warp_inclusive(p) + sum;
            const unsigned long long prev = __shfl_up_sync(kFull, incl, 1);
            if (__ballot_sync(kFull, i < nm && incl < (lane ? prev : sum))) mono = false;
            if (i < nm) {
                if (i < kNearMeets) s.mpre[i] = incl;
                else W.mpre[i] = incl;
            }
            sum = __shfl_sync(kFull, incl, 31);
        }
        __syncwarp();
        const uint2 e0 = s.meet[0];
        const uint32_t L = f.depth + st_dist(__ldcg(&W.ball[e0.y].st));
        if (sum == 0ull) return false;
        np = 1;
        if (A.alpha > 0. && sum > 1ull) {
            const double t = A.alpha * (double)sum;
            np = (t >= 2147483648.0) ? INT32_MIN : (int32_t)t;
        }
        pl = np >= 1 ? (int32_t)L : 0;
        if (pl > 0 && ((uint32_t)np > A.np_cap || (uint32_t)np > kWarpPaths ||
                       (uint64_t)draw_base + (uint64_t)np * (1ull + L) > 0xffffffffull))
            return false;
        // ---- paths (:172-197) and backtracks (:241-265): a path's two walks,
        // one from either end of its meeting edge, are one lane's each
        const uint32_t tasks = pl > 0 ? 2u * (uint32_t)np : 0u;
        for (uint32_t t0 = 0; t0 < tasks; t0 += 32) {
            const uint32_t task = t0 + lane;
            bool on = task < tasks;
            uint32_t a = 0, d = 0, pend = kNoKey, pend_old = 1u;
            if (on) {
                d = draw_base + (task >> 1) * (1u + L);
                const uint32_t r = mod_u64(draw32(seed, gidx, d++), sum);
                uint32_t ei = 0;
                auto pre = [&](uint32_t i) -> unsigned long long {
                    return i < kNearMeets ? s.mpre[i] : (unsigned long long)__ldcg(&W.mpre[i]);
                };
                if (mono) {  // first i with prefix > r
                    uint32_t h = nm - 1;
                    while (ei < h) {
                        const uint32_t mid = (ei + h) >> 1;
                        if (pre(mid) > r) h = mid;
                        else ei = mid + 1;
                    }
                } else {
                    while (ei < nm && !(pre(ei) > (unsigned long long)r)) ei++;
                    if (ei >= nm) ei = nm - 1;
                }
                const uint2 e = ei < kNearMeets ? s.meet[ei] : __ldcg(&W.meet[ei]);
                a = (task & 1u) ? e.y : e.x;
                if (task & 1u) d += f.depth;  // the draws of the first walk
            }
            __syncwarp();
            for (uint32_t steps = 0;; steps++) {
                // every step moves one level closer to a root, so a walk
                // longer than L or a position outside the ball is an internal
                // inconsistency: report it, never follow it
                if (on && (a >= f.end || steps > L)) {
                    status = SILVAN_E_STATE;
                    on = false;
                }
                bool find = false, push = false;
                uint32_t rr = 0, node = 0, st = 0, at = pend;
                if (on) {
                    uint4 x, y;
                    rec_load(&W.ball[a], x, y);
                    rr = draw32(seed, gidx, d++);
                    push = pend_old == 0u;
                    pend_old = 1u;
                    st = x.x;
                    node = y.z;
                    if (st_dist(st) == 0u) {  // u or v
                        on = false;
                    } else {
                        pend_old = atomicAdd(&W.ball[a].hit, 1u);
                        pend = a;
                        const unsigned long long sg =
                            (unsigned long long)x.z | ((unsigned long long)x.w << 32);
                        if (sg == 0ull) {
                            status = SILVAN_E_OVERFLOW;
                            on = false;
                        } else {
                            rr = mod_u64(rr, sg);
                            const uint32_t t = min(rr, x.y - 1u);
                            if (A.weighted && x.y > 1u) {
                                find = true;
                            } else if (t == 0u) {
                                a = y.x;
                            } else if (t == x.y - 1u) {
                                a = y.y;
                            } else {
                                rr = t;
                                find = true;
                            }
                        }
                    }
                }
                __syncwarp();
                const uint32_t pm = __ballot_sync(kFull, push);
                if (pm) {
                    const uint32_t i = nt + __popc(pm & lanemask_lt());
                    if (push) {
                        if (i < kNearTouched) s.touched[i] = at;
                        else W.touched[i] = at;
                    }
                    nt += __popc(pm);
                }
                uint32_t fm = __ballot_sync(kFull, find);
                while (fm) {
                    const int src = __ffs(fm) - 1;
                    fm &= fm - 1u;
                    const uint32_t q = ranked_pred(A, W, __shfl_sync(kFull, node, src),
                                                   __shfl_sync(kFull, st, src),
                                                   __shfl_sync(kFull, rr, src), A.weighted != 0);
                    if ((int)lane == src) a = q;  // kNoKey is outside the ball
                    __syncwarp();
                }
                if (!__ballot_sync(kFull, on)) break;
            }
            const bool push = pend_old == 0u;  // of a walk that ended in an error
            const uint32_t pm = __ballot_sync(kFull, push);
            if (pm) {
                const uint32_t i = nt + __popc(pm & lanemask_lt());
                if (push) {
                    if (i < kNearTouched) s.touched[i] = pend;
                    else W.touched[i] = pend;
                }
                nt += __popc(pm);
            }
            __syncwarp();
        }
        // one lane's error is the sample's
        const uint32_t em = __ballot_sync(kFull, status != 0);
        if (em) status = __shfl_sync(kFull, status, __ffs(em) - 1);
    }
    // ---- the path map ----------------------------------------------------------
    unsigned long long rb = ~0ull;
    if (nt > 0 && status == 0) {
        if (lane == 0) rb = atomicAdd(A.rec_cursor, (unsigned long long)nt);
        rb = __shfl_sync(kFull, rb, 0);
        if (rb + nt > A.rec_cap) status = SILVAN_E_CAPACITY;
    }
    if (status == 0) {
        for (uint32_t i = lane; i < nt; i += 32) {
            const uint32_t q = i < kNearTouched ? s.touched[i] : __ldcg(&W.touched[i]);
            const uint2 r = __ldcg(reinterpret_cast<const uint2 *>(&W.ball[q].node));
            PathRec pr;
            pr.node = r.x;
            pr.sample = sl;
            pr.count = r.y;
            A.recs[rb + i] = pr;
        }
    } else if (rb < A.rec_cap) {
        // a path map that did not fit may have reserved places below the
        // buffer's end: they get placeholders
        for (uint32_t i = lane; i < nt && rb + i < A.rec_cap; i += 32) {
            PathRec pr;
            pr.node = 0xffffffffu;
            pr.sample = sl;
            pr.count = 0;
            A.recs[rb + i] = pr;
        }
    }
    if (lane == 0) {
        A.out_pl[sl] = status == 0 ? pl : 0;
        A.out_np[sl] = status == 0 ? np : 0;
        A.out_vis[sl] = f.vis;
        A.out_status[sl] = status;
        A.out_ball[sl] = f.end;
        A.out_pred[sl] = f.hits;
    }
    __syncwarp();
    return true;
}

__global__ void __launch_bounds__(32, kWarpsPerSm) warp_sampler_kernel(WarpLaunch L) {
    __shared__ WarpSmem s;
    const uint32_t lane = threadIdx.x;
    const uint64_t slot = blockIdx.x;
    const View W{L.slots.ball + slot * L.slots.cap,    L.slots.rows + slot * L.slots.cap,
                 L.slots.touched + slot * L.slots.cap,
                 L.slots.meet + slot * kWarpMeets,     L.slots.mpre + slot * kWarpMeets,
                 L.slots.lvl + slot * 2u * kWarpLevels, L.slots.cap};
    const uint32_t total = L.hdr->total, nsegs = L.hdr->nsegs;
    const long long t0 = clock64();
    for (;;) {
        // the next work indices: up to one per lane while many are left
        uint32_t w0 = 0, take = 0;
        if (lane == 0) {
            const uint32_t taken = ld_acquire_u32(&L.hdr->warp_work);
            const uint32_t left = taken < total ? total - taken : 0u;
            take = min(max(left / (4u * gridDim.x), 1u), kScreenMax);
            w0 = atomicAdd(&L.hdr->warp_work, take);
        }
        w0 = __shfl_sync(kFull, w0, 0);
        take = __shfl_sync(kFull, take, 0);
        if (w0 >= total) break;
        // one lane each: endpoints (Sp_sampler.cpp:46,58-60) and the void test
        // (:62-74), and the rows the search starts from
        const uint32_t w = w0 + lane;
        uint32_t u = 0, v = 0, d = 0, seg = 0, sl = 0;
        uint2 row_u = make_uint2(0u, 0u), row_v = row_u;
        bool live = lane < take && w < total;
        if (live) {
            seg = segment_of(L.segs, nsegs, w);
            const SegDesc &A = L.segs[seg];
            sl = w - A.base;
            const uint32_t gidx = A.first_sample + sl;
            v = draw32(A.seed, gidx, d++) % A.n;
            u = draw32(A.seed, gidx, d++) % A.n;
            while (u == v) v = draw32(A.seed, gidx, d++) % A.n;
            const uint32_t cu = __ldg(&A.cc[u]), cv = __ldg(&A.cc[v]);
            if (A.directed ? cu < cv : cu != cv) {
                A.out_pl[sl] = 0;
                A.out_np[sl] = 0;
                A.out_vis[sl] = 0;
                A.out_status[sl] = 0;
                A.out_ball[sl] = 0;
                A.out_pred[sl] = 0;
                live = false;
            } else {
                row_u = __ldg(&A.out_rows[u]);
                row_v = __ldg(&A.in_rows[v]);
            }
        }
        __syncwarp();
        uint32_t todo = __ballot_sync(kFull, live);
        while (todo) {
            const int i = __ffs(todo) - 1;
            todo &= todo - 1u;
            const SegDesc &A = L.segs[__shfl_sync(kFull, seg, i)];
            const uint2 ru = make_uint2(__shfl_sync(kFull, row_u.x, i),
                                        __shfl_sync(kFull, row_u.y, i));
            const uint2 rv = make_uint2(__shfl_sync(kFull, row_v.x, i),
                                        __shfl_sync(kFull, row_v.y, i));
            const uint32_t si = __shfl_sync(kFull, sl, i);
            // a graph that is not tried is one whose samples are long: listed first
            uint32_t wide = 0xffffffffu;
            const bool done =
                (A.compact & kCompactOn) != 0u &&
                draw_sample(A, s, W, si, __shfl_sync(kFull, u, i), __shfl_sync(kFull, v, i),
                            __shfl_sync(kFull, d, i), ru, rv, wide);
            if (!done && lane == 0) {
                // by the larger frontier when the search was given up
                const uint32_t c = wide >= 16384u ? 0u : wide >= 4096u ? 1u : wide >= 1024u ? 2u : 3u;
                L.list[(uint64_t)c * L.list_cap + atomicAdd(&L.hdr->todo[c], 1u)] =
                    w0 + (uint32_t)i;
                if (A.left) atomicAdd(A.left, 1ull);
            }
            __syncwarp();
        }
    }
    if (lane == 0) atomicAdd(&L.hdr->warp_cycles, (unsigned long long)(clock64() - t0));
}

}  // namespace

cudaError_t warp_sampler_launch(const WarpLaunch &L, uint32_t grid, cudaStream_t stream) {
    if (grid == 0) return cudaSuccess;
    warp_sampler_kernel<<<grid, 32, 0, stream>>>(L);
    return cudaGetLastError();
}

int warp_sampler_per_sm() {
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, warp_sampler_kernel, 32, 0);
    return n;
}

}  // namespace silvan
