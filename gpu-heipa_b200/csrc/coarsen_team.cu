// One coarsening level in one launch: the two-hop matching of matching.cu and
// the contraction of contraction.cu run by a team (team.cuh), with the same
// mapping and the same coarse graph (rows in another order, which every
// consumer allows).
//
// What bounds it: on levels of a few dozen to about a million vertices the
// ~45 launches and six host reads of the per-phase path took longer than
// their work (0.32 ms per level of an RGG with 3001 vertices), and inside the
// round loop every phase is a chain of dependent L2 accesses between two
// barriers. Hence:
//  * every warp owns a contiguous vertex range and keeps its unmatched
//    vertices, their targets and states in a list of its own (shared memory
//    when short), so a commit sub-round reads one word of another vertex;
//  * the re-pick of a round also marks the receivers of the next one: nine
//    barriers per round;
//  * twins, leaves and relatives are grouped without sorting: a hash table (or
//    the vertex id) gives a group its slot, the members are collected per
//    group, and small groups rank their members by counting, large ones over a
//    bitmap of the vertex ids;
//  * a cluster has at most two members, so one scan over the vertices gives
//    coarse ids and row offsets together, and the rows follow in the same
//    launch (8 lanes, a warp or a block per row, hash tables in shared memory).
// Measured (one B200, matching + contraction of all levels of a partition, per-
// phase launches with a single-launch round loop before -> this kernel): RGG
// 3001 vertices 2.3 -> 0.6 ms, grid 256x256 5.4 -> 1.3 ms, RGG 200k 7.9 -> 2.2
// ms; HM of an RGG with 70001 vertices (17 sub-solves) 29 -> 15 ms as a whole.
#include <algorithm>
#include <mutex>
#include <optional>
#include <vector>

#include "coarsen.cuh"
#include "prims.cuh"
#include "team.cuh"

namespace hp {
namespace {

constexpr u32 EMPTY = 0xFFFFFFFFu;
constexpr u32 CT_OWN = 64;            // list entries of a warp in shared memory (vertex ranges up to this)
constexpr u32 CT_HUB = 1024;          // rows above this length are picked by a whole block
constexpr u32 CT_BIG = 64;            // groups above this size are ranked over a bitmap
constexpr u32 CT_WARP_SLOTS = 512;    // hash slots of a warp (contraction)
constexpr u32 CT_WARP_ROW = 256;      // coarse rows up to this capacity by a warp, longer ones by a block
constexpr u32 CT_MAX_ROUNDS = 100000;
constexpr u32 RECEIVER = SENTINEL - 1;  // vcmap: unmatched, takes offers in this sub-round
constexpr u32 HUB_PICK = SENTINEL - 2;  // list target: being picked by a block

enum { CC_ACTIVE = 0, CC_HUB = 2, CC_OPEN = 4, CC_ALLOC = 8, CC_BIG = 12, CC_ROWS = 16, CC_N = 20 };

struct CoarsenOut {
    unsigned long long m;  // coarse entries
    u32 n;                 // coarse vertices
    u32 err;
    u32 rounds;
    u32 too_long;          // a coarse row exceeds the block table: the rows were not built
    unsigned long long contract_ns;  // time from the coarse ids on
};

struct CoarsenArgs {
    u32 n;
    const u32 *rowptr, *rowlen, *adj;
    const s32 *ew, *vw;         // null: unit weights
    u32 *vcmap;                 // leader (smaller id) of a matched vertex, RECEIVER or SENTINEL
    u32 *mate;                  // partner of a leader
    u32 *ul, *hl, *sl;          // the warps' lists: vertex, target, state
    unsigned long long *table;  // 2n words: offers (first n) during the rounds, then the digest table
    u32 *cnt, *off;             // 2n + 1 words each: group sizes and member offsets
    u32 *hubs;                  // long rows; large groups; long coarse rows
    u32 *picked;                // targets of long rows
    u32 *mapping;
    u32 contract;               // build the coarse graph too
    u32 *c_rowptr, *c_rowlen;
    s32 *c_vw;
    u32 *c_adj;
    s32 *c_ew;
    unsigned long long *btot;   // per block: (leaders << 32) + capacity
    u32 *ctr;                   // CC_N counters, zero on entry
    u32 *bar;                   // zero on entry
    CoarsenOut *out;            // zero on entry
    u32 seed;
};

__device__ __forceinline__ bool receives(u32 u, u32 v, u32 r) {
    return r > 0 ? !(murmur3_u32(u + r) < murmur3_u32(v + r)) : !(u < v);
}

struct Best {
    unsigned long long key;
    u32 v;
};

// Heaviest eligible neighbour, ties by xorshift (pick_neighbor :102-188); the
// shift values of different neighbours differ. Coarse weights are sums modulo
// 2^32: rows of up to THREAD_DEG_MAX entries start from weight 0 and never take
// a negative one, longer ones take any but the smallest (as matching.cu).
template<bool INITIAL>
struct PickOp {
    u32 seed;
    __device__ __forceinline__ Best init() const { return Best{0, SENTINEL}; }
    __device__ __forceinline__ u32 gather(const CoarsenArgs &a, u32 v) const {
        return INITIAL ? SENTINEL : __ldcg(&a.vcmap[v]);
    }
    __device__ __forceinline__ void add(Best &s, u32 u, u32 len, u32 v, s32 w, u32 x) const {
        if (x < RECEIVER || w < (len <= THREAD_DEG_MAX ? 0 : -INT32_MAX)) return;  // matched, or too light
        const unsigned long long key =
            ((unsigned long long) ((u32) w ^ 0x80000000u) << 32) | xorshift32(v + xorshift32(u ^ seed));
        if (key > s.key) s = Best{key, v};
    }
    __device__ __forceinline__ void merge(Best &s, const Best &y) const {
        if (y.key > s.key) s = y;
    }
};

// Sum over the neighbours of h + h^2 (:454-466).
struct TwinOp {
    __device__ __forceinline__ Best init() const { return Best{0, 0}; }
    __device__ __forceinline__ u32 gather(const CoarsenArgs &, u32) const { return 0; }
    __device__ __forceinline__ void add(Best &s, u32, u32, u32 v, s32, u32) const {
        const unsigned long long y = murmur3_u32(v);
        s.key += y * y + y;
    }
    __device__ __forceinline__ void merge(Best &s, const Best &y) const { s.key += y.key; }
};

// Neighbour of minimum degree, then maximum weight, then lowest id (:545-565).
struct RelOp {
    __device__ __forceinline__ Best init() const { return Best{~0ull, SENTINEL}; }
    __device__ __forceinline__ u32 gather(const CoarsenArgs &a, u32 v) const { return __ldg(&a.rowlen[v]); }
    __device__ __forceinline__ void add(Best &s, u32, u32, u32 v, s32 w, u32 d) const {
        merge(s, Best{((unsigned long long) d << 32) | (u32) (INT32_MAX - w), v});
    }
    __device__ __forceinline__ void merge(Best &s, const Best &y) const {
        if (y.key < s.key || (y.key == s.key && y.v < s.v)) s = y;
    }
};

// Share of a row: entries first, first + step, ...
template<class Op>
__device__ __forceinline__ Best row_share(const CoarsenArgs &a, const Op &op, u32 u, u32 beg, u32 len, u32 first,
                                          u32 step) {
    Best s = op.init();
    for (u32 t0 = first; t0 < len; t0 += 4 * step) {
        u32 v[4], x[4];
        s32 w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const u32 t = t0 + j * step;
            v[j] = t < len ? __ldg(&a.adj[(u64) beg + t]) : SENTINEL;
            w[j] = t < len ? (a.ew ? __ldg(&a.ew[(u64) beg + t]) : 1) : 0;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) x[j] = v[j] != SENTINEL ? op.gather(a, v[j]) : 0;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (v[j] != SENTINEL) op.add(s, u, len, v[j], w[j], x[j]);
    }
    return s;
}

template<class Op, int GL>
__device__ __forceinline__ void row_merge(const Op &op, Best &s) {
#pragma unroll
    for (int d = GL / 2; d > 0; d >>= 1) {
        const Best y{__shfl_xor_sync(FULL, s.key, d), __shfl_xor_sync(FULL, s.v, d)};
        op.merge(s, y);
    }
}

// Evaluates the rows of the lanes in `need` (u, beg, len of each lane): rows
// of up to 32 entries four at a time by 8 lanes each, longer ones by the warp.
// Every lane receives its row's result. All lanes of the warp call this.
template<class Op>
__device__ __forceinline__ void rows_eval(const CoarsenArgs &a, const Op &op, bool need, u32 u, u32 beg, u32 len,
                                          Best &out) {
    const u32 lane = lane_id(), g = lane >> 3, gl = lane & 7;
    u32 m = __ballot_sync(FULL, need && len <= 32);
    while (m) {
        u32 mine = m, rest = m;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (i < (int) g) mine &= mine - 1;
            rest &= rest - 1;
        }
        const int src = mine ? __ffs(mine) - 1 : 0;
        const u32 ru = __shfl_sync(FULL, u, src), rb = __shfl_sync(FULL, beg, src);
        u32 rl = __shfl_sync(FULL, len, src);
        if (!mine) rl = 0;
        Best s = row_share(a, op, ru, rb, rl, gl, 8);
        __syncwarp();
        row_merge<Op, 8>(op, s);
        const u32 rank = __popc(m & ((1u << lane) - 1u));
        const bool take = (m >> lane & 1u) && rank < 4;
        const int from = (take ? rank : 0) * 8;
        const Best r{__shfl_sync(FULL, s.key, from), __shfl_sync(FULL, s.v, from)};
        if (take) out = r;
        m = rest;
    }
    m = __ballot_sync(FULL, need && len > 32);
    while (m) {
        const int src = __ffs(m) - 1;
        m &= m - 1;
        const u32 ru = __shfl_sync(FULL, u, src), rb = __shfl_sync(FULL, beg, src), rl = __shfl_sync(FULL, len, src);
        Best s = row_share(a, op, ru, rb, rl, lane, 32);
        __syncwarp();
        row_merge<Op, 32>(op, s);
        if ((int) lane == src) out = s;
    }
}

// Rows of a.hubs[0, count) by whole blocks; the picks go to a.picked.
template<class Op>
__device__ __forceinline__ void hubs_pick(const CoarsenArgs &a, const Op &op, u32 count, Best *sm) {
    for (u32 i = blockIdx.x; i < count; i += gridDim.x) {
        const u32 u = a.hubs[i];
        Best s = row_share(a, op, u, __ldg(&a.rowptr[u]), __ldg(&a.rowlen[u]), threadIdx.x, blockDim.x);
        __syncwarp();
        row_merge<Op, 32>(op, s);
        if (lane_id() == 0) sm[warp_in_block()] = s;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (u32 w = 1; w < (blockDim.x >> 5); ++w) op.merge(s, sm[w]);
            a.picked[u] = s.v;
        }
        __syncthreads();
    }
}

// Adds the block's total of a per-warp value (lane 0's) to *dst.
__device__ __forceinline__ void block_add_u32(u32 v, u32 *dst, u32 *sm) {
    if (lane_id() == 0) sm[warp_in_block()] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        u32 t = 0;
        for (u32 w = 0; w < (blockDim.x >> 5); ++w) t += sm[w];
        if (t) atomicAdd(dst, t);
    }
}

__device__ __forceinline__ u32 ct_slot(u32 key, u32 bits) { return (key * 2654435761u) >> (32 - bits); }

// Inserts (cv, w) into an open-addressing table of mask + 1 slots.
__device__ __forceinline__ void ct_insert(u32 *tk, s32 *tw, u32 mask, u32 h, u32 cv, s32 w, u32 *err) {
    for (u32 probe = 0; probe <= mask; ++probe) {
        const u32 prev = atomicCAS(&tk[h], EMPTY, cv);
        if (prev == EMPTY || prev == cv) {
            atomicAdd(&tw[h], w);
            return;
        }
        h = (h + 1) & mask;
    }
    set_error(err, DEV_ERR_HASH_FULL);
}

// Inserts entries first, first + step, ... of the rows (b0, l0) and (b1, cap -
// l0), without self loops of coarse vertex c, into a hash table.
__device__ __forceinline__ void ct_add(const CoarsenArgs &a, u32 c, u32 b0, u32 l0, u32 b1, u32 cap, u32 first, u32 step,
                                       u32 *tk, s32 *tw, u32 bits) {
    for (u32 t0 = first; t0 < cap; t0 += 4 * step) {
        u32 cv[4];
        s32 w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const u32 t = t0 + j * step;
            cv[j] = EMPTY;
            w[j] = 0;
            if (t < cap) {
                const u64 e = t < l0 ? (u64) b0 + t : (u64) b1 + (t - l0);
                cv[j] = __ldg(&a.adj[e]);
                w[j] = a.ew ? __ldg(&a.ew[e]) : 1;
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (cv[j] != EMPTY) cv[j] = __ldcg(&a.mapping[cv[j]]);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (cv[j] != EMPTY && cv[j] != c)
                ct_insert(tk, tw, (1u << bits) - 1u, ct_slot(cv[j], bits), cv[j], w[j], &a.out->err);
    }
}

#define TEAM_SYNC()                                                          \
    do {                                                                     \
        if (!team_barrier<TEAM>(a.bar, bar_target, &a.out->err)) return;     \
    } while (0)

// Dynamic shared memory: the warps' hash tables (keys of all warps, then
// weights) and lists; the large-group bitmap overlays the tables.
inline size_t coarsen_smem(u32 warps) { return (size_t) warps * (CT_WARP_SLOTS * 8 + 3 * CT_OWN * 4); }

template<int TEAM>
__global__ void __launch_bounds__(1024, 1) k_coarsen_team(const __grid_constant__ CoarsenArgs a) {
    extern __shared__ __align__(16) u32 ct_dsm[];
    __shared__ u32 su[33];
    __shared__ unsigned long long sl[33];
    __shared__ Best sb[32];
    const u32 tid = threadIdx.x, lane = lane_id(), warp = warp_in_block(), nw = blockDim.x >> 5;
    const u32 n = a.n, G = gridDim.x, lt = (1u << lane) - 1u, g = lane >> 3, gl = lane & 7;
    u32 *const tk_all = ct_dsm;
    s32 *const tw_all = (s32 *) (ct_dsm + nw * CT_WARP_SLOTS);
    u32 bar_target = 0;
    const u32 gwarps = G * nw, gw = blockIdx.x * nw + warp;
    const u32 per = (n + gwarps - 1) / gwarps;
    const u32 r0 = (u32) min((u64) n, (u64) gw * per), r1 = (u32) min((u64) n, (u64) r0 + per);
    const bool small = per <= CT_OWN;
    u32 *const own = ct_dsm + nw * CT_WARP_SLOTS * 2 + warp * 3 * CT_OWN;
    u32 *const ul = small ? own : a.ul + r0;
    u32 *const hl = small ? own + CT_OWN : a.hl + r0;
    u32 *const sl_ = small ? own + 2 * CT_OWN : a.sl + r0;
    u32 na = 0;  // entries of this warp's list

    // Fixes the targets picked by blocks and marks the receivers of sub-round 0.
    auto finish_hubs = [&]() {
        u32 kept = 0;
        for (u32 base = 0; base < na; base += 32) {
            const u32 i = base + lane;
            u32 u = 0, h = SENTINEL, st = SENTINEL;
            if (i < na) {
                u = ul[i];
                h = hl[i];
                st = sl_[i];
                if (h == HUB_PICK) {
                    h = __ldcg(&a.picked[u]);
                    if (h != SENTINEL && receives(u, h, 0)) {
                        st = RECEIVER;
                        a.vcmap[u] = RECEIVER;
                    }
                }
            }
            __syncwarp();
            const bool keep = i < na && h != SENTINEL;
            const u32 mask = __ballot_sync(FULL, keep);
            if (keep) {
                const u32 p = kept + __popc(mask & lt);
                ul[p] = u;
                hl[p] = h;
                sl_[p] = st;
            }
            kept += __popc(mask);
            __syncwarp();
        }
        na = kept;
    };

    // initial picks (:255-308)
    {
        const PickOp<true> op{a.seed};
        for (u32 base = r0; base < r1; base += 32) {
            const u32 u = base + lane;
            const bool act = u < r1;
            u32 beg = 0, len = 0, h = SENTINEL;
            if (act) {
                beg = __ldg(&a.rowptr[u]);
                len = __ldg(&a.rowlen[u]);
                a.mate[u] = SENTINEL;
                a.table[u] = ~0ull;
                if (!a.ew && len) h = __ldg(&a.adj[(u64) beg + (xorshift32(u ^ a.seed) % len)]);
            }
            const bool hub = act && a.ew && len > CT_HUB;
            if (a.ew) {
                Best s{0, SENTINEL};
                rows_eval(a, op, act && !hub && len > 0, u, beg, len, s);
                h = hub ? HUB_PICK : s.v;
            }
            u32 st = SENTINEL;
            if (act && h < HUB_PICK && receives(u, h, 0)) st = RECEIVER;
            if (act) a.vcmap[u] = st;
            const u32 sh = warp_append(&a.ctr[CC_HUB], hub);
            if (hub) a.hubs[sh] = u;
            const bool keep = act && h != SENTINEL;
            const u32 mask = __ballot_sync(FULL, keep);
            if (keep) {
                const u32 p = na + __popc(mask & lt);
                ul[p] = u;
                hl[p] = h;
                sl_[p] = st;
            }
            na += __popc(mask);
        }
        __syncwarp();
        TEAM_SYNC();
        const u32 nh = ld_fresh<TEAM>(&a.ctr[CC_HUB]);
        if (nh) {
            hubs_pick(a, op, nh, sb);
            TEAM_SYNC();
            finish_hubs();
            TEAM_SYNC();
        }
    }
    // rounds: four commit sub-rounds (:310-332), re-pick (:336-374)
    u32 epoch = 0, round = 0;
    for (;; ++round) {
        if (round >= CT_MAX_ROUNDS) {
            if (tid == 0 && blockIdx.x == 0) set_error(&a.out->err, DEV_ERR_RANGE);
            break;
        }
        u32 *const c_act = &a.ctr[CC_ACTIVE + (round & 1u)], *const c_hub = &a.ctr[CC_HUB + ((round & 1u) ^ 1u)];
        for (u32 r = 0; r < 4; ++r) {
            ++epoch;
            const u32 tag = 0xFFFFFFFFu - epoch;
            for (u32 i = lane; i < na; i += 32) {
                if (sl_[i] != SENTINEL) continue;
                const u32 v = hl[i];
                if (__ldcg(&a.vcmap[v]) == RECEIVER) atomicMin(&a.table[v], ((unsigned long long) tag << 32) | ul[i]);
            }
            TEAM_SYNC();
            if (r == 0 && blockIdx.x == 0 && tid == 0) {
                // the words of the previous round: everyone has read them
                a.ctr[CC_ACTIVE + ((round & 1u) ^ 1u)] = 0;
                a.ctr[CC_HUB + (round & 1u)] = 0;
            }
            for (u32 i = lane; i < na; i += 32) {
                u32 st = sl_[i];
                if (st != RECEIVER && st != SENTINEL) continue;  // matched in this round
                const u32 u = ul[i], v = hl[i];
                if (st == RECEIVER) {
                    const unsigned long long c = __ldcg(&a.table[u]);
                    st = (u32) (c >> 32) == tag ? min(u, (u32) c) : SENTINEL;
                } else {
                    const unsigned long long c = __ldcg(&a.table[v]);
                    if ((u32) (c >> 32) == tag && (u32) c == u) st = min(u, v);
                }
                if (r < 3 && st == SENTINEL && receives(u, v, r + 1)) st = RECEIVER;
                sl_[i] = st;
                a.vcmap[u] = st;
            }
            TEAM_SYNC();
        }
        // re-pick where the target got matched; what stays is compacted, and
        // the receivers of the next round's first sub-round are marked
        // (unmatched: RECEIVER or SENTINEL)
        const PickOp<false> op{a.seed ^ (round * 0x9e3779b1u)};
        u32 kept = 0;
        for (u32 base = 0; base < na; base += 32) {
            const u32 i = base + lane;
            u32 u = 0, h = SENTINEL, st = 0, beg = 0, len = 0;
            if (i < na) {
                u = ul[i];
                h = hl[i];
                st = sl_[i];
            }
            const bool open = i < na && st == SENTINEL;
            const bool again = open && __ldcg(&a.vcmap[h]) < RECEIVER;
            if (again) {
                beg = __ldg(&a.rowptr[u]);
                len = __ldg(&a.rowlen[u]);
            }
            const bool hub = again && len > CT_HUB;
            Best s{0, SENTINEL};
            rows_eval(a, op, again && !hub, u, beg, len, s);
            if (again) h = hub ? HUB_PICK : s.v;
            if (__any_sync(FULL, hub)) {
                const u32 sh = warp_append(c_hub, hub);
                if (hub) a.hubs[sh] = u;
            }
            const bool keep = open && h != SENTINEL;
            if (keep && h < HUB_PICK && receives(u, h, 0)) {
                st = RECEIVER;
                a.vcmap[u] = RECEIVER;
            }
            const u32 mask = __ballot_sync(FULL, keep);
            if (keep) {
                const u32 p = kept + __popc(mask & lt);
                ul[p] = u;
                hl[p] = h;
                sl_[p] = st;
            }
            kept += __popc(mask);
            __syncwarp();
        }
        na = kept;
        block_add_u32(na, c_act, su);
        TEAM_SYNC();
        const u32 left = ld_fresh<TEAM>(c_act), nh = ld_fresh<TEAM>(c_hub);
        if (nh) {
            hubs_pick(a, op, nh, sb);
            TEAM_SYNC();
            finish_hubs();
            TEAM_SYNC();
        }
        if (left == 0) break;
    }
    // leaves (:395-425), twins (:427-524), relatives (:526-571): each while
    // more than a quarter of the vertices is unmatched
    u32 *const slot_of = a.hl, *const members = a.sl;
    for (u32 pass = 0; pass < 4; ++pass) {
        u32 open_cnt = 0;
        for (u32 u = r0 + lane; u < r1; u += 32) open_cnt += a.vcmap[u] >= RECEIVER;
        open_cnt = warp_sum<u32>(open_cnt);
        block_add_u32(open_cnt, &a.ctr[CC_OPEN + pass], su);
        TEAM_SYNC();
        if (pass == 3 || (u64) ld_fresh<TEAM>(&a.ctr[CC_OPEN + pass]) * 4 <= (u64) n) break;
        // empty groups (and digests)
        const u64 gt = (u64) blockIdx.x * blockDim.x + tid, gs = (u64) G * blockDim.x;
        for (u64 i = gt; i < 2 * (u64) n + 1; i += gs) a.cnt[i] = 0;
        if (pass == 1)
            for (u64 i = gt; i < 2 * (u64) n; i += gs) a.table[i] = ~0ull;
        TEAM_SYNC();
        // slot of every candidate's group, group sizes
        for (u32 base = r0; base < r1; base += 32) {
            const u32 u = base + lane;
            const bool open = u < r1 && a.vcmap[u] >= RECEIVER;
            u32 beg = 0, len = 0, slot = EMPTY;
            if (open) {
                beg = __ldg(&a.rowptr[u]);
                len = __ldg(&a.rowlen[u]);
            }
            bool cand = open;
            if (pass == 0) {
                cand = open && len == 1;
                if (cand) slot = __ldg(&a.adj[beg]);
            } else if (pass == 1) {
                Best s{0, 0};
                rows_eval(a, TwinOp{}, open && len > 0, u, beg, len, s);
                if (open) {
                    slot = 2 * n;  // the one digest that marks an empty table word
                    if (s.key != ~0ull) {
                        const unsigned long long x = s.key * 0x9E3779B97F4A7C15ull;
                        u32 h = (u32) (((x >> 32) * (2ull * n)) >> 32);
                        for (u32 probe = 0; probe < 2 * n; ++probe) {
                            const unsigned long long prev = atomicCAS(&a.table[h], ~0ull, s.key);
                            if (prev == ~0ull || prev == s.key) {
                                slot = h;
                                break;
                            }
                            h = h + 1 == 2 * n ? 0 : h + 1;
                        }
                    }
                }
            } else {
                Best s{~0ull, SENTINEL};
                rows_eval(a, RelOp{}, open && len > 0, u, beg, len, s);
                if (open) slot = s.v == SENTINEL ? n : s.v;
            }
            if (open) slot_of[u] = EMPTY;
            if (!__any_sync(FULL, cand)) continue;
            const u32 peers = __match_any_sync(FULL, slot);
            if (cand) {
                // the group's first add owns its set-up in the next step
                bool first = false;
                if ((peers & lt) == 0) first = atomicAdd(&a.cnt[slot], (u32) __popc(peers)) == 0;
                slot_of[u] = slot | (first ? 0x80000000u : 0u);
            }
        }
        TEAM_SYNC();
        for (u32 u = r0 + lane; u < r1; u += 32) {
            if (a.vcmap[u] < RECEIVER) continue;
            const u32 so = slot_of[u];
            if (so == EMPTY || !(so & 0x80000000u)) continue;
            const u32 slot = so & 0x7FFFFFFFu, c = __ldcg(&a.cnt[slot]);
            if (c < 2) continue;
            a.off[slot] = atomicAdd(&a.ctr[CC_ALLOC + pass], c);
            if (c > CT_BIG) a.hubs[atomicAdd(&a.ctr[CC_BIG + pass], 1u)] = slot;
        }
        TEAM_SYNC();
        for (u32 base = r0; base < r1; base += 32) {
            const u32 u = base + lane;
            u32 slot = EMPTY;
            if (u < r1 && a.vcmap[u] >= RECEIVER) {
                slot = slot_of[u];
                if (slot != EMPTY) slot &= 0x7FFFFFFFu;
                if (slot != EMPTY && __ldcg(&a.cnt[slot]) < 2) slot = EMPTY;
            }
            if (!__any_sync(FULL, slot != EMPTY)) continue;
            const u32 peers = __match_any_sync(FULL, slot);
            u32 at = 0;
            if (slot != EMPTY && (peers & lt) == 0) at = atomicAdd(&a.off[slot], (u32) __popc(peers));
            at = __shfl_sync(FULL, at, __ffs(peers) - 1);
            if (slot != EMPTY) members[at + __popc(peers & lt)] = u;
        }
        TEAM_SYNC();
        // ranks 2j and 2j + 1 of a group match (off now points behind it)
        const u32 nbig = ld_fresh<TEAM>(&a.ctr[CC_BIG + pass]);
        for (u32 u = r0 + lane; u < r1; u += 32) {
            if (a.vcmap[u] < RECEIVER) continue;  // (a large group's block may have written it)
            const u32 so = slot_of[u];
            if (so == EMPTY) continue;
            const u32 slot = so & 0x7FFFFFFFu, c = __ldcg(&a.cnt[slot]);
            if (c < 2 || c > CT_BIG) continue;
            const u32 s0 = __ldcg(&a.off[slot]) - c;
            u32 rank = 0, next = SENTINEL;  // of a vertex of even rank: the next larger one
            for (u32 i = 0; i < c; ++i) {
                const u32 x = __ldcg(&members[s0 + i]);
                if (x < u) ++rank;
                else if (x > u && x < next) next = x;
            }
            u32 prev = 0;
            if (rank & 1u) {
                for (u32 i = 0; i < c; ++i) {
                    const u32 x = __ldcg(&members[s0 + i]);
                    if (x < u && x >= prev) prev = x;
                }
                a.vcmap[u] = prev;
            } else if (next != SENTINEL) {
                a.vcmap[u] = u;
            }
        }
        for (u32 i = blockIdx.x; i < nbig; i += G) {
            // large group: its members set bits, every thread walks its words
            __syncthreads();
            u32 *const bits = ct_dsm;
            const u32 words = (n + 31) >> 5, share = (words + blockDim.x - 1) / blockDim.x;
            const u32 slot = __ldcg(&a.hubs[i]), c = __ldcg(&a.cnt[slot]), s0 = __ldcg(&a.off[slot]) - c;
            for (u32 x = tid; x < words; x += blockDim.x) bits[x] = 0;
            __syncthreads();
            for (u32 x = tid; x < c; x += blockDim.x) {
                const u32 u = __ldcg(&members[s0 + x]);
                atomicOr(&bits[u >> 5], 1u << (u & 31));
            }
            __syncthreads();
            const u32 w0 = min(tid * share, words), w1 = min(w0 + share, words);
            u32 sum = 0, last = 0;  // members of this share, id + 1 of the last one
            for (u32 x = w0; x < w1; ++x) {
                const u32 b = bits[x];
                sum += __popc(b);
                if (b) last = x * 32 + 32 - __clz(b);
            }
            u32 tot;
            u32 rank = block_exclusive_scan<u32>(sum, tot, su);
            // last member before this share: running maximum over the threads
            u32 before = last;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const u32 y = __shfl_up_sync(FULL, before, d);
                if ((int) lane >= d) before = max(before, y);
            }
            if (lane == 31) su[warp] = before;
            before = __shfl_up_sync(FULL, before, 1);
            if (lane == 0) before = 0;
            __syncthreads();
            for (u32 w = 0; w < warp; ++w) before = max(before, su[w]);
            for (u32 x = w0; x < w1; ++x) {
                u32 b = bits[x];
                while (b) {
                    const u32 u = x * 32 + __ffs(b) - 1;
                    b &= b - 1;
                    if (rank & 1u) {
                        a.vcmap[before - 1] = before - 1;
                        a.vcmap[u] = before - 1;
                    }
                    before = u + 1;
                    ++rank;
                }
            }
        }
        TEAM_SYNC();
    }
    const unsigned long long t0 = global_ns();
    // coarse ids (:611-641): leaders (unmatched ones lead themselves) in
    // ascending id, and the row capacity of their clusters
    for (u32 u = r0 + lane; u < r1; u += 32) {
        u32 l = a.vcmap[u];
        if (l >= RECEIVER) {
            l = u;
            a.vcmap[u] = u;
        }
        if (l != u) a.mate[l] = u;
    }
    // the tables are empty from here on (the bitmap has used their space)
    __syncthreads();
    for (u32 s = tid; s < nw * CT_WARP_SLOTS; s += blockDim.x) {
        tk_all[s] = EMPTY;
        tw_all[s] = 0;
    }
    TEAM_SYNC();
    unsigned long long mine = 0;
    for (u32 u = r0 + lane; u < r1; u += 32) {
        if (a.vcmap[u] != u) continue;
        const u32 p = __ldcg(&a.mate[u]);
        mine += (1ull << 32) + __ldg(&a.rowlen[u]) + (p != SENTINEL ? __ldg(&a.rowlen[p]) : 0u);
    }
    mine = warp_sum<unsigned long long>(mine);
    if (lane == 0) sl[warp] = mine;
    __syncthreads();
    unsigned long long run = 0;  // before this warp
    for (u32 w = 0; w < warp; ++w) run += sl[w];
    if (tid == 0) {
        unsigned long long t = 0;
        for (u32 w = 0; w < nw; ++w) t += sl[w];
        a.btot[blockIdx.x] = t;
    }
    TEAM_SYNC();
    {
        unsigned long long x = 0;
        for (u32 b = tid; b < blockIdx.x; b += blockDim.x) x += __ldcg(&a.btot[b]);
        x = warp_sum<unsigned long long>(x);
        __syncthreads();
        if (lane == 0) sl[warp] = x;
        __syncthreads();
        for (u32 w = 0; w < nw; ++w) run += sl[w];
    }
    for (u32 base = r0; base < r1; base += 32) {
        const u32 u = base + lane;
        const bool lead = u < r1 && a.vcmap[u] == u;
        u32 p = SENTINEL, cap = 0;
        if (lead) {
            p = __ldcg(&a.mate[u]);
            cap = __ldg(&a.rowlen[u]) + (p != SENTINEL ? __ldg(&a.rowlen[p]) : 0u);
        }
        unsigned long long inc = lead ? (1ull << 32) + cap : 0ull;
        const unsigned long long x = inc;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned long long y = __shfl_up_sync(FULL, inc, d);
            if ((int) lane >= d) inc += y;
        }
        if (lead) {
            const unsigned long long at = run + inc - x;
            const u32 c = (u32) (at >> 32);
            a.mapping[u] = c;
            if (p != SENTINEL) a.mapping[p] = c;
            if (a.contract) {
                a.c_rowptr[c] = (u32) at;
                a.c_vw[c] = wadd(a.vw ? __ldg(&a.vw[u]) : 1, p != SENTINEL ? (a.vw ? __ldg(&a.vw[p]) : 1) : 0);
            }
            if (cap > nw * CT_WARP_SLOTS / 2) a.out->too_long = 1;
        }
        run += __shfl_sync(FULL, inc, 31);
    }
    if (blockIdx.x == G - 1 && warp == nw - 1 && lane == 0) {
        // the last warp's range ends at n or is empty: run is the total
        a.out->n = (u32) (run >> 32);
        a.out->rounds = round + 1;
        if (a.contract) a.c_rowptr[(u32) (run >> 32)] = (u32) run;
    }
    if (!a.contract) return;
    TEAM_SYNC();
    if (ld_fresh<TEAM>(&a.out->too_long)) return;
    // coarse rows: 8 lanes up to 32 entries, a warp up to CT_WARP_ROW, else a block
    unsigned long long msum = 0;
    for (u32 base = r0; base < r1; base += 32) {
        const u32 u = base + lane;
        const bool lead = u < r1 && a.vcmap[u] == u;
        u32 c = 0, b0 = 0, l0 = 0, b1 = 0, cap = 0, at = 0;
        if (lead) {
            c = a.mapping[u];
            b0 = __ldg(&a.rowptr[u]);
            l0 = cap = __ldg(&a.rowlen[u]);
            const u32 p = __ldcg(&a.mate[u]);
            if (p != SENTINEL) {
                b1 = __ldg(&a.rowptr[p]);
                cap += __ldg(&a.rowlen[p]);
            }
            at = a.c_rowptr[c];
        }
        u32 m = __ballot_sync(FULL, lead && cap <= 32);
        while (m) {
            u32 pick = m, rest = m;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (i < (int) g) pick &= pick - 1;
                rest &= rest - 1;
            }
            const int src = pick ? __ffs(pick) - 1 : 0;
            const u32 xc = __shfl_sync(FULL, c, src), x0 = __shfl_sync(FULL, b0, src), xl = __shfl_sync(FULL, l0, src),
                      x1 = __shfl_sync(FULL, b1, src), xa = __shfl_sync(FULL, at, src);
            u32 xcap = __shfl_sync(FULL, cap, src);
            if (!pick) xcap = 0;
            u32 *tk = tk_all + warp * CT_WARP_SLOTS + g * 64;
            s32 *tw = tw_all + warp * CT_WARP_SLOTS + g * 64;
            ct_add(a, xc, x0, xl, x1, xcap, gl, 8, tk, tw, 6);
            __syncwarp();
            u32 cnt = 0;
#pragma unroll
            for (u32 s0 = 0; s0 < 64; s0 += 8) {
                const u32 key = tk[s0 + gl];
                const u32 mask = __ballot_sync(FULL, key != EMPTY) >> (g * 8) & 0xFFu;
                if (key != EMPTY) {
                    const u32 p = xa + cnt + __popc(mask & ((1u << gl) - 1u));
                    a.c_adj[p] = key;
                    a.c_ew[p] = tw[s0 + gl];
                    tk[s0 + gl] = EMPTY;
                    tw[s0 + gl] = 0;
                }
                cnt += __popc(mask);
            }
            if (pick && gl == 0) {
                a.c_rowlen[xc] = cnt;
                msum += cnt;
            }
            __syncwarp();
            m = rest;
        }
        m = __ballot_sync(FULL, lead && cap > 32 && cap <= CT_WARP_ROW);
        while (m) {
            const int src = __ffs(m) - 1;
            m &= m - 1;
            const u32 xc = __shfl_sync(FULL, c, src), x0 = __shfl_sync(FULL, b0, src), xl = __shfl_sync(FULL, l0, src),
                      x1 = __shfl_sync(FULL, b1, src), xa = __shfl_sync(FULL, at, src),
                      xcap = __shfl_sync(FULL, cap, src);
            const u32 bits = 32 - __clz(2 * xcap - 1);  // smallest table of at least twice the capacity
            u32 *tk = tk_all + warp * CT_WARP_SLOTS;
            s32 *tw = tw_all + warp * CT_WARP_SLOTS;
            ct_add(a, xc, x0, xl, x1, xcap, lane, 32, tk, tw, bits);
            __syncwarp();
            u32 cnt = 0;
            for (u32 s0 = 0; s0 < 1u << bits; s0 += 32) {
                const u32 key = tk[s0 + lane];
                const u32 mask = __ballot_sync(FULL, key != EMPTY);
                if (key != EMPTY) {
                    const u32 p = xa + cnt + __popc(mask & lt);
                    a.c_adj[p] = key;
                    a.c_ew[p] = tw[s0 + lane];
                    tk[s0 + lane] = EMPTY;
                    tw[s0 + lane] = 0;
                }
                cnt += __popc(mask);
            }
            if (lane == 0) {
                a.c_rowlen[xc] = cnt;
                msum += cnt;
            }
            __syncwarp();
        }
        const bool lng = lead && cap > CT_WARP_ROW;
        if (__any_sync(FULL, lng)) {
            const u32 s = warp_append(&a.ctr[CC_ROWS], lng);
            if (lng) a.hubs[s] = u;
        }
    }
    TEAM_SYNC();
    const u32 nl = ld_fresh<TEAM>(&a.ctr[CC_ROWS]);
    for (u32 i = blockIdx.x; i < nl; i += G) {
        const u32 u = __ldcg(&a.hubs[i]), c = __ldcg(&a.mapping[u]), p = __ldcg(&a.mate[u]);
        const u32 l0 = __ldg(&a.rowlen[u]), cap = l0 + (p != SENTINEL ? __ldg(&a.rowlen[p]) : 0u);
        const u32 bits = 32 - __clz(2 * cap - 1), at = __ldcg(&a.c_rowptr[c]);
        ct_add(a, c, __ldg(&a.rowptr[u]), l0, p != SENTINEL ? __ldg(&a.rowptr[p]) : 0u, cap, tid, blockDim.x, tk_all,
               tw_all, bits);
        __syncthreads();
        u32 cnt = 0;
        for (u32 s = tid; s < 1u << bits; s += blockDim.x) cnt += tk_all[s] != EMPTY;
        u32 tot;
        u32 q = at + block_exclusive_scan<u32>(cnt, tot, su);
        for (u32 s = tid; s < 1u << bits; s += blockDim.x) {
            const u32 key = tk_all[s];
            if (key != EMPTY) {
                a.c_adj[q] = key;
                a.c_ew[q] = tw_all[s];
                ++q;
                tk_all[s] = EMPTY;
                tw_all[s] = 0;
            }
        }
        if (tid == 0) {
            a.c_rowlen[c] = tot;
            msum += tot;
        }
        __syncthreads();
    }
    msum = warp_sum<unsigned long long>(msum);
    if (lane == 0 && msum) atomicAdd(&a.out->m, msum);
    if (blockIdx.x == 0 && tid == 0) a.out->contract_ns = global_ns() - t0;
}

#undef TEAM_SYNC

const void *coarsen_kernel(int team) {
    return team == TEAM_BLOCK ? (const void *) k_coarsen_team<TEAM_BLOCK>
                              : (team == TEAM_CLUSTER ? (const void *) k_coarsen_team<TEAM_CLUSTER>
                                                      : (const void *) k_coarsen_team<TEAM_GRID>);
}

// Per device, once: the kernels' limits; returns the largest cluster.
u32 coarsen_limits(int device) {
    static std::mutex mu;
    static std::vector<std::pair<int, u32> > done;
    std::lock_guard<std::mutex> lock(mu);
    for (const auto &d: done)
        if (d.first == device) return d.second;
    for (int team: {TEAM_BLOCK, TEAM_GRID})
        HP_CUDA(cudaFuncSetAttribute(coarsen_kernel(team), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int) coarsen_smem(team_threads(team) / 32)));
    const u32 best = team_cluster_limit(coarsen_kernel(TEAM_CLUSTER), coarsen_smem(TEAM_CLUSTER_THREADS / 32),
                                        TEAM_CLUSTER_MAX);
    done.emplace_back(device, best);
    return best;
}

} // namespace

// Team of a level (one B200, see coarsen_team): one block, a cluster, a grid.
constexpr u32 COARSEN_BLOCK_MAX_N = 1024;
constexpr u64 COARSEN_BLOCK_MAX_M = 1u << 14;
constexpr u32 COARSEN_CLUSTER_MAX_N = 16384;
constexpr u64 COARSEN_CLUSTER_MAX_M = 1u << 19;
constexpr u32 COARSEN_CLUSTER_ROWS = 64;  // vertices per block of a cluster (up to its largest size)
constexpr u32 COARSEN_GRID_ROWS = 512;    // vertices (or 16 times as many entries) per block of a grid

bool coarsen_team_applies(const Ctx &ctx, const DGraph &g) {
    return g.n >= 2 && g.n <= std::min<u32>(ctx.tune.match_coop_max_n, COARSEN_TEAM_MAX_N) &&
           g.m <= ctx.tune.match_coop_max_m;
}

// Runs the kernel; `rows` (with adj and ew set, capacity g.m) receives the
// coarse graph when given.
CoarsenResult coarsen_team(Ctx &ctx, const DGraph &g, u32 *mapping, DGraph *rows) {
    const u32 n = g.n;
    const u32 max_cluster = coarsen_limits(ctx.device);
    int team = TEAM_GRID;
    u32 blocks = 1;
    if (n <= COARSEN_BLOCK_MAX_N && g.m <= COARSEN_BLOCK_MAX_M) {
        team = TEAM_BLOCK;
    } else if (n <= COARSEN_CLUSTER_MAX_N && g.m <= COARSEN_CLUSTER_MAX_M) {
        team = TEAM_CLUSTER;
        blocks = std::max<u32>(1, std::min<u32>(max_cluster, (n + COARSEN_CLUSTER_ROWS - 1) / COARSEN_CLUSTER_ROWS));
    }
    const u32 threads = team_threads(team);
    const size_t smem = coarsen_smem(threads / 32);
    if (team == TEAM_GRID) {
        blocks = team_grid_blocks(ctx, coarsen_kernel(team), smem,
                                  (std::max<u64>(n, g.m / 16) + COARSEN_GRID_ROWS - 1) / COARSEN_GRID_ROWS);
        if (!blocks) throw CoopSpin{};
    }
    // the large-group bitmap overlays the hash tables
    static_assert((size_t) COARSEN_TEAM_MAX_N / 8 <= (size_t) TEAM_GRID_THREADS / 32 * CT_WARP_SLOTS * 8, "grid bitmap");
    static_assert((size_t) COARSEN_CLUSTER_MAX_N / 8 <= (size_t) TEAM_CLUSTER_THREADS / 32 * CT_WARP_SLOTS * 8 &&
                      COARSEN_BLOCK_MAX_N <= COARSEN_CLUSTER_MAX_N, "cluster and block bitmap");
    CoarsenArgs a{};
    a.n = n;
    a.rowptr = g.rowptr;
    a.rowlen = g.rowlen;
    a.adj = g.adj;
    a.ew = g.ew;
    a.vw = g.vw;
    a.vcmap = ctx.balloc<u32>(n);
    a.mate = ctx.balloc<u32>(n);
    a.ul = ctx.balloc<u32>(n);
    a.hl = ctx.balloc<u32>(n);
    a.sl = ctx.balloc<u32>(n);
    a.table = ctx.balloc<unsigned long long>(2 * (size_t) n);
    a.cnt = ctx.balloc<u32>(2 * (size_t) n + 1);
    a.off = ctx.balloc<u32>(2 * (size_t) n + 1);
    a.hubs = ctx.balloc<u32>(n);
    a.picked = a.off;  // groups come after the rounds
    a.mapping = mapping;
    a.contract = rows != nullptr;
    CoarsenResult r;
    if (rows) {
        // sized for n until the coarse size is known
        a.c_rowptr = r.rowptr = rows->rowptr ? rows->rowptr : ctx.balloc<u32>((size_t) n + 1);
        a.c_rowlen = r.rowlen = rows->rowlen ? rows->rowlen : ctx.balloc<u32>(n);
        a.c_vw = r.vw = rows->vw ? rows->vw : ctx.balloc<s32>(n);
        a.c_adj = rows->adj;
        a.c_ew = rows->ew;
    }
    a.btot = ctx.balloc<unsigned long long>(blocks);
    const size_t zero_bytes = sizeof(CoarsenOut) + (CC_N + 2) * sizeof(u32);
    char *z = ctx.balloc<char>(zero_bytes);
    HP_CUDA(cudaMemsetAsync(z, 0, zero_bytes, ctx.stream));
    a.out = (CoarsenOut *) z;
    a.ctr = (u32 *) (a.out + 1);
    a.bar = a.ctr + CC_N;
    a.seed = MATCH_SEED;
    std::optional<CoopGuard> coop;
    if (team == TEAM_GRID) coop.emplace(ctx.device, ctx.stream, blocks, (u32) ctx.sm_count);
    {
        KernTimer kt(ctx, "k_coarsen_team");
        cudaLaunchAttribute attr;
        const cudaLaunchConfig_t cfg = team_config(blocks, threads, smem, ctx.stream, attr, team);
        void *args[] = {&a};
        HP_CUDA(cudaLaunchKernelExC(&cfg, coarsen_kernel(team), args));
        note_launch();
    }
    static_assert(sizeof(CoarsenOut) <= sizeof(DevStatus), "the outcome is read through the pinned status mirror");
    HP_CUDA(cudaMemcpyAsync(ctx.h_status, a.out, sizeof(CoarsenOut), cudaMemcpyDeviceToHost, ctx.stream));
    ctx.sync();
    const CoarsenOut o = *(const CoarsenOut *) ctx.h_status;
    if ((o.err & DEV_ERR_SPIN) || (ctx.tune.team_give_up & 1u)) throw CoopSpin{};
    if (o.err) throw HpError{HP_ERR_DEVICE, "matching or contraction reported error bits " + std::to_string(o.err)};
    r.contract_ms = (double) o.contract_ns * 1e-6;
    r.n = o.n;
    r.m = o.m;
    r.contracted = rows && !o.too_long;
    return r;
}

} // namespace hp
