// The whole Jet level loop of one level in one launch (included by jet.cu).
//
// A team of blocks runs every iteration of jet_refine: the iteration control
// (ratios, weak / strong switching, best-labelling tracking) and the steps of
// the per-kernel path, with the same result. The team is one block whose
// shared memory holds the level (graph and state) on the smallest levels, a
// thread-block cluster on small levels (hardware barrier, co-scheduled by the
// hardware), or a cooperative grid on larger ones (bounded grid barrier).
//
// What bounds it: the latency of one iteration (levels of a few dozen to a few
// million vertices, tens to hundreds of iterations, everything in L2). A phase
// with little work is a chain of dependent L2 accesses of 0.3 us each, so the
// design minimises barriers and dependent accesses per iteration:
//  * a label-propagation iteration has three barriers: gains and filter, then
//    afterburner and moves, then the objective change. A vertex word holds
//    label, previous label and the iteration that changed it, so moves are
//    applied while other blocks still read the previous labels, and nothing
//    has to be unmarked afterwards;
//  * every warp owns a contiguous vertex range and keeps its candidates and
//    moves in a list of its own: no shared counters, no list lengths to read;
//  * a rebalance iteration sorts nothing. Candidates add their weight to a
//    histogram over the mini-bucket keys; per overloaded block the histogram
//    gives the mini-bucket in which the limit falls, and only the candidates
//    of that one need their order (ascending vertex id): per-warp weight sums
//    over the vertex ranges, prefix sums over them and a prefix within 32
//    vertices. Strong rebalancing needs the exact prefix of every evicted
//    vertex: the few evicted ones are ranked among each other;
//  * rows of up to 32 entries are evaluated by 8 lanes with a block table in
//    shared memory (direct-indexed, or 64 hashed slots for k > 256): an entry
//    costs one add and one exchange, which collects each distinct block once
//    and clears the table; no pass over all k blocks;
//  * long rows are shared by the warps of their block (afterburner, objective
//    change), so that no warp scans a hub row alone.
// Measured (one B200, mean time of one iteration): the levels of an RGG with
// 3001 vertices, 27 us with one 1024-thread block per level in global memory,
// 14 us as cluster teams with shared lists, now 10 us on the levels that fit
// a block team and 12 us as cluster; levels of up to 65536 vertices of a
// 256x256 grid, 62 us as a cooperative grid whose block 0 sorted the
// candidates, now 16 us (all forms); the levels of an R-MAT graph with 65536
// vertices, 280 us (largest two) before, now 60 us (all).
#pragma once

// Rows of up to TEAM_ZERO_ROW entries take a block whose connection is 0 for a
// neighbour, longer ones don't (nor do the per-kernel passes, which keep
// short rows in registers). 16 weights add up to 0 modulo 2^32 only if one of
// them is 2^28 or more, or below 1 (a coarse weight that wrapped): weight - 1
// then has one of the bits from TEAM_ZERO_BIT on.
constexpr u32 TEAM_ZERO_ROW = JT;
constexpr u32 TEAM_ZERO_BIT = 27;
// Tables of rows of up to 32 entries: direct-indexed, direct-indexed with that
// rule (for graphs whose rows can weigh 2^32 or more, DGraph::row_ew: looking
// for such weights costs the others 2%), or hashed, where the rule is free.
enum TeamTable { TAB_DIRECT = 0, TAB_ZERO = 1, TAB_HASH = 2 };
constexpr u32 TEAM_HUB = 1024;         // rows above this length are evaluated by a whole block
constexpr u32 TEAM_LONG = 64;          // afterburner / delta rows above this length take a whole warp ...
constexpr u32 TEAM_SHARE = 256;        // ... and above this one the warps of the block, 128 entries at a time
constexpr u32 TEAM_SHARE_MAX = 128;    // rows a block shares in one phase (others stay with their warp)
constexpr u32 TEAM_DIRECT_K = 256;     // direct-indexed tables per 8 lanes up to this k, hashed ones above
constexpr u32 TEAM_LIST = 128;         // distinct-block list slots per warp (mapping objective; at least k)
constexpr u32 TEAM_OWN = 48;           // candidates / moves of a warp kept in shared memory up to this range
static_assert(2 * TEAM_OWN >= 3 * 32, "the lists' space holds a tile of three words per thread");

enum TeamCnt { TC_HUB = 0, TC_MOVES = 1, TC_FAIL = 2, TC_N = 4 };
enum TeamSum { TS_MOVES = 0, TS_DELTA = 1, TS_N = 2 };  // (moves << 32) + their row entries; objective change
constexpr u32 LOCK_HUB = 2;            // lock word of a hub row that is a candidate of this iteration
constexpr u32 TW_STILL = 0x80000000u;  // stamp flag: in the move list with an unchanged label

// Vertex word: label (16 bits), previous label (16 bits), iteration that
// changed the label (32 bits).
__device__ __forceinline__ u32 tw_label(unsigned long long x) { return (u32) x & 0xFFFFu; }
__device__ __forceinline__ u32 tw_old(unsigned long long x) { return ((u32) x >> 16); }
__device__ __forceinline__ u32 tw_stamp(unsigned long long x) { return (u32) (x >> 32); }

struct TeamCtl {
    u32 n_ratios;
    u32 ratios[17];
    long long obj;   // objective of the input labelling
    s32 maxw;        // its maximum block weight
};

// Outcome, written by the kernel.
struct TeamOut {
    long long obj;   // best objective
    s32 maxw;        // its maximum block weight
    u32 iterations;
    u32 gave_up;     // 1: too many evicted vertices in one step to rank (TeamArgs::rank_pairs), nothing was decided
    u32 err;         // DevErr bits
    u32 hubs;        // some row is longer than TEAM_HUB
    unsigned long long setup_ns;  // time of the set-up (projection, block weights) on block 0
};

struct TeamArgs {
    u32 n;
    const u32 *rowptr, *rowlen;  // block team: rowlen unused, rows are contiguous
    const u32 *adj;
    const s32 *ew, *vw;          // null: unit weights (never null in a block team)
    u32 k;
    s32 lmax;
    s32 opt;
    s32 weak_max, strong_max;
    u32 sections, width;
    u32 promap;
    const u32 *code;
    const s32 *bitdist;
    unsigned long long inval_all_min;
    u32 rank_pairs;             // pairs of evicted vertices that a warp compares at most
    u32 *part;                  // in: labels (unless projected); out: best labelling
    const u32 *cpart, *cmap;    // projection: labels of the coarse vertices, fine -> coarse map (or null)
    u32 *saved;                 // receives a copy of the input labels (or null)
    unsigned long long *tw;     // vertex words
    unsigned long long *abrec;  // afterburner records: gain, target (16 bits), label (16 bits)
    u32 *dest_cache;
    s32 *gain_cache;
    u32 *lock;
    u32 *dest;                  // rebalance targets
    u32 *keys;                  // mini-bucket keys
    u32 *clist, *mlist;         // candidates and moves of each warp, from the start of its vertex range
    u32 *hubs, *fails;          // long rows of a pass; evicted vertices that need a fallback slot
    unsigned long long *mcomp;  // strong: (key, vertex) of every evicted vertex
    unsigned long long *mow;    // strong: (block, vertex weight)
    s32 *bw;                    // zero on entry
    u32 *hist;                  // k * width + 2 weights, zero on entry
    s32 *tsum;                  // k * blocks
    s32 *ea;                    // k
    u32 *cnt;                   // 2 sets of TC_N counters, zero on entry
    long long *sum;             // 2 sets of TS_N sums, zero on entry
    u32 *bar;                   // grid barrier word, zero on entry
    TeamOut *out;  // zero on entry
};

// Shared-memory arrays (dynamic): per warp the block tables, then k-word
// arrays of the block.
struct TeamSm {
    s32 *tab;      // this warp's tables
    s32 *tab0;     // the block's first table
    u32 stride;    // words between the tables of two warps
    unsigned long long *list;  // this warp's distinct-block list (mapping objective)
    u32 *own;      // this warp's candidate and move lists (2 * TEAM_OWN) ...
    u32 *own0;     // ... and the block's first
    s32 *bw, *bd, *cutbase, *tot, *spill, *toff;
    u32 *under, *olist, *cutkey;
    long long *es, *pre;
    u32 *code;
    s32 *dist;
};

// vertex words 8, records (or targets and keys) 8, evicted 16, row offset,
// weight, cached target, cached gain, lock, two lists 4 each
constexpr size_t TEAM_VERTEX_BYTES = 8 + 8 + 16 + 7 * 4;

// Bytes of dynamic shared memory of a team block of `warps` warps.
__host__ __device__ inline u32 team_stride(u32 k) { return k <= TEAM_DIRECT_K ? 4 * k : (k < 512 ? 512 : k); }

inline size_t team_smem(u32 k, u32 warps, bool promap) {
    size_t b = (size_t) warps * team_stride(k) * 4;
    b = (b + 15) & ~(size_t) 15;
    if (promap) b += (size_t) warps * std::max<u32>(TEAM_LIST, k) * 8;
    b += ((size_t) k + 2) * 8 * 2 + (size_t) k * 4 * 10 + 32 * 4 + (size_t) warps * 2 * TEAM_OWN * 4;
    return (b + 15) & ~(size_t) 15;
}

// Bytes of a level (graph, state, bins) in the shared memory of a block team.
inline size_t team_level_smem(u32 n, u64 m, u32 k, u32 width) {
    return (size_t) n * TEAM_VERTEX_BYTES + m * 8 + ((size_t) k * width + 2) * 4 + 64 +
           (2 * TS_N) * 8 + (2 * TC_N + k + k) * 4 + 64;
}

__device__ __forceinline__ TeamSm team_carve(unsigned char *base, u32 k, u32 warps, u32 warp, bool promap) {
    TeamSm S;
    S.stride = team_stride(k);
    S.tab0 = (s32 *) base;
    S.tab = S.tab0 + warp * S.stride;
    size_t off = ((size_t) warps * S.stride * 4 + 15) & ~(size_t) 15;
    const u32 ln = k > TEAM_LIST ? k : TEAM_LIST;
    S.list = nullptr;
    if (promap) {
        S.list = (unsigned long long *) (base + off) + (size_t) warp * ln;
        off += (size_t) warps * ln * 8;
    }
    S.es = (long long *) (base + off);
    S.pre = S.es + k + 2;
    s32 *p = (s32 *) (S.pre + k + 2);
    S.bw = p;
    S.bd = p + k;
    S.cutbase = p + 2 * k;
    S.tot = p + 3 * k;
    S.spill = p + 4 * k;
    S.toff = p + 5 * k;
    S.under = (u32 *) (p + 6 * k);
    S.olist = (u32 *) (p + 7 * k);
    S.cutkey = (u32 *) (p + 8 * k);
    S.code = (u32 *) (p + 9 * k);
    S.dist = p + 10 * k;
    S.own0 = (u32 *) (S.dist + 32);
    S.own = S.own0 + warp * 2 * TEAM_OWN;
    return S;
}

// Graph reads: the level is in shared memory (block team) or constant in
// global memory.
template<int TEAM, typename T>
__device__ __forceinline__ T ld_graph(const T *p) {
    return TEAM == TEAM_BLOCK ? *p : __ldg(p);
}
template<int TEAM>
__device__ __forceinline__ s32 ld_ew(const TeamArgs &a, u64 e) {
    return TEAM == TEAM_BLOCK ? a.ew[e] : (a.ew ? __ldg(&a.ew[e]) : 1);
}
template<int TEAM>
__device__ __forceinline__ s32 ld_vw(const TeamArgs &a, u32 u) {
    return TEAM == TEAM_BLOCK ? a.vw[u] : (a.vw ? __ldg(&a.vw[u]) : 1);
}
template<int TEAM>
__device__ __forceinline__ void ld_row(const TeamArgs &a, u32 u, u32 &beg, u32 &len) {
    beg = ld_graph<TEAM>(&a.rowptr[u]);
    len = TEAM == TEAM_BLOCK ? a.rowptr[u + 1] - beg : __ldg(&a.rowlen[u]);
}
// ---- row evaluation --------------------------------------------------------------------

enum TeamOp { OP_CUT = 0, OP_MAP = 1, OP_WEAK = 2, OP_STRONG = 3 };

struct RowOut {
    unsigned long long bk;  // best block key
    s32 own;                // connection to the own block
    s32 sum, count;         // strong: connection to and number of the eligible blocks
};

__device__ __forceinline__ s32 team_dist(const TeamSm &S, u32 x, u32 y) {
    if (x == y) return 0;
    return S.dist[31 - __clz(S.code[x] ^ S.code[y])];
}

// One distinct neighbour block b with connection c of a row of block o.
template<int OP>
__device__ __forceinline__ void row_take(const TeamSm &S, u32 o, s32 max_b_w, u32 b, s32 c, RowOut &r) {
    if (b == o) {
        r.own = c;
        return;
    }
    if (OP == OP_STRONG) {
        if (S.bw[b] < max_b_w) {
            r.sum = wadd(r.sum, c);
            ++r.count;
        }
    } else if (OP == OP_CUT || S.bw[b] < max_b_w) {
        const unsigned long long key = cut_key(c, b);
        r.bk = key > r.bk ? key : r.bk;
    }
}

// Mapping objective: scores the distinct blocks list[0, cnt) (block in the
// high word, connection in the low word) of a row of block o; lanes first,
// first + step, ... of the list.
__device__ __forceinline__ void row_score(const TeamSm &S, const unsigned long long *list, u32 cnt, u32 o, u32 first,
                                          u32 step, RowOut &r) {
    for (u32 i = first; i < cnt; i += step) {
        const u32 b = (u32) (list[i] >> 32);
        if (b == o) continue;
        s32 d = 0;
        for (u32 t = 0; t < cnt; ++t) {
            const unsigned long long e = list[t];
            const u32 id = (u32) (e >> 32);
            d = wadd(d, wmul((s32) (u32) e, wsub(team_dist(S, o, id), team_dist(S, b, id))));
        }
        const unsigned long long key = delta_key(d, b);
        r.bk = key > r.bk ? key : r.bk;
    }
}

// Reduces a row result over groups of GL lanes (every lane of a group
// receives it).
template<int OP, int GL>
__device__ __forceinline__ void row_reduce(RowOut &r) {
#pragma unroll
    for (int d = GL / 2; d > 0; d >>= 1) {
        if (OP != OP_MAP) r.own += __shfl_xor_sync(FULL, r.own, d);  // one lane holds it
        if (OP == OP_STRONG) {
            r.sum = wadd(r.sum, __shfl_xor_sync(FULL, r.sum, d));
            r.count += __shfl_xor_sync(FULL, r.count, d);
        } else {
            const unsigned long long y = __shfl_xor_sync(FULL, r.bk, d);
            r.bk = y > r.bk ? y : r.bk;
        }
    }
}

__device__ __forceinline__ u32 label_of(const TeamArgs &a, u32 v) { return ((const u32 *) a.tw)[2 * (u64) v] & 0xFFFFu; }

// Evaluates the rows of the lanes in `need` (beg, len <= 32, own block o of
// each lane's row), four rows at a time, 8 lanes per row; every lane receives
// its row's result. TAB_HASH: 64 slots of (block + 1, connection) per row instead
// of a direct-indexed table; both are all zero between rows. All lanes of the
// warp call this.
template<int TEAM, int OP, int TAB>
__device__ __forceinline__ void rows_short(const TeamArgs &a, const TeamSm &S, u32 need, u32 beg, u32 len, u32 o,
                                           s32 max_b_w, RowOut &out) {
    constexpr int NG = 4, GL = 8;
    constexpr bool HASH = TAB == TAB_HASH;
    const u32 lane = lane_id(), g = lane / GL, gl = lane % GL;
    s32 *tv = S.tab + g * (HASH ? 128 : a.k);
    while (need) {
        u32 m = need, rest = need;
#pragma unroll
        for (int i = 0; i < NG; ++i) {
            if (i < (int) g) m &= m - 1;
            rest &= rest - 1;
        }
        const int src = m ? __ffs(m) - 1 : 0;
        const u32 rb = __shfl_sync(FULL, beg, src);
        u32 rl = __shfl_sync(FULL, len, src);
        const u32 ro = __shfl_sync(FULL, o, src);
        if (!m) rl = 0;
        u32 b[4];
        s32 w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const u32 t = gl + j * GL;
            b[j] = t < rl ? ld_graph<TEAM>(&a.adj[(u64) rb + t]) : EMPTY;
            w[j] = t < rl ? ld_ew<TEAM>(a, (u64) rb + t) : 0;
        }
        u32 bits = 0;
        if (TAB == TAB_ZERO)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (b[j] != EMPTY) bits |= (u32) w[j] - 1u;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (b[j] != EMPTY) b[j] = label_of(a, b[j]);
        u32 at[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            at[j] = b[j];
            if (HASH && b[j] != EMPTY) {  // at most 32 keys in 64 slots
                const u32 h0 = (b[j] * 2654435761u) >> 26;
                u32 h = h0;
                for (;;) {
                    const u32 prev = atomicCAS((u32 *) &tv[h], 0u, b[j] + 1);
                    if (prev == 0 || prev == b[j] + 1) break;
                    h = (h + 1) & 63u;
                    if (h == h0) {  // all slots seen
                        set_error(&a.out->err, DEV_ERR_HASH_FULL);
                        break;
                    }
                }
                at[j] = 64 + h;
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (b[j] != EMPTY) atomicAdd(&tv[at[j]], w[j]);
        __syncwarp();
        // an exchange returns a block's connection to one of its entries and
        // clears the table; of a hashed table it takes the key, because a
        // connection can be 0 (weights are added modulo 2^32) and a key that
        // stayed behind would fill the table for the rows that follow
        bool rep[4];  // the entry stands for its block
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (!HASH) {
                w[j] = b[j] != EMPTY ? atomicExch(&tv[at[j]], 0) : 0;
                rep[j] = w[j] != 0;
            } else {
                // (only the entry that takes the key uses what it read)
                if (b[j] != EMPTY) w[j] = tv[at[j]];
                rep[j] = b[j] != EMPTY && atomicExch(&tv[at[j] - 64], 0) != 0;
                if (rep[j]) tv[at[j]] = 0;
                rep[j] = rep[j] && (w[j] != 0 || rl <= TEAM_ZERO_ROW);
            }
        }
        if (TAB == TAB_ZERO && __any_sync(FULL, bits >> TEAM_ZERO_BIT)) {
            // the blocks with a connection are marked, and of
            // the others the first exchange stands for its block
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (rep[j]) tv[at[j]] = 1;
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (b[j] != EMPTY && !rep[j] && rl <= TEAM_ZERO_ROW) rep[j] = atomicExch(&tv[at[j]], 1) == 0;
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (b[j] != EMPTY) tv[at[j]] = 0;
        }
        __syncwarp();
        RowOut r{0, 0, 0, 0};
        if (OP == OP_MAP) {
            unsigned long long *list = S.list + g * (4 * GL);
            u32 cnt = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const u32 mask = (__ballot_sync(FULL, rep[j]) >> (g * GL)) & 0xFFu;
                if (rep[j]) list[cnt + __popc(mask & ((1u << gl) - 1u))] = ((unsigned long long) b[j] << 32) | (u32) w[j];
                cnt += __popc(mask);
            }
            __syncwarp();
            row_score(S, list, cnt, ro, gl, GL, r);
            __syncwarp();
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (rep[j]) row_take<OP>(S, ro, max_b_w, b[j], w[j], r);
        }
        row_reduce<OP, GL>(r);
        // back to the lanes that own the rows
        const u32 rank = __popc(need & ((1u << lane) - 1u));
        const bool mine = (need >> lane & 1u) && rank < (u32) NG;
        const int from = (mine ? rank : 0) * GL;
        const unsigned long long bk = __shfl_sync(FULL, r.bk, from);
        const s32 own = __shfl_sync(FULL, r.own, from);
        const s32 sum = OP == OP_STRONG ? __shfl_sync(FULL, r.sum, from) : 0;
        const s32 count = OP == OP_STRONG ? __shfl_sync(FULL, r.count, from) : 0;
        if (mine) out = RowOut{bk, own, sum, count};
        need = rest;
    }
}

// Adds entries first, first + step, ... of a row to the direct table tv.
template<int TEAM>
__device__ __forceinline__ void row_add(const TeamArgs &a, u32 beg, u32 len, u32 first, u32 step, s32 *tv) {
    for (u32 t0 = first; t0 < len; t0 += 4 * step) {
        u32 b[4];
        s32 w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const u32 t = t0 + j * step;
            b[j] = t < len ? ld_graph<TEAM>(&a.adj[(u64) beg + t]) : EMPTY;
            w[j] = t < len ? ld_ew<TEAM>(a, (u64) beg + t) : 0;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (b[j] != EMPTY) b[j] = label_of(a, b[j]);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (b[j] != EMPTY) atomicAdd(&tv[b[j]], w[j]);
    }
}

// Result of a filled table (one warp; clears it).
template<int OP>
__device__ __forceinline__ RowOut row_finish(const TeamArgs &a, const TeamSm &S, s32 *tv, u32 o, s32 max_b_w) {
    const u32 lane = lane_id();
    RowOut r{0, 0, 0, 0};
    if (OP == OP_MAP) {
        u32 cnt = 0;
        for (u32 s0 = 0; s0 < a.k; s0 += 32) {
            const u32 s = s0 + lane;
            const s32 c = s < a.k ? tv[s] : 0;
            const u32 mask = __ballot_sync(FULL, c != 0);
            if (c != 0) {
                S.list[cnt + __popc(mask & ((1u << lane) - 1u))] = ((unsigned long long) s << 32) | (u32) c;
                tv[s] = 0;
            }
            cnt += __popc(mask);
        }
        __syncwarp();
        row_score(S, S.list, cnt, o, lane, 32, r);
    } else {
        for (u32 s = lane; s < a.k; s += 32) {
            const s32 c = tv[s];
            if (c != 0) {
                tv[s] = 0;
                row_take<OP>(S, o, max_b_w, s, c, r);
            }
        }
    }
    __syncwarp();
    row_reduce<OP, 32>(r);
    return r;
}

// Evaluates the rows of the lanes in `need`, one at a time by the whole warp.
template<int TEAM, int OP>
__device__ __forceinline__ void rows_long(const TeamArgs &a, const TeamSm &S, u32 need, u32 beg, u32 len, u32 o,
                                          s32 max_b_w, RowOut &out) {
    while (need) {
        const int src = __ffs(need) - 1;
        need &= need - 1;
        const u32 rb = __shfl_sync(FULL, beg, src), rl = __shfl_sync(FULL, len, src), ro = __shfl_sync(FULL, o, src);
        row_add<TEAM>(a, rb, rl, lane_id(), 32, S.tab);
        __syncwarp();
        const RowOut r = row_finish<OP>(a, S, S.tab, ro, max_b_w);
        if (lane_id() == src) out = r;
    }
}

// Target and gain of a row (jet_lp :193-238 / ProMap_jet_lp :219-263).
template<bool MAP>
__device__ __forceinline__ void lp_decide(const RowOut &r, u32 ratio, u32 &best, s32 &gain) {
    best = NO_MOVE;
    gain = 0;
    if (!r.bk) return;
    if (MAP) {
        const s32 d = (s32) ((u32) (r.bk >> 32) ^ 0x80000000u);
        if (d >= 0) {
            best = ~(u32) r.bk;
            gain = d;
        }
    } else {
        const s32 bc = (s32) (u32) (r.bk >> 32);
        if (bc >= r.own || (s64) r.own - (s64) bc < ((s64) ratio * (s64) r.own) / 100) {
            best = ~(u32) r.bk;
            gain = wsub(bc, r.own);
        }
    }
}

// Filter of one vertex (:247-258): its afterburner record; true when it is a
// candidate.
__device__ __forceinline__ bool lp_filter_one(const TeamArgs &a, u32 u, u32 o, u32 dest, s32 gain, u32 lock) {
    const bool c = dest != NO_MOVE && lock == 0;
    if (!c && lock) a.lock[u] = 0;
    a.abrec[u] = (unsigned long long) (u32) (c ? gain : GAIN_MIN) | ((unsigned long long) (dest & 0xFFFFu) << 32) |
                 ((unsigned long long) o << 48);
    return c;
}

// Moves u from ou to nu (perform_moves :753-924).
__device__ __forceinline__ void team_move(const TeamArgs &a, const TeamSm &S, u32 u, u32 ou, u32 nu, s32 vw, u32 stamp) {
    if (ou != nu) {
        atomicSub(&S.bd[ou], vw);
        atomicAdd(&S.bd[nu], vw);
    }
    a.tw[u] = (unsigned long long) nu | ((unsigned long long) ou << 16) |
              ((unsigned long long) (ou != nu ? stamp : stamp | TW_STILL) << 32);
    a.dest_cache[u] = NULL_PART;
}

// Afterburner terms of up to four loaded entries (ab_batch over abrec).
template<int TEAM, bool MAP>
__device__ __forceinline__ s32 team_ab(const TeamArgs &a, const TeamSm &S, u32 u, s32 ug, u32 ou, u32 nu, u32 beg,
                                       u32 len, u32 first, u32 step) {
    s32 change = 0;
    for (u32 t0 = first; t0 < len; t0 += 4 * step) {
        u32 v[4];
        s32 w[4];
        unsigned long long x[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const u32 t = t0 + j * step;
            v[j] = t < len ? ld_graph<TEAM>(&a.adj[(u64) beg + t]) : SENTINEL;
            w[j] = t < len ? ld_ew<TEAM>(a, (u64) beg + t) : 0;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) x[j] = v[j] != SENTINEL ? a.abrec[v[j]] : 0ull;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const s32 vg = (s32) (u32) x[j];
            if (v[j] == SENTINEL || !(vg > ug || (vg == ug && v[j] < u))) continue;
            const u32 nv = (u32) (x[j] >> 32) & 0xFFFFu, ov = (u32) (x[j] >> 48);
            s32 t;
            if (!MAP) {
                t = wmul(w[j], (s32) (nv == nu) - (s32) (nv == ou) + (s32) (ov == ou) - (s32) (ov == nu));
            } else {
                const s32 before_u = wsub(team_dist(S, ou, ov), team_dist(S, nu, ov));
                const s32 after_u = wsub(team_dist(S, ou, nv), team_dist(S, nu, nv));
                t = wmul(w[j], wsub(after_u, before_u));
            }
            change = wadd(change, t);
        }
    }
    return change;
}

// Objective change and cache resets over a moved row (delta_batch).
template<int TEAM, bool MAP>
__device__ __forceinline__ long long team_delta(const TeamArgs &a, const TeamSm &S, u32 ou, u32 nu, bool moved,
                                                u32 stamp, u32 beg, u32 len, u32 first, u32 step, bool inval) {
    long long acc = 0;
    for (u32 t0 = first; t0 < len; t0 += 4 * step) {
        u32 v[4];
        s32 w[4];
        unsigned long long x[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const u32 t = t0 + j * step;
            v[j] = t < len ? ld_graph<TEAM>(&a.adj[(u64) beg + t]) : SENTINEL;
            w[j] = t < len ? ld_ew<TEAM>(a, (u64) beg + t) : 0;
        }
        if (moved) {
#pragma unroll
            for (int j = 0; j < 4; ++j) x[j] = v[j] != SENTINEL ? a.tw[v[j]] : 0ull;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (v[j] == SENTINEL) continue;
                const bool mv = tw_stamp(x[j]) == stamp;
                const u32 nv = tw_label(x[j]), ov = mv ? tw_old(x[j]) : nv;
                long long c;
                if (!MAP) c = (long long) w[j] * ((long long) (nu != nv) - (long long) (ou != ov));
                else c = (long long) w[j] * ((long long) team_dist(S, nu, nv) - (long long) team_dist(S, ou, ov));
                acc += mv ? c : 2 * c;
            }
        }
        if (inval) {
            // only where a target is cached: most neighbours have been reset
            // already, and a cached read is cheaper than a scattered store
            u32 x[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) x[j] = v[j] != SENTINEL ? a.dest_cache[v[j]] : NULL_PART;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (x[j] != NULL_PART) a.dest_cache[v[j]] = NULL_PART;
        }
    }
    return acc;
}

// Exclusive prefix (p) and total (t) of v over the lanes of `mask` (this
// lane's peers). All lanes of the warp call this.
__device__ __forceinline__ void peer_prefix(u32 mask, s32 v, s32 &p, s32 &t) {
    const u32 lane = lane_id();
    p = 0;
    t = 0;
#pragma unroll
    for (u32 i = 0; i < 32; ++i) {
        const s32 x = __shfl_sync(FULL, v, i);
        if (mask >> i & 1u) {
            t += x;
            if (i < lane) p += x;
        }
    }
}

// Weight of overloaded block o above the limit (all weights together fit 31
// bits, so a limit far below zero may be cut off there).
__device__ __forceinline__ s32 excess_of(const TeamArgs &a, const TeamSm &S, u32 o) {
    const s64 x = (s64) S.bw[o] - (s64) a.lmax;
    return x > INT32_MAX ? INT32_MAX : (s32) x;
}

// Adds v over all threads to *slot with one atomic per block. No block
// barrier follows: the team barrier does.
__device__ __forceinline__ void team_add(long long v, long long *slot, long long *sm) {
    v = warp_sum<long long>(v);
    if (lane_id() == 0) sm[warp_in_block()] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        long long r = 0;
        for (u32 w = 0; w < (blockDim.x >> 5); ++w) r += sm[w];
        if (r) atomicAdd((unsigned long long *) slot, (unsigned long long) r);
    }
}

// Adds the block's weight changes to the block weights (after a
// __syncthreads() that follows the last team_move).
__device__ __forceinline__ void team_flush_bw(const TeamArgs &a, const TeamSm &S) {
    for (u32 b = threadIdx.x; b < a.k; b += blockDim.x)
        if (S.bd[b]) {
            atomicAdd(&a.bw[b], S.bd[b]);
            S.bd[b] = 0;
        }
}

// Copies the block weights to shared memory and returns their maximum (at
// least 0). All threads call this.
template<int TEAM>
__device__ __forceinline__ s32 team_load_bw(const TeamArgs &a, const TeamSm &S, s32 *smx) {
    s32 m = 0;
    for (u32 b = threadIdx.x; b < a.k; b += blockDim.x) {
        const s32 x = ld_fresh<TEAM>(&a.bw[b]);
        S.bw[b] = x;
        m = x > m ? x : m;
    }
    m = __reduce_max_sync(FULL, m);
    if (lane_id() == 0) smx[warp_in_block()] = m;
    __syncthreads();
    s32 r = 0;
    for (u32 w = 0; w < (blockDim.x >> 5); ++w) r = smx[w] > r ? smx[w] : r;
    __syncthreads();
    return r;
}

#define TEAM_SYNC()                                                          \
    do {                                                                     \
        if (!team_barrier<TEAM>(a.bar, bar_target, &a.out->err)) return;     \
    } while (0)

// The level loop of one team of gridDim.x blocks. TAB: tables of short rows
// (TeamTable; hashed above TEAM_DIRECT_K blocks).
// MAP: process-mapping objective.
template<int TEAM, int TAB, bool MAP>
__device__ __forceinline__ void team_loop(const TeamArgs &a, const TeamCtl &ctl, const TeamSm &S) {
    __shared__ long long sl[33];
    __shared__ u32 su[33], su2[33];
    __shared__ s32 smx[32];
    // rows shared by the block: candidates (vertex, row, record, sum of the
    // afterburner terms) and moved vertices (row, vertex word)
    __shared__ u32 c_cnt, m_cnt, c_u[TEAM_SHARE_MAX], c_beg[TEAM_SHARE_MAX], c_len[TEAM_SHARE_MAX],
        m_beg[TEAM_SHARE_MAX], m_len[TEAM_SHARE_MAX];
    __shared__ unsigned long long c_rec[TEAM_SHARE_MAX], m_tw[TEAM_SHARE_MAX];
    __shared__ s32 c_sum[TEAM_SHARE_MAX];
    const u32 tid = threadIdx.x, lane = lane_id(), warp = warp_in_block(), nw = blockDim.x >> 5;
    const u32 n = a.n, k = a.k, G = gridDim.x;
    const u32 g = lane >> 3, gl = lane & 7;  // 8-lane groups of the list passes
    const u32 lt = (1u << lane) - 1u;
    u32 bar_target = 0;
    // contiguous vertex range of every warp (ascending with block and warp)
    const u32 gwarps = G * nw, gw = blockIdx.x * nw + warp;
    const u32 per = (n + gwarps - 1) / gwarps;
    const u32 r0 = (u32) min((u64) n, (u64) gw * per), r1 = (u32) min((u64) n, (u64) r0 + per);
    const bool small = per <= TEAM_OWN;
    u32 *const cl = small ? S.own : a.clist + r0;
    u32 *const ml = small ? S.own + TEAM_OWN : a.mlist + r0;
    bool hub = false;
    const unsigned long long t0 = global_ns();
    for (u32 u = r0 + lane; u < r1; u += 32) {
        u32 o;
        if (a.cmap) a.part[u] = o = __ldg(&a.cpart[__ldg(&a.cmap[u])]);
        else o = a.part[u];
        if (a.saved) a.saved[u] = o;
        a.tw[u] = o;
        a.dest_cache[u] = NULL_PART;
        a.lock[u] = 0;
        atomicAdd(&S.bd[o], ld_vw<TEAM>(a, u));
        u32 beg, len;
        ld_row<TEAM>(a, u, beg, len);
        hub |= len > TEAM_HUB;
    }
    if (__any_sync(FULL, hub) && lane == 0) atomicOr(&a.out->hubs, 1u);
    __syncthreads();
    team_flush_bw(a, S);
    if (tid == 0) c_cnt = m_cnt = 0;
    TEAM_SYNC();
    if (blockIdx.x == 0 && tid == 0) a.out->setup_ns = global_ns() - t0;
    const bool hubs = ld_fresh<TEAM>(&a.out->hubs) != 0;
    team_load_bw<TEAM>(a, S, smx);
    long long obj = ctl.obj, best_obj = obj;
    s32 maxw = ctl.maxw, best_max = maxw;
    u32 iterations = 0;
    for (u32 ri = 0; ri < ctl.n_ratios; ++ri) {
        const u32 ratio = ctl.ratios[ri];
        u32 balance_iteration = 0, iteration = 0;
        while (iteration < JET_MAX_ITERATIONS) {
            iteration += 1;
            ++iterations;
            const u32 stamp = iterations;
            // counter set of this iteration (zero); block 0 clears the other
            // one after the first barrier, when every thread has read it
            u32 *const cnt = a.cnt + (iterations & 1u) * TC_N;
            long long *const sum = a.sum + (iterations & 1u) * TS_N;
            u32 *const cnt_o = a.cnt + ((iterations & 1u) ^ 1u) * TC_N;
            long long *const sum_o = a.sum + ((iterations & 1u) ^ 1u) * TS_N;
            bool lp_iter = false;
            int step;
            if (maxw <= a.lmax) {
                step = 0;
                lp_iter = true;
                balance_iteration = 0;
            } else if (!MAP) {
                step = balance_iteration < JET_MAX_WEAK_ITERATIONS ? 1 : 2;
            } else {
                balance_iteration++;
                step = balance_iteration < JET_MAX_WEAK_ITERATIONS ? 1 : 2;
            }
            long long moved = 0;  // (moves << 32) + their row entries, of this thread
            u32 n_own = 0;        // moves in this warp's list
            u32 n_over = 0;       // overloaded blocks (rebalance steps)
            long long evicted = 0;  // evicted weight of all blocks (strong)
            if (step == 0) {
                // gains (cached targets, else recomputed) and filter
                constexpr int OP = MAP ? OP_MAP : OP_CUT;
                u32 nc = 0;  // candidates in this warp's list
                for (u32 base = r0; base < r1; base += 32) {
                    const u32 u = base + lane;
                    const bool act = u < r1;
                    u32 dest = NO_MOVE, lock = 0, o = 0, len = 0, beg = 0;
                    s32 gain = 0;
                    if (act) {
                        dest = a.dest_cache[u];
                        lock = a.lock[u];
                        gain = a.gain_cache[u];
                        o = label_of(a, u);
                        if (small) ld_row<TEAM>(a, u, beg, len);  // one dependent access less
                    }
                    const bool need = act && dest == NULL_PART;
                    if (need && !small) ld_row<TEAM>(a, u, beg, len);
                    const bool hb = need && len > TEAM_HUB;
                    RowOut r{0, 0, 0, 0};
                    rows_short<TEAM, OP, TAB>(a, S, __ballot_sync(FULL, need && len <= 32), beg, len, o, 0, r);
                    rows_long<TEAM, OP>(a, S, __ballot_sync(FULL, need && len > 32 && !hb), beg, len, o, 0, r);
                    if (need && !hb) {
                        lp_decide<MAP>(r, ratio, dest, gain);
                        a.dest_cache[u] = dest;
                        a.gain_cache[u] = gain;
                    }
                    if (hubs) {
                        const u32 sh = warp_append(&cnt[TC_HUB], hb);
                        if (hb) a.hubs[sh] = u;
                    }
                    // a hub row's lock word says later whether it is a candidate
                    const bool c = hb || (act && lp_filter_one(a, u, o, dest, gain, lock));
                    const u32 mask = __ballot_sync(FULL, c);
                    if (c) cl[nc + __popc(mask & lt)] = u;
                    nc += __popc(mask);
                }
                TEAM_SYNC();
                if (blockIdx.x == 0 && tid < TC_N) cnt_o[tid] = 0;
                if (blockIdx.x == 0 && tid < TS_N) sum_o[tid] = 0;
                const u32 nhub = hubs ? ld_fresh<TEAM>(&cnt[TC_HUB]) : 0;
                if (nhub) {
                    for (u32 i = blockIdx.x; i < nhub; i += G) {
                        const u32 u = a.hubs[i], o = label_of(a, u);
                        u32 beg, len;
                        ld_row<TEAM>(a, u, beg, len);
                        row_add<TEAM>(a, beg, len, tid, blockDim.x, S.tab0);
                        __syncthreads();
                        if (warp == 0) {
                            const RowOut r = row_finish<OP>(a, S, S.tab0, o, 0);
                            if (lane == 0) {
                                u32 dest;
                                s32 gain;
                                lp_decide<MAP>(r, ratio, dest, gain);
                                a.dest_cache[u] = dest;
                                a.gain_cache[u] = gain;
                                if (lp_filter_one(a, u, o, dest, gain, a.lock[u])) a.lock[u] = LOCK_HUB;
                            }
                        }
                        __syncthreads();
                    }
                    TEAM_SYNC();
                }
                // afterburner and moves: 8 lanes per candidate, long rows by the warp
                for (u32 base = 0; base < nc; base += 4) {
                    const u32 i = base + g;
                    bool act = i < nc;
                    u32 u = 0, len = 0, beg = 0;
                    unsigned long long rec = 0;
                    if (act) {
                        u = cl[i];
                        ld_row<TEAM>(a, u, beg, len);
                        rec = a.abrec[u];
                        if (len > TEAM_HUB && a.lock[u] != LOCK_HUB) {  // a hub row that is none
                            act = false;
                            len = 0;
                        }
                    }
                    const s32 ug = (s32) (u32) rec;
                    const u32 nu = (u32) (rec >> 32) & 0xFFFFu, ou = (u32) (rec >> 48);
                    s32 ch = 0;
                    if (act && len <= TEAM_LONG) ch = team_ab<TEAM, MAP>(a, S, u, ug, ou, nu, beg, len, gl, 8);
                    __syncwarp();
#pragma unroll
                    for (int d = 4; d > 0; d >>= 1) ch = wadd(ch, __shfl_xor_sync(FULL, ch, d));
                    bool mine = act && gl == 0;  // decided here
                    if (mine && len > TEAM_HUB) a.lock[u] = 0;
                    if (mine && len > TEAM_SHARE) {
                        const u32 p = atomicAdd(&c_cnt, 1u);
                        if (p < TEAM_SHARE_MAX) {
                            c_u[p] = u;
                            c_beg[p] = beg;
                            c_len[p] = len;
                            c_rec[p] = rec;
                            c_sum[p] = 0;
                            mine = false;
                        }
                    }
                    u32 lng = __ballot_sync(FULL, mine && len > TEAM_LONG);
                    while (lng) {
                        const int src = __ffs(lng) - 1;
                        lng &= lng - 1;
                        const u32 xu = __shfl_sync(FULL, u, src), xl = __shfl_sync(FULL, len, src),
                                  xb = __shfl_sync(FULL, beg, src), xo = __shfl_sync(FULL, ou, src),
                                  xn = __shfl_sync(FULL, nu, src);
                        const s32 xg = __shfl_sync(FULL, ug, src);
                        const s32 c =
                            (s32) warp_sum<u32>((u32) team_ab<TEAM, MAP>(a, S, xu, xg, xo, xn, xb, xl, lane, 32));
                        if ((int) lane == src) ch = c;
                    }
                    const bool mv = mine && wadd(ug, ch) >= 0;
                    if (mv) {
                        a.lock[u] = 1;
                        team_move(a, S, u, ou, nu, ld_vw<TEAM>(a, u), stamp);
                        moved += (1ll << 32) + len;
                    }
                    const u32 mask = __ballot_sync(FULL, mv);
                    if (mv) ml[n_own + __popc(mask & lt)] = u;
                    n_own += __popc(mask);
                }
                // the block's long candidates, 128 entries per warp and turn
                __syncthreads();
                const u32 n_long = min(c_cnt, TEAM_SHARE_MAX);
                if (n_long) {
                    for (u32 i = 0; i < n_long; ++i) {
                        const u32 len = c_len[i], beg = c_beg[i], u = c_u[i];
                        const unsigned long long rec = c_rec[i];
                        const s32 ug = (s32) (u32) rec;
                        const u32 nu = (u32) (rec >> 32) & 0xFFFFu, ou = (u32) (rec >> 48);
                        s32 part = 0;
                        bool any = false;
                        for (u32 t = ((warp + 5 * i) % nw) * 128; t < len; t += nw * 128) {
                            part = wadd(part, team_ab<TEAM, MAP>(a, S, u, ug, ou, nu, beg + t, min(len - t, 128u), lane, 32));
                            any = true;
                        }
                        if (any) {
                            part = (s32) warp_sum<u32>((u32) part);
                            if (lane == 0) atomicAdd(&c_sum[i], part);
                        }
                    }
                    __syncthreads();
                    if (tid < n_long) {
                        const u32 u = c_u[tid], len = c_len[tid];
                        const unsigned long long rec = c_rec[tid];
                        if (wadd((s32) (u32) rec, c_sum[tid]) >= 0) {
                            const u32 nu = (u32) (rec >> 32) & 0xFFFFu, ou = (u32) (rec >> 48);
                            a.lock[u] = 1;
                            team_move(a, S, u, ou, nu, ld_vw<TEAM>(a, u), stamp);
                            moved += (1ll << 32) + len;
                            const u32 p = atomicAdd(&m_cnt, 1u);  // at most n_long
                            m_beg[p] = c_beg[tid];
                            m_len[p] = len;
                            m_tw[p] = a.tw[u];
                        }
                    }
                }
            } else {
                const bool strong = step == 2;
                const s32 max_b_w = strong ? a.strong_max : a.weak_max;
                const u32 sft = strong ? 1u : 0u;  // own keys of block o: [o * width + sft, (o + 1) * width + sft)
                // blocks with room (weak) or the largest room (strong), and
                // the overloaded blocks, from the block weights in shared memory
                u32 n_under = 0;
                s32 maxv = INT32_MIN;
                for (u32 b0 = 0; b0 < k; b0 += blockDim.x) {
                    const u32 b = b0 + tid;
                    const s32 x = b < k ? S.bw[b] : INT32_MAX;
                    const bool un = b < k && x < max_b_w, ov = b < k && x > a.lmax;
                    if (un && max_b_w - x > maxv) maxv = max_b_w - x;
                    const u32 mu = __ballot_sync(FULL, un), mo = __ballot_sync(FULL, ov);
                    const s32 mv = __reduce_max_sync(FULL, maxv);
                    if (lane == 0) {
                        su[warp] = __popc(mu);
                        su2[warp] = __popc(mo);
                        smx[warp] = mv;
                    }
                    __syncthreads();
                    const u32 used = (min(k - b0, blockDim.x) + 31) >> 5;
                    u32 pu = n_under, po = n_over;
                    for (u32 w = 0; w < used; ++w) {
                        if (w == warp) {
                            pu = n_under;
                            po = n_over;
                        }
                        n_under += su[w];
                        n_over += su2[w];
                        maxv = smx[w] > maxv ? smx[w] : maxv;
                    }
                    if (un) S.under[pu + __popc(mu & lt)] = b;
                    if (ov) S.olist[po + __popc(mo & lt)] = b;
                    __syncthreads();
                }
                if (strong && blockIdx.x == 0)
                    for (u32 b = tid; b < k; b += blockDim.x) a.ea[b] = 0;
                // picks: target and mini-bucket key of every candidate, whose
                // weight goes to the key's bin
                auto finish = [&](u32 u, u32 o, s32 vw, const RowOut &r) -> u32 {
                    if (strong) {
                        const s32 gain = wsub(r.sum / (r.count ? r.count : 1), r.own);
                        const s32 excess = wsub(S.bw[o], a.lmax);  // of 32 bits, as the reference's
                        return (MAX_BUCKETS * o + gain_bucket(gain, vw < excess ? vw : excess)) * a.sections +
                               (u % a.sections) + 1;
                    }
                    u32 best = o;
                    s32 gain = 0;
                    const s32 best_w = r.bk ? (s32) (u32) (r.bk >> 32) : 0;
                    if (best_w <= 0) {
                        if (n_under > 0) best = S.under[u % n_under];
                        gain = -r.own;
                    } else {
                        best = ~(u32) r.bk;
                        gain = wsub(best_w, r.own);
                    }
                    a.dest[u] = best;
                    return o != best ? (MAX_BUCKETS * o + gain_bucket(gain, vw)) * a.sections + (u % a.sections) : NOKEY;
                };
                for (u32 base = r0; base < r1; base += 32) {
                    const u32 u = base + lane;
                    const bool act = u < r1;
                    u32 o = 0, len = 0, beg = 0;
                    s32 vw = 0;
                    if (act) {
                        o = label_of(a, u);
                        vw = ld_vw<TEAM>(a, u);
                        if (small) ld_row<TEAM>(a, u, beg, len);
                    }
                    bool need = false;
                    if (act) {
                        const s64 ow = S.bw[o];
                        if (ow > a.lmax)
                            need = strong ? ((s64) vw <= 2 * (s64) maxv && (s64) vw < 2 * (ow - a.opt))
                                          : 2 * (s64) vw < 3 * (ow - a.opt);
                    }
                    if (need && !small) ld_row<TEAM>(a, u, beg, len);
                    const bool hb = need && len > TEAM_HUB;
                    RowOut r{0, 0, 0, 0};
                    const u32 ms = __ballot_sync(FULL, need && len <= 32);
                    const u32 mg = __ballot_sync(FULL, need && len > 32 && !hb);
                    if (strong) {
                        rows_short<TEAM, OP_STRONG, TAB>(a, S, ms, beg, len, o, max_b_w, r);
                        rows_long<TEAM, OP_STRONG>(a, S, mg, beg, len, o, max_b_w, r);
                    } else {
                        rows_short<TEAM, OP_WEAK, TAB>(a, S, ms, beg, len, o, max_b_w, r);
                        rows_long<TEAM, OP_WEAK>(a, S, mg, beg, len, o, max_b_w, r);
                    }
                    u32 key = NOKEY;
                    if (need && !hb) key = finish(u, o, vw, r);
                    if (act && !hb) a.keys[u] = key;
                    // one add per distinct key of the warp
                    if (__any_sync(FULL, key != NOKEY)) {
                        const u32 peers = __match_any_sync(FULL, key);
                        s32 p, t;
                        peer_prefix(peers, vw, p, t);
                        if (key != NOKEY && (peers & lt) == 0) atomicAdd(&a.hist[key], (u32) t);
                    }
                    if (hubs) {
                        const u32 sh = warp_append(&cnt[TC_HUB], hb);
                        if (hb) a.hubs[sh] = u;
                    }
                }
                TEAM_SYNC();
                if (blockIdx.x == 0 && tid < TC_N) cnt_o[tid] = 0;
                if (blockIdx.x == 0 && tid < TS_N) sum_o[tid] = 0;
                const u32 nhub = hubs ? ld_fresh<TEAM>(&cnt[TC_HUB]) : 0;
                if (nhub) {
                    for (u32 i = blockIdx.x; i < nhub; i += G) {
                        const u32 u = a.hubs[i], o = label_of(a, u);
                        u32 beg, len;
                        ld_row<TEAM>(a, u, beg, len);
                        row_add<TEAM>(a, beg, len, tid, blockDim.x, S.tab0);
                        __syncthreads();
                        if (warp == 0) {
                            const RowOut r = strong ? row_finish<OP_STRONG>(a, S, S.tab0, o, max_b_w)
                                                    : row_finish<OP_WEAK>(a, S, S.tab0, o, max_b_w);
                            if (lane == 0) {
                                const s32 vw = ld_vw<TEAM>(a, u);
                                const u32 key = finish(u, o, vw, r);
                                a.keys[u] = key;
                                if (key != NOKEY) atomicAdd(&a.hist[key], (u32) vw);
                            }
                        }
                        __syncthreads();
                    }
                    TEAM_SYNC();
                }
                // per overloaded block: the bin in which the limit falls, by 8
                // lanes over contiguous shares of the block's bins
                if (strong) {
                    for (u32 b = tid; b < k; b += blockDim.x) S.tot[b] = 0;
                    __syncthreads();
                }
                const u32 share = (a.width + 7) / 8;
                for (u32 i0 = warp * 4; i0 < n_over; i0 += nw * 4) {
                    const u32 i = i0 + g;
                    const bool act = i < n_over;
                    const u32 o = act ? S.olist[i] : 0;
                    const u32 b0 = min(gl * share, a.width), b1 = min(b0 + share, a.width);
                    const u32 *h = a.hist + (u64) o * a.width + sft;
                    s32 mine = 0, last = 0, spill = 0;
                    s32 hv[8];
                    if (act) {
                        if (share <= 8) {
#pragma unroll
                            for (u32 x = 0; x < 8; ++x) hv[x] = b0 + x < b1 ? (s32) ld_fresh<TEAM>(&h[b0 + x]) : 0;
#pragma unroll
                            for (u32 x = 0; x < 8; ++x) mine += hv[x];
                        } else {
#pragma unroll 8
                            for (u32 x = b0; x < b1; ++x) mine += (s32) ld_fresh<TEAM>(&h[x]);
                        }
                        if (strong) {
                            last = (s32) ld_fresh<TEAM>(&h[a.width - 1]);
                            spill = (s32) ld_fresh<TEAM>(h - 1);
                        }
                    }
                    s32 inc = mine;
#pragma unroll
                    for (int d = 1; d < 8; d <<= 1) {
                        const s32 y = __shfl_up_sync(FULL, inc, d, 8);
                        if ((int) gl >= d) inc += y;
                    }
                    const s32 total = __shfl_sync(FULL, inc, 7, 8) + spill;
                    s32 run = spill + inc - mine;
                    const s32 limit = act ? excess_of(a, S, o) : 0;
                    if (act && gl == 0) {
                        S.toff[o] = 0;
                        // all bins but the last one of strong keys, which the
                        // next block's range starts with (key = (o + 1) * width)
                        S.tot[o] = strong ? total - last : total;
                        S.spill[o] = spill;
                        // no bin reaches the limit: all are taken; the bin of
                        // the previous block reaches it: none is
                        if (total < limit || spill >= limit) {
                            S.cutkey[o] = total < limit ? NOKEY : 0u;
                            S.cutbase[o] = 0;
                        }
                    }
                    if (act && run < limit && limit <= run + mine) {
                        u32 x = b0;
                        if (share <= 8) {
                            bool done = false;
#pragma unroll
                            for (u32 y = 0; y < 8; ++y) {
                                done = done || limit <= run + hv[y];
                                if (!done) {
                                    run += hv[y];
                                    ++x;
                                }
                            }
                        } else {
                            for (; x < b1; ++x) {
                                const s32 c = (s32) ld_fresh<TEAM>(&h[x]);
                                if (limit <= run + c) break;
                                run += c;
                            }
                        }
                        S.cutkey[o] = o * a.width + sft + x;
                        S.cutbase[o] = run;
                    }
                }
                __syncthreads();
                if (strong)
                    // a block after an overloaded one whose own weight is
                    // within the limit holds only that block's last bin
                    for (u32 i = tid; i < n_over; i += blockDim.x) {
                        const u32 o = S.olist[i];
                        if (o + 1 < k && S.bw[o + 1] <= a.lmax)
                            S.tot[o + 1] = (s32) ld_fresh<TEAM>(&a.hist[(u64) (o + 1) * a.width]);
                    }
                // weight of each warp's candidates in the cut bins
                for (u32 base = r0; base < r1; base += 32) {
                    const u32 u = base + lane;
                    if (u < r1) {
                        const u32 key = a.keys[u];
                        if (key != NOKEY) {
                            const u32 o = (key - sft) / a.width;
                            if (key == S.cutkey[o]) atomicAdd(&S.tab[o], ld_vw<TEAM>(a, u));
                        }
                    }
                }
                if (TEAM == TEAM_CLUSTER) {
                    // weight in the cut bins before this block's vertices: a
                    // cluster's levels are small enough for every block to
                    // look at all keys before its own (one barrier less)
                    const u32 first = (u32) min((u64) n, (u64) blockIdx.x * nw * per);
                    for (u32 u = tid; u < first; u += blockDim.x) {
                        const u32 key = __ldcg(&a.keys[u]);
                        if (key != NOKEY) {
                            const u32 o = (key - sft) / a.width;
                            if (key == S.cutkey[o]) atomicAdd(&S.toff[o], ld_vw<TEAM>(a, u));
                        }
                    }
                }
                __syncthreads();
                for (u32 i = tid; i < n_over; i += blockDim.x) {
                    const u32 o = S.olist[i];
                    s32 run = 0;
                    for (u32 w = 0; w < nw; ++w) {
                        s32 *p = S.tab0 + w * S.stride + o;
                        const s32 x = *p;
                        *p = run;
                        run += x;
                    }
                    if (TEAM == TEAM_GRID) a.tsum[(u64) o * G + blockIdx.x] = run;
                }
                if (TEAM == TEAM_GRID) {
                    TEAM_SYNC();
                    // weight before this block's share of the cut bins
                    for (u32 i0 = warp * 4; i0 < n_over; i0 += nw * 4) {
                        const u32 i = i0 + g;
                        const bool act = i < n_over;
                        const u32 o = act ? S.olist[i] : 0;
                        s32 x = 0;
                        if (act)
#pragma unroll 4
                            for (u32 b = gl; b < blockIdx.x; b += 8) x += __ldcg(&a.tsum[(u64) o * G + b]);
#pragma unroll
                        for (int d = 4; d > 0; d >>= 1) x += __shfl_xor_sync(FULL, x, d);
                        if (act && gl == 0) S.toff[o] = x;
                    }
                }
                __syncthreads();
                // selection in ascending vertex id
                for (u32 base = r0; base < r1; base += 32) {
                    const u32 u = base + lane;
                    const u32 key = u < r1 ? a.keys[u] : NOKEY;
                    if (__ballot_sync(FULL, key != NOKEY) == 0) continue;
                    u32 o = 0;
                    s32 vw = 0;
                    bool take = false, cut = false;
                    if (key != NOKEY) {
                        o = (key - sft) / a.width;
                        vw = ld_vw<TEAM>(a, u);
                        cut = key == S.cutkey[o];
                        take = key < S.cutkey[o];
                    }
                    if (__any_sync(FULL, cut)) {
                        const u32 peers = __match_any_sync(FULL, cut ? o : EMPTY);
                        s32 p, t;
                        peer_prefix(peers, vw, p, t);
                        s32 before = 0;
                        if (cut) before = S.tab[o];
                        __syncwarp();
                        if (cut) {
                            if ((peers & lt) == 0) S.tab[o] = before + t;
                            const s32 score = S.cutbase[o] + S.toff[o] + before + p;
                            const s32 limit = excess_of(a, S, o);
                            take = score < limit;
                            if (strong && take && score + vw >= limit) a.ea[o] = score + vw;
                        }
                        __syncwarp();
                    }
                    if (strong) {
                        if (!__any_sync(FULL, take)) continue;
                        const u32 s = warp_append(&cnt[TC_MOVES], take);
                        if (take) {
                            a.mcomp[s] = ((unsigned long long) key << 32) | u;
                            a.mow[s] = ((unsigned long long) o << 32) | (u32) vw;
                        }
                    } else {
                        if (take) {
                            u32 beg, len;
                            ld_row<TEAM>(a, u, beg, len);
                            team_move(a, S, u, o, a.dest[u], vw, stamp);
                            moved += (1ll << 32) + len;
                        }
                        const u32 mask = __ballot_sync(FULL, take);
                        if (take) ml[n_own + __popc(mask & lt)] = u;
                        n_own += __popc(mask);
                    }
                }
                __syncwarp();
                for (u32 i = lane; i < n_over; i += 32) S.tab[S.olist[i]] = 0;
                if (strong) {
                    TEAM_SYNC();
                    const u32 ns = ld_fresh<TEAM>(&cnt[TC_MOVES]);
                    if (TEAM != TEAM_BLOCK && (u64) ns * ns > (u64) a.rank_pairs * gwarps) {
                        if (blockIdx.x == 0 && tid == 0) a.out->gave_up = 1;
                        return;
                    }
                    // cookie cutter (:524-551): evicted weight before each
                    // block and free capacity up to each block
                    long long c1 = 0, c2 = 0;
                    for (u32 b0 = 0; b0 < k; b0 += blockDim.x) {
                        const u32 b = b0 + tid;
                        long long add = 0, cap = 0;
                        if (b < k) {
                            add = ld_fresh<TEAM>(&a.ea[b]);
                            if (add == 0) add = S.tot[b];
                            cap = max_b_w > S.bw[b] ? (long long) max_b_w - S.bw[b] : 0;
                        }
                        long long t1, t2;
                        const long long p1 = block_exclusive_scan<long long>(add, t1, sl);
                        const long long p2 = block_exclusive_scan<long long>(cap, t2, sl);
                        if (b < k) {
                            S.pre[b] = c1 + p1;
                            S.es[b + 1] = c2 + p2 + cap;
                        }
                        c1 += t1;
                        c2 += t2;
                    }
                    evicted = c1;
                    if (tid == 0) S.es[0] = 0;
                    __syncthreads();
                    // exact prefix of each evicted vertex among its block's
                    // and the first slot attempt (adjust_scores :560-584). A
                    // warp ranks two vertices against tiles of all in shared
                    // memory, because warps that read the list from L2
                    // were bound by its bandwidth (8000 vertices, 148 blocks:
                    // 211 us a step, now 46)
                    u32 *const t_key = S.own0, *const t_u = t_key + blockDim.x;
                    s32 *const t_vw = (s32 *) (t_u + blockDim.x);
                    for (u32 j0 = 0; j0 < ns; j0 += 2 * gwarps) {
                        unsigned long long comp[2], ow[2], low[2];
                        s32 x[2] = {0, 0};
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            const u32 j = j0 + q * gwarps + gw;
                            comp[q] = j < ns ? a.mcomp[j] : 0ull;
                            ow[q] = j < ns ? a.mow[j] : 0ull;
                            low[q] = (unsigned long long) ((u32) (ow[q] >> 32) * a.width + sft) << 32;
                        }
                        for (u32 t0 = 0; t0 < ns; t0 += blockDim.x) {
                            const u32 tn = min(ns - t0, blockDim.x);
                            if (j0 == 0 || ns > blockDim.x) {
                                __syncthreads();
                                if (tid < tn) {
                                    const unsigned long long c = a.mcomp[t0 + tid];
                                    t_key[tid] = (u32) (c >> 32);
                                    t_u[tid] = (u32) c;
                                    t_vw[tid] = (s32) (u32) a.mow[t0 + tid];
                                }
                                __syncthreads();
                            }
                            for (u32 i = lane; i < tn; i += 32) {
                                const unsigned long long c = ((unsigned long long) t_key[i] << 32) | t_u[i];
                                const s32 vw = t_vw[i];
#pragma unroll
                                for (int q = 0; q < 2; ++q)  // keys of the same block that are smaller
                                    if (c - low[q] < comp[q] - low[q]) x[q] += vw;
                            }
                        }
                        __syncwarp();
#pragma unroll
                        for (int q = 0; q < 2; ++q)
                            for (int d = 16; d > 0; d >>= 1) x[q] += __shfl_xor_sync(FULL, x[q], d);
                        if (lane < 2 && j0 + lane * gwarps + gw < ns) {
                            const u32 u = (u32) (lane ? comp[1] : comp[0]), o = (u32) ((lane ? ow[1] : ow[0]) >> 32);
                            const s32 vw = (s32) (u32) (lane ? ow[1] : ow[0]);
                            const long long tg = (long long) S.spill[o] + (lane ? x[1] : x[0]) + S.pre[o];
                            const s32 id = chunk_of(S.es, k, tg);
                            const bool fits = id < (s32) k && (long long) (vw / 2) <= S.es[id + 1] - tg;
                            if (!fits && id < (s32) k) {
                                a.fails[atomicAdd(&cnt[TC_FAIL], 1u)] = u;
                            } else {
                                team_move(a, S, u, o, fits ? (u32) id : o, vw, stamp);
                            }
                            u32 beg, len;
                            ld_row<TEAM>(a, u, beg, len);
                            moved += (1ll << 32) + len;
                        }
                        __syncwarp();
                    }
                }
            }
            team_add(moved, &sum[TS_MOVES], sl);
            team_flush_bw(a, S);
            TEAM_SYNC();
            if (step == 2) {
                const u32 nf = ld_fresh<TEAM>(&cnt[TC_FAIL]);
                if (nf) {
                    // fallback slots in ascending vertex id (block 0)
                    if (blockIdx.x == 0) {
                        for (u32 j = tid; j < nf; j += blockDim.x) {
                            const u32 u = a.fails[j];
                            u32 p = 0;
                            for (u32 i = 0; i < nf; ++i) p += a.fails[i] < u;
                            a.hubs[p] = u;
                        }
                        __syncthreads();
                        if (tid == 0) {
                            long long mv = evicted;
                            for (u32 j = 0; j < nf; ++j) {
                                const u32 u = a.hubs[j];
                                const u32 o = label_of(a, u);
                                const s32 vw = ld_vw<TEAM>(a, u);
                                u32 dest = o;
                                for (u32 guard = 0; guard < 2 * k + 4; ++guard) {
                                    const long long tg = mv;
                                    mv += vw;
                                    const s32 id = chunk_of(S.es, k, tg);
                                    if (id >= (s32) k) break;
                                    if ((long long) (vw / 2) <= S.es[id + 1] - tg) {
                                        dest = (u32) id;
                                        break;
                                    }
                                }
                                team_move(a, S, u, o, dest, vw, stamp);
                            }
                        }
                        __syncthreads();
                        team_flush_bw(a, S);
                    }
                    TEAM_SYNC();
                }
            }
            // exact objective change and the neighbours' cache resets
            const unsigned long long ent = (unsigned long long) ld_fresh<TEAM>(&sum[TS_MOVES]);
            const u32 nm = (u32) (ent >> 32);
            const bool inval = (ent & 0xFFFFFFFFull) < a.inval_all_min;
            const s32 new_maxw = team_load_bw<TEAM>(a, S, smx);
            // the bins are not read any more: clear them
            if (step != 0)
                for (u32 i = blockIdx.x; i < n_over; i += G) {
                    u32 *h = a.hist + (u64) S.olist[i] * a.width;
                    for (u32 x = tid; x <= a.width; x += blockDim.x) h[x] = 0;
                }
            long long acc = 0;
            {
                // this warp's own moves, or its share of the evicted vertices
                const bool shared_list = step == 2;
                const u32 first = shared_list ? gw * 4 : 0, stride = shared_list ? gwarps * 4 : 4;
                const u32 total = shared_list ? nm : n_own;
                for (u32 base = first; base < total; base += stride) {
                    const u32 i = base + g;
                    u32 u = 0, len = 0, beg = 0;
                    unsigned long long x = 0;
                    if (i < total) {
                        u = shared_list ? (u32) a.mcomp[i] : ml[i];
                        ld_row<TEAM>(a, u, beg, len);
                        x = a.tw[u];
                    }
                    if (len <= TEAM_LONG)
                        acc += team_delta<TEAM, MAP>(a, S, tw_old(x), tw_label(x), tw_stamp(x) == stamp, stamp, beg, len,
                                                     gl, 8, inval);
                    __syncwarp();
                    bool mine = gl == 0 && len > TEAM_LONG;
                    if (mine && len > TEAM_SHARE) {
                        const u32 p = atomicAdd(&m_cnt, 1u);
                        if (p < TEAM_SHARE_MAX) {
                            m_beg[p] = beg;
                            m_len[p] = len;
                            m_tw[p] = x;
                            mine = false;
                        }
                    }
                    u32 lng = __ballot_sync(FULL, mine);
                    while (lng) {
                        const int src = __ffs(lng) - 1;
                        lng &= lng - 1;
                        const u32 xl = __shfl_sync(FULL, len, src), xb = __shfl_sync(FULL, beg, src);
                        const unsigned long long xx = __shfl_sync(FULL, x, src);
                        acc += team_delta<TEAM, MAP>(a, S, tw_old(xx), tw_label(xx), tw_stamp(xx) == stamp, stamp, xb, xl,
                                                     lane, 32, inval);
                    }
                }
            }
            if (!inval)
                for (u32 u = r0 + lane; u < r1; u += 32) a.dest_cache[u] = NULL_PART;
            // the block's long moved rows, 128 entries per warp and turn
            __syncthreads();
            const u32 m_long = min(m_cnt, TEAM_SHARE_MAX);
            for (u32 i = 0; i < m_long; ++i) {
                const u32 len = m_len[i], beg = m_beg[i];
                const unsigned long long x = m_tw[i];
                for (u32 t = ((warp + 5 * i) % nw) * 128; t < len; t += nw * 128)
                    acc += team_delta<TEAM, MAP>(a, S, tw_old(x), tw_label(x), tw_stamp(x) == stamp, stamp, beg + t,
                                                 min(len - t, 128u), lane, 32, inval);
            }
            team_add(acc, &sum[TS_DELTA], sl);  // (every thread has read m_cnt after its barrier)
            if (tid == 0) c_cnt = m_cnt = 0;
            TEAM_SYNC();
            const long long d = ld_fresh<TEAM>(&sum[TS_DELTA]);
            // control (jet_label_propagation.h:966-1030, promap :1250-1305)
            if (!MAP) {
                if (nm == 0) {
                    if (lp_iter || balance_iteration >= JET_MAX_WEAK_ITERATIONS) break;
                    balance_iteration = JET_MAX_WEAK_ITERATIONS;
                    continue;
                }
                if (!lp_iter) balance_iteration++;
            } else if (nm == 0) {
                continue;
            }
            obj += MAP ? d : d / 2;
            maxw = new_maxw;
            bool copy = false;
            const bool leq = MAP ? (maxw < best_max) : (maxw <= best_max);
            if (best_max > a.lmax && maxw < best_max) {
                copy = true;
                iteration = 0;
            } else if (obj < best_obj && (maxw <= a.lmax || leq)) {
                if (1000 * obj < 999 * best_obj) iteration = 0;  // PHI = 0.999
                copy = true;
            }
            if (copy) {
                best_obj = obj;
                best_max = maxw;
                // labels change again after the next barrier at the earliest
                for (u32 u = r0 + lane; u < r1; u += 32) a.part[u] = label_of(a, u);
            }
        }
    }
    if (blockIdx.x == 0 && tid == 0) {
        a.out->obj = best_obj;
        a.out->maxw = best_max;
        a.out->iterations = iterations;
    }
}

#undef TEAM_SYNC

// Zeroes the tables and loads the distance oracle.
template<bool MAP>
__device__ __forceinline__ TeamSm team_setup(const TeamArgs &a, unsigned char *dsm) {
    const u32 tid = threadIdx.x, nw = blockDim.x >> 5;
    const TeamSm S = team_carve(dsm, a.k, nw, warp_in_block(), MAP);
    for (u32 i = tid; i < nw * S.stride; i += blockDim.x) S.tab0[i] = 0;
    for (u32 b = tid; b < a.k; b += blockDim.x) {
        S.bd[b] = 0;
        if (MAP) S.code[b] = a.code[b];
    }
    if (MAP && tid < 32) S.dist[tid] = a.bitdist[tid];
    __syncthreads();
    return S;
}

// A cluster or a cooperative grid on a level in global memory.
template<int TEAM, int TAB, bool MAP>
__global__ void __launch_bounds__(1024, 1) k_jet_team(const __grid_constant__ TeamArgs a,
                                                        const __grid_constant__ TeamCtl ctl) {
    extern __shared__ __align__(16) unsigned char team_dsm[];
    const TeamSm S = team_setup<MAP>(a, team_dsm);
    team_loop<TEAM, TAB, MAP>(a, ctl, S);
}

// One block that copies the level to shared memory first (rows made
// contiguous). `level` is the offset of the level's arrays.
template<int TAB, bool MAP>
__global__ void __launch_bounds__(512, 1) k_jet_block(const __grid_constant__ TeamArgs ga,
                                                        const __grid_constant__ TeamCtl ctl, u32 m, u32 level) {
    extern __shared__ __align__(16) unsigned char team_dsm[];
    __shared__ u32 scan_sm[32];
    const TeamSm S = team_setup<MAP>(ga, team_dsm);
    const u32 n = ga.n, k = ga.k, tid = threadIdx.x, lane = lane_id();
    TeamArgs a = ga;
    unsigned long long *q = (unsigned long long *) (team_dsm + level);
    a.tw = q;
    a.abrec = q + n;
    a.dest = (u32 *) a.abrec;  // records belong to label propagation, targets and keys to rebalancing
    a.keys = a.dest + n;
    a.mcomp = q + 2 * (u64) n;
    a.mow = q + 3 * (u64) n;
    q += 4 * (u64) n;
    TeamOut *out = (TeamOut *) q;
    a.out = out;
    a.sum = (long long *) (out + 1);
    u32 *p = (u32 *) (a.sum + 2 * TS_N);
    u32 *rowptr = p;
    p += n + 1;
    a.dest_cache = p;
    a.gain_cache = (s32 *) (p + n);
    a.lock = p + 2 * n;
    s32 *vw = (s32 *) (p + 3 * n);
    a.clist = a.fails = p + 4 * n;
    a.mlist = a.hubs = p + 5 * n;
    p += 6 * n;
    u32 *adj = p;
    s32 *ew = (s32 *) (p + m);
    p += 2 * m;
    a.cnt = p;
    a.bw = (s32 *) (p + 2 * TC_N);
    a.ea = a.bw + k;
    a.hist = (u32 *) (a.ea + k);
    const u32 bins = k * a.width + 2;
    if (tid == 0) {
        out->hubs = 0;
        out->gave_up = 0;
        out->err = 0;
    }
    if (tid < 2 * TS_N) a.sum[tid] = 0;
    if (tid < 2 * TC_N) a.cnt[tid] = 0;
    for (u32 b = tid; b < k; b += blockDim.x) a.bw[b] = 0;
    for (u32 b = tid; b < bins; b += blockDim.x) a.hist[b] = 0;
    // row offsets, then the rows, 8 lanes each
    u32 run = 0;
    for (u32 u0 = 0; u0 < n; u0 += blockDim.x) {
        const u32 u = u0 + tid;
        const u32 len = u < n ? __ldg(&ga.rowlen[u]) : 0;
        u32 tot;
        const u32 pos = run + block_exclusive_scan<u32>(len, tot, scan_sm);
        if (u < n) {
            rowptr[u] = pos;
            vw[u] = ga.vw ? __ldg(&ga.vw[u]) : 1;
        }
        run += tot;
    }
    if (tid == 0) rowptr[n] = run;
    __syncthreads();
    for (u32 u = tid >> 3; u < n; u += blockDim.x >> 3) {
        const u32 src = __ldg(&ga.rowptr[u]), dst = rowptr[u], len = rowptr[u + 1] - dst;
        for (u32 t = lane & 7; t < len; t += 8) {
            adj[dst + t] = __ldg(&ga.adj[src + t]);
            ew[dst + t] = ga.ew ? __ldg(&ga.ew[src + t]) : 1;
        }
    }
    __syncthreads();
    a.rowptr = rowptr;
    a.adj = adj;
    a.ew = ew;
    a.vw = vw;
    team_loop<TEAM_BLOCK, TAB, MAP>(a, ctl, S);
    if (tid == 0) {
        ga.out->obj = out->obj;
        ga.out->maxw = out->maxw;
        ga.out->iterations = out->iterations;
        ga.out->gave_up = out->gave_up;
        ga.out->err = out->err;
        ga.out->setup_ns = out->setup_ns;
    }
}
