// Coarsening: two-hop heavy-edge matching and hash contraction.
#pragma once
#include "graph.cuh"

namespace hp {

// two_hop_matcher_get_mapping (src/coarsening/two_hop_matching.h:573-650)
// with the deterministic commit rule (smallest proposer wins a receiver) and
// digest grouping by exact value for the leaf/twin/relative passes. Writes the
// fine->coarse map (device, n entries) and returns the coarse vertex count.
// one_launch: try the single launch below first, where it applies.
u32 match_graph(Ctx &ctx, const DGraph &g, u32 *mapping, bool one_launch = true);

// from_Graph_Mapping (src/datastructures/graph.h:127-390): coarse vertex
// weights are summed members, coarse edges aggregate all fine edges between
// two clusters (parallel edge weights summed, self loops dropped). The
// coarse graph is allocated from the front of the arena. Rows are written in
// hash-slot order; the row contents are exact.
DGraph contract_graph(Ctx &ctx, const DGraph &g, const u32 *mapping, u32 n_c);

// One coarsening level in one launch (coarsen_team.cu). `mapping` receives
// the fine->coarse map. With `rows` (adj and ew allocated with room for g.m
// entries), the coarse rows are written there, and the coarse graph's row
// bounds and vertex weights to its rowptr (room for n + 1), rowlen and vw, or,
// where those are null, to scratch that is valid until the caller releases it
// (the result's rowptr, rowlen and vw). contracted is false when a
// coarse row is too long for the kernel's tables (contract_graph then builds
// the graph). Throws CoopSpin when the launch cannot be made or gave up.
struct CoarsenResult {
    u32 n = 0;
    u64 m = 0;
    bool contracted = false;
    double contract_ms = 0;
    u32 *rowptr = nullptr, *rowlen = nullptr;
    s32 *vw = nullptr;
};
constexpr u32 COARSEN_TEAM_MAX_N = 1u << 20;  // upper bound of Tunables::match_coop_max_n

bool coarsen_team_applies(const Ctx &ctx, const DGraph &g);
CoarsenResult coarsen_team(Ctx &ctx, const DGraph &g, u32 *mapping, DGraph *rows);

} // namespace hp
