// Teams: the blocks that run a whole level loop in one launch. A team is one
// block, one thread-block cluster (hardware barrier, co-scheduled by the
// hardware) or one cooperative grid (bounded barrier in global memory).
#pragma once
#include "context.h"

namespace hp {

enum TeamKind { TEAM_BLOCK = 0, TEAM_CLUSTER = 1, TEAM_GRID = 2 };

constexpr u32 TEAM_CLUSTER_MAX = 16;        // blocks of a cluster team
constexpr u32 TEAM_BLOCK_THREADS = 512;     // threads of a block team ...
constexpr u32 TEAM_CLUSTER_THREADS = 512;   // ... of a block of a cluster team ...
constexpr u32 TEAM_GRID_THREADS = 1024;     // ... and of a grid team
constexpr size_t TEAM_SMEM_MAX = 220 * 1024;  // dynamic shared memory of a block (7 KB are left for static arrays)

inline u32 team_threads(int team) {
    return team == TEAM_GRID ? TEAM_GRID_THREADS : (team == TEAM_CLUSTER ? TEAM_CLUSTER_THREADS : TEAM_BLOCK_THREADS);
}

// Grid barrier: one counter that only grows; thread 0 of every block adds one
// and waits for it to reach a multiple of the grid size. The wait is bounded:
// after TEAM_SPINS polls (about a second) a block sets TEAM_POISON, which ends
// every wait, and all blocks leave (false; the host redoes the level).
constexpr u32 TEAM_POISON = 0x80000000u;
constexpr u32 TEAM_SPINS = 1u << 21;

template<int TEAM>
__device__ __forceinline__ bool team_barrier(u32 *bar, u32 &target, u32 *err) {
    if (TEAM == TEAM_BLOCK) {
        __syncthreads();
        return true;
    }
    if (TEAM == TEAM_CLUSTER) {
        asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
        return true;
    }
    __shared__ u32 s_ok;
    target += gridDim.x;
    __syncthreads();
    if (threadIdx.x == 0) {
        u32 v;
        asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(v) : "l"(bar) : "memory");
        v += 1;
        u32 spins = 0;
        while (v < target) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
            if (++spins > TEAM_SPINS) {
                set_error(err, DEV_ERR_SPIN);
                atomicOr(bar, TEAM_POISON);
                v = TEAM_POISON;
            }
        }
        s_ok = v < TEAM_POISON ? 1u : 0u;
    }
    __syncthreads();
    return s_ok != 0u;
}

// A word that other blocks wrote before the last barrier and that steers the
// control flow: from L2, or (block team) shared memory or this SM's view.
template<int TEAM, typename T>
__device__ __forceinline__ T ld_fresh(const T *p) {
    return TEAM == TEAM_BLOCK ? *(const volatile T *) p : __ldcg(p);
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// Launch configuration of a team of `blocks` blocks (attr must outlive it).
inline cudaLaunchConfig_t team_config(u32 blocks, u32 threads, size_t smem, cudaStream_t stream,
                                      cudaLaunchAttribute &attr, int team) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    if (team == TEAM_CLUSTER) {
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = blocks;
        attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = 1;
    } else {
        attr.id = cudaLaunchAttributeCooperative;
        attr.val.cooperative = 1;
    }
    cfg.attrs = &attr;
    cfg.numAttrs = team == TEAM_BLOCK ? 0 : 1;
    return cfg;
}

// Sets the limits of a cluster kernel that uses up to `smem` bytes and returns
// the largest cluster (a power of two up to `most`) that the device can run.
inline u32 team_cluster_limit(const void *kernel, size_t smem, u32 most) {
    HP_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
    HP_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    for (; most > 1; most /= 2) {
        cudaLaunchAttribute attr;
        const cudaLaunchConfig_t cfg = team_config(most, TEAM_CLUSTER_THREADS, smem, nullptr, attr, TEAM_CLUSTER);
        int fits = 0;
        if (cudaOccupancyMaxActiveClusters(&fits, kernel, &cfg) == cudaSuccess && fits > 0) break;
        cudaGetLastError();
    }
    return most;
}

// Blocks of a grid team for `want` of them, one SM each: at least two, at most
// what fits on the GPU at once. Beside other solves a grid takes a share of the
// SMs, so that grids run side by side instead of one after another at full
// width (HM RGG 8M: 403 ms uncapped, 342 ms with shares of 32 blocks). The
// sub-solves of a multisection are alike and finish together: small shares
// serve them best (16 / 24 / 40 / 56 blocks: 244 / 251 / 264 / 294 ms). Batch
// and server jobs differ, and often few of them run a grid at a time (146 / 135
// / 127 / 127 ms for the batch of 32 graphs).
constexpr u32 HM_PEER_BLOCKS = 20;

inline u32 team_grid_blocks(const Ctx &ctx, const void *kernel, size_t smem, u64 want) {
    int per_sm = 0;
    HP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, TEAM_GRID_THREADS, smem));
    if (per_sm <= 0) return 0;
    u64 cap = (u64) per_sm * ctx.sm_count;
    if (ctx.peers > 1) {
        u64 share = 2 * (u64) ctx.sm_count / ctx.peers;
        if (share < ctx.peer_blocks) share = ctx.peer_blocks;
        if (share < cap) cap = share;
    }
    want = want < cap ? want : cap;
    return (u32) (want < 2 ? 2 : want);
}

} // namespace hp
