// Chains of small levels in one launch.
#pragma once
#include <atomic>
#include <stdexcept>
#include <string>

#include "launch.h"

namespace grgx {

__device__ __forceinline__ void cluster_barrier() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

// The levels of p one after the other, by one cluster of thread blocks: every row by G lanes, or as
// many groups of them as the level's split says, as in short_rows_kernel.  A level waits for the one
// before at the cluster's barrier (the hardware's: nothing spins), and a row's offset and first ids
// are loaded before it.  Rows are gathered from L2, where the other SMs' stores of this launch are.
//
// A launch per level costs 3-4 us however small the level, most of it the launch, its end and the chain
// of dependent loads offset -> id -> row; here a level of one round takes about 2.5 us, the row's load,
// its sum and the barrier.  One cluster is 16 SMs: levels with more work than that stay launches of
// their own (launch_levels).
template <class Op, int VW, int G, class Params>
__device__ __forceinline__ void chain_levels(const Params& p) {
    using S = typename Op::S;
    const unsigned threads = gridDim.x * blockDim.x, lane = threadIdx.x & 31;
    const unsigned warp0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u);
    struct Item {
        unsigned row, e, end;
        int sub, col;
        bool live;
        uint32_t id[kShortBatch];
    };
    // Lane `lane` of the 32 items from `base` on: columns of one tile after the other.
    auto fetch = [&](const ChainLevel& v, unsigned base) {
        Item t;
        const unsigned perRow = G * v.split, perTile = (v.rows * perRow + 31u) & ~31u;
        const unsigned tile = base / perTile, x = base - tile * perTile + lane;
        t.row = x / perRow;
        t.sub = static_cast<int>(x / G) & (v.split - 1);
        t.col = static_cast<int>(tile) * (G * VW) + static_cast<int>(lane % G) * VW;
        t.live = t.row < v.rows && t.col < p.stride;
        t.e = t.end = 0;
        if (t.live) {
            t.e = __ldg(v.off + t.row) + kShortBatch * t.sub;
            t.end = __ldg(v.off + t.row + 1);
        }
#pragma unroll
        for (int u = 0; u < kShortBatch; u++) t.id[u] = (t.e + u < t.end) ? __ldg(v.adj + t.e + u) : 0u;
        return t;
    };
    auto items = [&](const ChainLevel& v) { return ((v.rows * G * v.split + 31u) & ~31u) * static_cast<unsigned>(p.tiles); };
    Item next = fetch(p.level[0], warp0 < items(p.level[0]) ? warp0 : 0);
    for (int l = 0; l < p.count; l++) {
        const ChainLevel v = p.level[l];
        SweepParams<S> q{};
        q.src = static_cast<const S*>(v.src);
        q.dst = static_cast<S*>(p.vals);
        q.stride = p.stride;
        q.rmw = v.rmw;
        q.rows = v.nodes;
        q.state = p.state;
        q.state_base = p.state_base;
        q.state_mode = 2;
        const unsigned total = items(v);
        for (unsigned base = warp0; base < total; base += threads) {
            Item t = (base == warp0) ? next : fetch(v, base);
            short_row<Op, VW, G, true>(q, v.adj, t.row, t.col, v.split, t.sub, t.live, t.e, t.end, t.id);
        }
        if (l + 1 < p.count) {
            next = fetch(p.level[l + 1], warp0 < items(p.level[l + 1]) ? warp0 : 0);
            cluster_barrier();
        }
    }
}

template <class Op, int VW, int G>
__global__ void __launch_bounds__(kChainThreads, 1) chain_kernel(const ChainParams p) {
    if constexpr (std::is_same<Op, AddF64S>::value) {
        if (p.gate != nullptr && *p.gate != 0) {
            chain_levels<AddF64, VW, G>(p);
            return;
        }
    }
    chain_levels<Op, VW, G>(p);
}

// One cluster of kChainBlocks blocks.
struct ChainLaunch {
    cudaLaunchAttribute attr{};
    cudaLaunchConfig_t config{};
    explicit ChainLaunch(cudaStream_t s) {
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = kChainBlocks;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        config.gridDim = dim3(kChainBlocks);
        config.blockDim = dim3(kChainThreads);
        config.stream = s;
        config.attrs = &attr;
        config.numAttrs = 1;
    }
};

template <class Op, int VW, int G> void chain_as(const ChainParams& p, cudaStream_t s) {
    auto kernel = chain_kernel<Op, VW, G>;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    const ChainLaunch c(s);
    const cudaError_t e = cudaLaunchKernelEx(&c.config, kernel, p);
    if (e != cudaSuccess) throw std::runtime_error(std::string("chain of levels: ") + cudaGetErrorString(e));
}

#define GRGX_CHAIN_CASE(OP, VWV, GV) \
    if (vw == VWV && g == GV) {      \
        chain_as<OP, VWV, GV>(p, s); \
        return;                      \
    }
#define GRGX_CHAIN4(OP)        \
    GRGX_CHAIN_CASE(OP, 1, 1)  \
    GRGX_CHAIN_CASE(OP, 2, 1)  \
    GRGX_CHAIN_CASE(OP, 4, 1)  \
    GRGX_CHAIN_CASE(OP, 4, 2)  \
    GRGX_CHAIN_CASE(OP, 4, 4)  \
    GRGX_CHAIN_CASE(OP, 4, 8)  \
    GRGX_CHAIN_CASE(OP, 4, 16) \
    GRGX_CHAIN_CASE(OP, 4, 32)
#define GRGX_CHAIN8(OP)        \
    GRGX_CHAIN_CASE(OP, 1, 1)  \
    GRGX_CHAIN_CASE(OP, 2, 1)  \
    GRGX_CHAIN_CASE(OP, 2, 2)  \
    GRGX_CHAIN_CASE(OP, 2, 4)  \
    GRGX_CHAIN_CASE(OP, 2, 8)  \
    GRGX_CHAIN_CASE(OP, 2, 16) \
    GRGX_CHAIN_CASE(OP, 2, 32)

}  // namespace grgx
