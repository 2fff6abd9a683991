// Pair form of a graph (pair_plan.h): the runs, the blocks and their patterns, found on the device
// from the resident UP CSR the first time a call may use the form.
//
//   runs      prev_kernel walks the nodes with height-0 children in original id order, one thread
//             block per stretch of them, keeping for every height-0 node the last node that had it
//             as a child; a node's largest such predecessor tells whether a run reaches back too
//             far to hold it, and the host cuts the runs in one pass over these numbers.  The
//             nodes of a run hold at most h0 height-0 children between them, so a stretch that
//             starts reading h0 children early sees every predecessor that matters; that no entry
//             was lost is checked afterwards by counting.
//   blocks    two consecutive runs (one, where two would have too many possible pairs)
//   patterns  per block, one thread block counts the pairs in shared memory (direct addressed by
//             the two local node numbers) and numbers the distinct ones
// The passes are a few reads of the edges and of a 16-bit matrix (run x height-0 node) held a batch
// of blocks at a time: about as long as the copy a split form builds.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <vector>

#include "device_plan.h"

namespace grgx {

namespace {

std::atomic<int> g_pair_mode{0};  // 0 by the rules below, 1 wherever possible, 2 never

constexpr int kThreads = 1024;
// Possible pairs of one block: a counter each in shared memory (192 KB).
constexpr long long kMaxPairs = 49152;

// Device scratch of the build, freed on every exit path; take() hands one out for keeps.
struct Temps {
    std::vector<void*> ptrs;
    template <typename T> T* get(size_t count) {
        void* p = nullptr;
        GRGX_CUDA(cudaMalloc(&p, std::max<size_t>(count, 1) * sizeof(T)));
        ptrs.push_back(p);
        return static_cast<T*>(p);
    }
    template <typename T> T* copy(const std::vector<T>& v) {
        T* p = get<T>(v.size());
        if (!v.empty()) GRGX_CUDA(cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice));
        return p;
    }
    void keep(DevicePlan& d, void* p, size_t bytes) {
        d.allocs.push_back(p);
        d.bytes += bytes;
        ptrs.erase(std::remove(ptrs.begin(), ptrs.end(), p), ptrs.end());
    }
    ~Temps() {
        for (void* p : ptrs) cudaFree(p);
    }
};

unsigned blocks_for(unsigned long long items, unsigned perBlock) {
    const unsigned long long b = (items + perBlock - 1) / perBlock, cap = static_cast<unsigned long long>(sm_count()) * 64;
    return static_cast<unsigned>(b < 1 ? 1 : (b > cap ? cap : b));
}

// Height-0 children of each UP row (one warp per row).
__global__ void low_count_kernel(const uint32_t* __restrict__ adj, const long long* __restrict__ off, long long R,
                                 unsigned h0, unsigned* __restrict__ low) {
    const int lane = threadIdx.x & 31;
    const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
    for (long long i = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < R; i += warps) {
        unsigned n = 0;
#pragma unroll 4
        for (long long x = off[i] + lane; x < off[i + 1]; x += 32) n += ((adj[x] & 0x7fffffffu) < h0) ? 1u : 0u;
        for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
        if (lane == 0) low[i] = n;
    }
}

// pv[q] = the last position before q whose node shares a height-0 child with node q (-1: none seen).
// Block b covers positions seg[b] .. seg[b+1]-1 and reads from warm[b] on; last = h0 entries of -1
// for each block.
__global__ void __launch_bounds__(kThreads) prev_kernel(const uint32_t* __restrict__ adj, const long long* __restrict__ off,
                                                        const int* __restrict__ seqRow, const long long* __restrict__ seg,
                                                        const long long* __restrict__ warm, unsigned h0, int* lastAll,
                                                        int* __restrict__ pv) {
    __shared__ int best[3];
    int* last = lastAll + (long long)blockIdx.x * h0;
    if (threadIdx.x < 3) best[threadIdx.x] = -1;
    __syncthreads();
    const long long q0 = seg[blockIdx.x], q1 = seg[blockIdx.x + 1];
    for (long long q = warm[blockIdx.x]; q < q1; q++) {
        const long long r = seqRow[q], e = off[r + 1];
        int m = -1;
        for (long long x = off[r] + threadIdx.x; x < e; x += kThreads) {
            const uint32_t c = adj[x] & 0x7fffffffu;
            if (c < h0) {
                m = max(m, last[c]);
                last[c] = static_cast<int>(q);
            }
        }
        for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
        if ((threadIdx.x & 31) == 0 && m >= 0) atomicMax(&best[q % 3], m);
        // the next node's reads of `last` come after this node's writes; thread 0 clears the slot
        // of node q + 2, which nobody writes before the barrier of node q + 1
        __syncthreads();
        if (threadIdx.x == 0) {
            if (q >= q0) pv[q] = best[q % 3];
            best[(q + 2) % 3] = -1;
        }
    }
}

// par[run - run0][height-0 node] = local number (from 1) of the run's node that has it (one warp
// per node of the batch; the matrix starts at zero).
__global__ void fill_parents_kernel(const uint32_t* __restrict__ adj, const long long* __restrict__ off,
                                    const int* __restrict__ seqRow, const int* __restrict__ runOf,
                                    const int* __restrict__ runStart, long long qBegin, long long qEnd, int run0, unsigned h0,
                                    unsigned short* __restrict__ par) {
    const int lane = threadIdx.x & 31;
    const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
    for (long long q = qBegin + (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); q < qEnd; q += warps) {
        const long long r = seqRow[q], e = off[r + 1];
        const int run = runOf[q];
        const unsigned short local = static_cast<unsigned short>(q - runStart[run] + 1);
        unsigned short* row = par + (long long)(run - run0) * h0;
#pragma unroll 4
        for (long long x = off[r] + lane; x < e; x += 32) {
            const uint32_t c = adj[x] & 0x7fffffffu;
            if (c < h0) row[c] = local;
        }
    }
}

struct PairBlock {
    int run;      // first run
    int q0, q1;   // first position of its runs (q1: of the second)
    int n0, n1;   // nodes in each (n1 = 0: a block of one run)
};

// Counts of the block's pairs in `cnt` (n0+1 x n1+1 entries; the empty pair is not counted);
// returns this thread's count of entries set in the matrix.
__device__ __forceinline__ unsigned count_pairs(const PairBlock& B, int run0, unsigned h0,
                                                const unsigned short* __restrict__ par, unsigned* cnt) {
    const int w = B.n1 + 1, size = (B.n0 + 1) * w;
    for (int k = threadIdx.x; k < size; k += kThreads) cnt[k] = 0;
    __syncthreads();
    const unsigned short* a = par + (long long)(B.run - run0) * h0;
    const unsigned short* b = a + h0;
    unsigned set = 0;
    for (unsigned s = threadIdx.x; s < h0; s += kThreads) {
        const int i = a[s], j = B.n1 ? b[s] : 0;
        set += (i > 0) + (j > 0);
        if (i | j) atomicAdd(&cnt[i * w + j], 1u);
    }
    __syncthreads();
    return set;
}

// npat[block] = distinct pairs + 1 (the empty pair always has number 0); *set += matrix entries set.
__global__ void __launch_bounds__(kThreads) distinct_kernel(const PairBlock* __restrict__ blocks, int run0, unsigned h0,
                                                            const unsigned short* __restrict__ par, unsigned* npat,
                                                            unsigned long long* set) {
    extern __shared__ unsigned cnt[];
    __shared__ unsigned total, found;
    const PairBlock B = blocks[blockIdx.x];
    if (threadIdx.x == 0) total = found = 0;
    const unsigned mine = count_pairs(B, run0, h0, par, cnt);
    unsigned d = 0;
    for (int k = threadIdx.x; k < (B.n0 + 1) * (B.n1 + 1); k += kThreads) d += cnt[k] != 0;
    atomicAdd(&total, d);
    atomicAdd(&found, mine);
    __syncthreads();
    if (threadIdx.x == 0) {
        npat[blockIdx.x] = total + 1;
        atomicAdd(set, static_cast<unsigned long long>(found));
    }
}

// Numbers the block's pairs in (first, second) order and writes the patterns' nodes and every
// height-0 node's pattern.
__global__ void __launch_bounds__(kThreads) emit_kernel(const PairBlock* __restrict__ blocks, int run0, long long blk0,
                                                        unsigned h0, const unsigned short* __restrict__ par,
                                                        const unsigned* __restrict__ patBase, const int* __restrict__ seqNode,
                                                        long long groups, uint2* __restrict__ patNodes,
                                                        unsigned short* __restrict__ ids) {
    extern __shared__ unsigned cnt[];
    __shared__ unsigned sums[kThreads / 32];
    const PairBlock B = blocks[blockIdx.x];
    count_pairs(B, run0, h0, par, cnt);
    const int w = B.n1 + 1, size = (B.n0 + 1) * w;
    const long long blk = blk0 + blockIdx.x;
    const unsigned base = patBase[blockIdx.x];
    // exclusive count of distinct pairs before each thread's contiguous share of the table
    const int per = (size + kThreads - 1) / kThreads, k0 = threadIdx.x * per, k1 = min(size, k0 + per);
    unsigned mine = 0;
    for (int k = k0; k < k1; k++) mine += cnt[k] != 0;
    unsigned inc = mine;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(0xffffffffu, inc, o);
        if ((threadIdx.x & 31) >= (unsigned)o) inc += t;
    }
    if ((threadIdx.x & 31) == 31) sums[threadIdx.x >> 5] = inc;
    __syncthreads();
    unsigned at = 1 + inc - mine;  // number 0 is the empty pair
    for (unsigned v = 0; v < (threadIdx.x >> 5); v++) at += sums[v];
    if (threadIdx.x == 0) patNodes[base] = make_uint2(INVALID_NODE, INVALID_NODE);
    for (int k = k0; k < k1; k++) {
        if (cnt[k] == 0) continue;
        const int i = k / w, j = k % w;
        patNodes[base + at] = make_uint2(i ? static_cast<unsigned>(seqNode[B.q0 + i - 1]) : INVALID_NODE,
                                         j ? static_cast<unsigned>(seqNode[B.q1 + j - 1]) : INVALID_NODE);
        cnt[k] = at++;
    }
    __syncthreads();
    const unsigned short* a = par + (long long)(B.run - run0) * h0;
    const unsigned short* b = a + h0;
    for (unsigned s = threadIdx.x; s < h0; s += kThreads) {
        const int i = a[s], j = B.n1 ? b[s] : 0;
        const unsigned p = (i | j) ? cnt[i * w + j] : 0u;
        ids[(((long long)(s >> 5) * groups + (blk >> 2)) * 32 + (s & 31)) * 4 + (blk & 3)] = static_cast<unsigned short>(p);
    }
}

// The runs, as first positions (with the end), from each position's predecessor.
std::vector<int> cut_runs(const std::vector<int>& pv) {
    std::vector<int> start;
    const int most = static_cast<int>(kMaxPairs) / 2 - 1;
    for (size_t q = 0; q < pv.size(); q++)
        if (start.empty() || pv[q] >= start.back() || static_cast<int>(q) - start.back() >= most)
            start.push_back(static_cast<int>(q));
    start.push_back(static_cast<int>(pv.size()));
    return start;
}

void build_pair_plan(DevicePlan& d) {
    PairPlan& P = d.pair;
    if (d.num_levels < 2 || d.up_off.size() < 2) return;
    const long long h0 = static_cast<long long>(d.level_begin[1]);
    const long long n = static_cast<long long>(d.level_begin[d.num_levels]);
    const long long R = n - h0;
    const bool forced = g_pair_mode.load() == 1;
    // 16-bit matrix entries and 32-bit positions; small graphs stay as they are
    if (d.up_off.back() < (forced ? 1 : kPairMinEdges) || h0 > 0x3fffffff) return;
    Temps tmp;
    long long* dOff = reinterpret_cast<long long*>(tmp.copy(d.up_off));
    unsigned* dLow = tmp.get<unsigned>(R);
    low_count_kernel<<<blocks_for(R, 8), 256>>>(d.up.adj, dOff, R, static_cast<unsigned>(h0), dLow);
    GRGX_CUDA(cudaGetLastError());
    std::vector<unsigned> low(R);
    std::vector<uint32_t> old2new(n);
    GRGX_CUDA(cudaMemcpy(low.data(), dLow, R * sizeof(unsigned), cudaMemcpyDeviceToHost));
    GRGX_CUDA(cudaMemcpy(old2new.data(), d.old2new, n * sizeof(uint32_t), cudaMemcpyDeviceToHost));

    // ---- the nodes with height-0 children, in original id order --------------------------------
    std::vector<int> seqRow, seqNode;
    std::vector<long long> cum(1, 0);
    for (long long v = 0; v < n; v++) {
        const long long r = static_cast<long long>(old2new[v]) - h0;
        if (r < 0 || low[r] == 0) continue;
        seqRow.push_back(static_cast<int>(r));
        seqNode.push_back(static_cast<int>(old2new[v]));
        cum.push_back(cum.back() + low[r]);
    }
    const long long Q = static_cast<long long>(seqRow.size()), E0 = cum.back();
    if (Q == 0 || E0 < (forced ? 1 : kPairMinEdges) || 2 * E0 < d.up_off.back()) return;

    // ---- runs ------------------------------------------------------------------------------------
    // stretches of at least 16 average haplotype sets, one thread block each
    const long long S = std::max<long long>(1, std::min<long long>({2LL * sm_count(), E0 / h0 / 16, (1LL << 30) / h0 + 1, Q}));
    std::vector<long long> seg, warm;
    for (long long b = 0; b <= S; b++)
        seg.push_back(b == S ? Q : std::lower_bound(cum.begin(), cum.end(), E0 * b / S) - cum.begin());
    for (long long b = 0; b < S; b++)
        warm.push_back(std::lower_bound(cum.begin(), cum.end(), std::max<long long>(0, cum[seg[b]] - h0)) -
                       cum.begin());
    const int* dRow = tmp.copy(seqRow);
    const int* dNode = tmp.copy(seqNode);
    std::vector<int> pv(Q);
    {
        Temps t2;
        const long long* dSeg = t2.copy(seg);
        const long long* dWarm = t2.copy(warm);
        int* last = t2.get<int>(S * h0);
        int* dPv = t2.get<int>(Q);
        GRGX_CUDA(cudaMemsetAsync(last, 0xff, S * h0 * sizeof(int), cudaStreamLegacy));
        prev_kernel<<<static_cast<unsigned>(S), kThreads>>>(d.up.adj, dOff, dRow, dSeg, dWarm, static_cast<unsigned>(h0), last,
                                                            dPv);
        GRGX_CUDA(cudaGetLastError());
        GRGX_CUDA(cudaMemcpy(pv.data(), dPv, Q * sizeof(int), cudaMemcpyDeviceToHost));
    }
    const std::vector<int> run = cut_runs(pv);
    const int nruns = static_cast<int>(run.size()) - 1;

    // ---- blocks ----------------------------------------------------------------------------------
    std::vector<PairBlock> blocks;
    for (int r = 0; r < nruns;) {
        PairBlock B{r, run[r], 0, run[r + 1] - run[r], 0};
        if (r + 1 < nruns && (B.n0 + 1LL) * (run[r + 2] - run[r + 1] + 1) <= kMaxPairs) {
            B.q1 = run[r + 1];
            B.n1 = run[r + 2] - run[r + 1];
        }
        r += B.n1 ? 2 : 1;
        blocks.push_back(B);
    }
    const long long nblk = static_cast<long long>(blocks.size());
    if (!forced && static_cast<double>(nblk) * h0 > kPairMaxCost * static_cast<double>(E0)) return;

    // ---- patterns, a batch of blocks at a time -----------------------------------------------------
    std::vector<int> runOf(Q);
    for (int r = 0; r < nruns; r++) std::fill(runOf.begin() + run[r], runOf.begin() + run[r + 1], r);
    const int* dRunOf = tmp.copy(runOf);
    const int* dRun = tmp.copy(run);
    const PairBlock* dBlocks = tmp.copy(blocks);
    const long long groups = (nblk + 3) / 4;
    const long long tiles = (h0 + 127) / 128 * 4;  // whole groups of 128 nodes: a warp's largest share
    const size_t idBytes = static_cast<size_t>(tiles) * groups * 128 * sizeof(unsigned short);
    unsigned short* ids = tmp.get<unsigned short>(idBytes / sizeof(unsigned short));
    GRGX_CUDA(cudaMemsetAsync(ids, 0, idBytes, cudaStreamLegacy));
    const long long batch = std::max<long long>(1, std::min(nblk, (1LL << 27) / h0));
    unsigned short* par = tmp.get<unsigned short>(2 * batch * h0);
    unsigned* dNpat = tmp.get<unsigned>(batch);
    unsigned* dBase = tmp.get<unsigned>(batch);
    unsigned long long* dSet = tmp.get<unsigned long long>(1);
    GRGX_CUDA(cudaMemsetAsync(dSet, 0, sizeof(unsigned long long), cudaStreamLegacy));
    GRGX_CUDA(cudaFuncSetAttribute(distinct_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxPairs * 4));
    GRGX_CUDA(cudaFuncSetAttribute(emit_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxPairs * 4));
    std::vector<long long> patBase(1, 0);
    struct Part {
        uint2* nodes;
        long long count;
    };
    std::vector<Part> parts;
    for (long long b0 = 0; b0 < nblk; b0 += batch) {
        const long long b1 = std::min(nblk, b0 + batch), nb = b1 - b0;
        const PairBlock& last = blocks[b1 - 1];
        const int run0 = blocks[b0].run, run1 = last.run + (last.n1 ? 2 : 1);
        const unsigned H = static_cast<unsigned>(h0);
        GRGX_CUDA(cudaMemsetAsync(par, 0, static_cast<size_t>(run1 - run0) * h0 * sizeof(unsigned short), cudaStreamLegacy));
        fill_parents_kernel<<<blocks_for(run[run1] - run[run0], 8), 256>>>(d.up.adj, dOff, dRow, dRunOf, dRun, run[run0],
                                                                           run[run1], run0, H, par);
        size_t most = 0;
        for (long long b = b0; b < b1; b++)
            most = std::max<size_t>(most, (blocks[b].n0 + 1LL) * (blocks[b].n1 + 1) * sizeof(unsigned));
        distinct_kernel<<<static_cast<unsigned>(nb), kThreads, most>>>(dBlocks + b0, run0, H, par, dNpat, dSet);
        GRGX_CUDA(cudaGetLastError());
        std::vector<unsigned> npat(nb), rel(nb);
        GRGX_CUDA(cudaMemcpy(npat.data(), dNpat, nb * sizeof(unsigned), cudaMemcpyDeviceToHost));
        unsigned long long total = 0;
        for (long long b = 0; b < nb; b++) {
            rel[b] = static_cast<unsigned>(total);
            total += npat[b];
            patBase.push_back(patBase.back() + npat[b]);
        }
        // worth it so far?  (and pattern rows are numbered in 31 bits)
        if (patBase.back() >= 0x7fffffffLL ||
            (!forced && b0 == 0 && nb * h0 + kPairPatternCost * static_cast<double>(total) >
                                       kPairMaxCost * static_cast<double>(cum[run[run1]] - cum[run[run0]])))
            return;
        GRGX_CUDA(cudaMemcpy(dBase, rel.data(), nb * sizeof(unsigned), cudaMemcpyHostToDevice));
        parts.push_back({tmp.get<uint2>(total), static_cast<long long>(total)});
        emit_kernel<<<static_cast<unsigned>(nb), kThreads, most>>>(dBlocks + b0, run0, b0, H, par, dBase, dNode, groups,
                                                                   parts.back().nodes, ids);
        GRGX_CUDA(cudaGetLastError());
    }
    unsigned long long set = 0;
    GRGX_CUDA(cudaMemcpy(&set, dSet, sizeof(set), cudaMemcpyDeviceToHost));
    // every edge has its entry: no height-0 node has two parents in one run, or the same one twice
    if (static_cast<long long>(set) != E0) return;
    P.npat = patBase.back();
    if (!forced && nblk * h0 + kPairPatternCost * static_cast<double>(P.npat) > kPairMaxCost * static_cast<double>(E0)) return;

    uint2* nodes = tmp.get<uint2>(P.npat);
    long long at = 0;
    for (const Part& p : parts) {
        GRGX_CUDA(cudaMemcpyAsync(nodes + at, p.nodes, p.count * sizeof(uint2), cudaMemcpyDeviceToDevice, cudaStreamLegacy));
        at += p.count;
    }
    std::vector<unsigned> base(groups * 4, 0);  // padding blocks point at an empty pair
    for (long long b = 0; b < nblk; b++) base[b] = static_cast<unsigned>(patBase[b]);
    for (long long b = nblk; b < groups * 4; b++) base[b] = base[nblk - 1];
    unsigned* dB = tmp.copy(base);
    GRGX_CUDA(cudaStreamSynchronize(cudaStreamLegacy));
    tmp.keep(d, ids, idBytes);
    tmp.keep(d, nodes, P.npat * sizeof(uint2));
    tmp.keep(d, dB, base.size() * sizeof(unsigned));
    P.h0 = h0;
    P.nblk = nblk;
    P.pat_base = std::move(patBase);
    P.base = dB;
    P.pat_nodes = nodes;
    P.ids = ids;
    P.usable = true;
}

}  // namespace

void set_pair_mode(int mode) { g_pair_mode.store(mode); }

bool use_pair_form(grgx_graph* g, DevicePlan* dp, const Layout&) {
    const int mode = g_pair_mode.load();
    if (mode == 2) return false;
    std::lock_guard<std::mutex> lk(g->mu);
    if (!dp->pair.tried) {
        dp->pair.tried = true;
        try {
            build_pair_plan(*dp);
        } catch (const Error& e) {
            // no memory for it: the other forms need none of this
            if (e.code != GRGX_ERR_OUT_OF_MEMORY) throw;
            cudaGetLastError();
        }
    }
    return dp->pair.usable;
}

}  // namespace grgx
