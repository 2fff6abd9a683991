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
#include <cub/device/device_radix_sort.cuh>
#include <new>
#include <vector>

#include "device_plan.h"

namespace grgx {

namespace {

std::atomic<int> g_pair_mode{0};  // 0 by the rules below, 1 wherever possible, 2 never
std::atomic<long long> g_most_rows{kPairMostRows};

constexpr int kThreads = 1024;
// Possible pairs of one block: a counter each in shared memory (192 KB).
constexpr long long kMaxPairs = 49152;

// Device scratch of the build, freed on every exit path; take() hands one out for keeps.
struct Temps {
    std::vector<void*> ptrs;
    template <typename T> T* get(size_t count) {
        void* p = plan_alloc(count * sizeof(T));
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
    void release(void* p) {
        cudaFree(p);
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
        // (a node's children are distinct: the loads of a batch need not wait for its stores)
        for (long long x = off[r] + threadIdx.x; x < e; x += 8 * kThreads) {
            uint32_t c[8];
            int l[8];
#pragma unroll
            for (int u = 0; u < 8; u++) c[u] = (x + u * kThreads < e) ? adj[x + u * kThreads] & 0x7fffffffu : 0xffffffffu;
#pragma unroll
            for (int u = 0; u < 8; u++) l[u] = c[u] < h0 ? last[c[u]] : -1;
#pragma unroll
            for (int u = 0; u < 8; u++) {
                m = max(m, l[u]);
                if (c[u] < h0) last[c[u]] = static_cast<int>(q);
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

// What emit_kernel writes (null: left out).  Patterns are numbered from patBase[block] on.
struct PairOut {
    const unsigned* patBase;
    const int* seqNode;     // new id at each position
    uint2* nodes;           // each pattern's parents
    unsigned* count;        // ... and height-0 nodes
    unsigned short* ids;    // DOWN: each height-0 node's pattern in each block
    long long groups;
    unsigned *keys, *vals;  // UP: (pattern, height-0 node), block by block
};

// Numbers the block's pairs in (first, second) order.
__global__ void __launch_bounds__(kThreads) emit_kernel(const PairBlock* __restrict__ blocks, int run0, long long blk0,
                                                        unsigned h0, const unsigned short* __restrict__ par,
                                                        const PairOut out) {
    extern __shared__ unsigned cnt[];
    __shared__ unsigned sums[kThreads / 32];
    const PairBlock B = blocks[blockIdx.x];
    const unsigned set = count_pairs(B, run0, h0, par, cnt);
    (void)set;
    const int w = B.n1 + 1, size = (B.n0 + 1) * w;
    const long long blk = blk0 + blockIdx.x;
    const unsigned base = out.patBase[blockIdx.x];
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
    if (threadIdx.x == 0 && out.nodes) out.nodes[base] = make_uint2(INVALID_NODE, INVALID_NODE);
    for (int k = k0; k < k1; k++) {
        if (cnt[k] == 0) continue;
        const int i = k / w, j = k % w;
        if (out.nodes)
            out.nodes[base + at] = make_uint2(i ? static_cast<unsigned>(out.seqNode[B.q0 + i - 1]) : INVALID_NODE,
                                              j ? static_cast<unsigned>(out.seqNode[B.q1 + j - 1]) : INVALID_NODE);
        if (out.count) out.count[base + at] = cnt[k];
        cnt[k] = at++;
    }
    __syncthreads();
    const unsigned short* a = par + (long long)(B.run - run0) * h0;
    const unsigned short* b = a + h0;
    for (unsigned s = threadIdx.x; s < h0; s += kThreads) {
        const int i = a[s], j = B.n1 ? b[s] : 0;
        const unsigned p = (i | j) ? cnt[i * w + j] : 0u;
        if (out.ids)
            out.ids[(((long long)(s >> 5) * out.groups + (blk >> 2)) * 32 + (s & 31)) * 4 + (blk & 3)] =
                static_cast<unsigned short>(p);
        if (out.keys) {
            // height-0 nodes with the empty pair are sorted past the others
            out.keys[(long long)blockIdx.x * h0 + s] = p ? base + p : 0x7fffffffu;
            out.vals[(long long)blockIdx.x * h0 + s] = s;
        }
    }
}

// (position, table row) pairs: the rows' first parents, then their second ones; none = `none`.
__global__ void node_pairs_kernel(const uint2* __restrict__ nodes, long long rows, unsigned none,
                                  unsigned* __restrict__ keys, unsigned* __restrict__ vals) {
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < rows; p += (long long)gridDim.x * blockDim.x) {
        const uint2 nd = nodes[p];
        keys[p] = min(nd.x, none);
        keys[rows + p] = min(nd.y, none);
        vals[p] = vals[rows + p] = static_cast<unsigned>(p);
    }
}

// The lists' ids: the children below h0 of the UP rows' edges from[i].x .. from[i].y - 1 (whose first ids
// carry a row mark).
__global__ void few_ids_kernel(const PairList* __restrict__ lists, const longlong2* __restrict__ from, long long count,
                               unsigned h0, const uint32_t* __restrict__ adj, uint32_t* __restrict__ out) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (long long)gridDim.x * blockDim.x) {
        const PairList l = lists[i];
        int k = 0;
        for (long long x = from[i].x; x < from[i].y && k < l.len; x++) {
            const uint32_t id = adj[x] & 0x7fffffffu;
            if (id < h0) out[l.e0 + k++] = id;
        }
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

// Pairs sorted by key (stable), on the legacy stream; returns the sorted keys and values.
void sort_pairs(Temps& tmp, unsigned*& keys, unsigned*& vals, unsigned* keys2, unsigned* vals2, long long count, int bits) {
    cub::DoubleBuffer<unsigned> k(keys, keys2), v(vals, vals2);
    size_t bytes = 0;
    GRGX_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, bytes, k, v, count, 0, bits));
    unsigned char* t = tmp.get<unsigned char>(bytes);
    GRGX_CUDA(cub::DeviceRadixSort::SortPairs(t, bytes, k, v, count, 0, bits));
    keys = k.Current();
    vals = v.Current();
    tmp.release(t);
}

// The UP lists, by segments: the patterns' pieces (a table row each), the nodes' table rows.  False: more
// rows than lists can number.
bool build_up_lists(DevicePlan& d, Temps& tmp, const std::vector<long long>& patBase, const std::vector<unsigned>& counts,
                    uint32_t* patAdj, long long patEdges, const uint2* nodes) {
    PairPlan& P = d.pair;
    const long long h0 = static_cast<long long>(d.level_begin[1]);
    const long long Q = static_cast<long long>(P.seq.size()), nblk = static_cast<long long>(P.blocks.size());
    std::vector<uint2> patNodes(patBase.back());
    GRGX_CUDA(cudaMemcpy(patNodes.data(), nodes, patNodes.size() * sizeof(uint2), cudaMemcpyDeviceToHost));

    // Stable sort of lists by length, longest first (a counting sort).
    auto longest_first = [](PairList* v, size_t count) {
        int most = 0;
        for (size_t i = 0; i < count; i++) most = std::max(most, v[i].len);
        std::vector<size_t> at(most + 2, 0);
        for (size_t i = 0; i < count; i++) at[most - v[i].len + 1]++;
        for (int l = 0; l <= most; l++) at[l + 1] += at[l];
        std::vector<PairList> sorted(count);
        for (size_t i = 0; i < count; i++) sorted[at[most - v[i].len]++] = v[i];
        std::copy(sorted.begin(), sorted.end(), v);
    };
    const long long nseg = (nblk + kPairSegment - 1) / kPairSegment;
    auto first_pattern = [&](long long s) { return patBase[std::min(nblk, s * kPairSegment)]; };
    auto first_position = [&](long long s) {
        return s * kPairSegment < nblk ? static_cast<long long>(P.blocks[s * kPairSegment].q0) : Q;
    };
    auto pieces_of = [](long long c) { return (c + kPairPiece - 1) / kPairPiece; };
    // position of each UP row in the sequence; a node's patterns are all of its own segment
    std::vector<unsigned> posOf(d.up_off.size(), 0);
    for (long long q = 0; q < Q; q++) posOf[P.seq[q]] = static_cast<unsigned>(q);
    auto few = [&](long long q) { return P.low[P.seq[q]] <= kPairFew; };
    auto position = [&](unsigned node) { return node == INVALID_NODE ? INVALID_NODE : posOf[node - h0]; };
    std::vector<PairPlan::Segment> segments(nseg + 1);
    std::vector<long long> edge0(nseg + 1, 0), sub0(nseg + 1, 0), nedge0(nseg + 1, 0);
    std::vector<unsigned> deg(Q, 0);
    run_threads(nseg, [&](long long s) {
        PairPlan::Segment& next = segments[s + 1];
        for (long long p = first_pattern(s); p < first_pattern(s + 1); p++) {
            const long long n = pieces_of(counts[p]);
            edge0[s + 1] += counts[p];
            next.pat0 += n;
            for (unsigned q : {position(patNodes[p].x), position(patNodes[p].y)})
                if (q != INVALID_NODE) deg[q] += static_cast<unsigned>(n);
        }
        for (long long q = first_position(s); q < first_position(s + 1); q++) {
            const long long n = pieces_of(deg[q]);
            nedge0[s + 1] += deg[q];
            if (few(q)) continue;
            next.node0 += n;
            next.top0 += n > 1;
            sub0[s + 1] += n > 1 ? n : 0;
        }
        next.row0 = next.pat0 + sub0[s + 1];
    });
    for (long long s = 0; s < nseg; s++) {
        edge0[s + 1] += edge0[s];
        nedge0[s + 1] += nedge0[s];
        sub0[s + 1] += sub0[s];
        segments[s + 1].row0 += segments[s].row0;
        segments[s + 1].pat0 += segments[s].pat0;
        segments[s + 1].node0 += segments[s].node0;
        segments[s + 1].top0 += segments[s].top0;
    }
    const long long rows = segments.back().row0, ne = nedge0.back();
    GRGX_CHECK(edge0.back() == patEdges, GRGX_ERR_CUDA, "pair form edge count mismatch");
    if (rows >= g_most_rows.load()) return false;
    std::vector<PairList> patLists(segments.back().pat0), nodeLists(segments.back().node0), topLists(segments.back().top0);
    std::vector<uint2> rowNodes(rows, uint2{INVALID_NODE, INVALID_NODE});
    std::vector<uint32_t> topAdj(sub0.back());
    run_threads(nseg, [&](long long s) {
        const PairPlan::Segment& a = segments[s];
        long long e = edge0[s], row = a.row0, at = a.pat0;
        auto cut = [](PairList* out, long long e, long long c, long long n, long long i, int dst) {
            const long long k0 = c * i / n, k1 = c * (i + 1) / n;
            *out = {e + k0, static_cast<int>(k1 - k0), dst};
        };
        for (long long p = first_pattern(s); p < first_pattern(s + 1); p++) {
            const long long n = pieces_of(counts[p]);
            for (long long i = 0; i < n; i++, row++) {
                cut(&patLists[at++], e, counts[p], n, i, ~static_cast<int>(row));
                rowNodes[row] = uint2{position(patNodes[p].x), position(patNodes[p].y)};
            }
            e += counts[p];
        }
        e = nedge0[s];
        long long node = a.node0, top = a.top0, sub = sub0[s];
        for (long long q = first_position(s); q < first_position(s + 1); q++) {
            const long long n = few(q) ? 0 : pieces_of(deg[q]);
            if (n > 1) topLists[top++] = {sub, static_cast<int>(n), P.seq[q]};
            for (long long i = 0; i < n; i++) {
                cut(&nodeLists[node++], e, deg[q], n, i, n > 1 ? ~static_cast<int>(row) : P.seq[q]);
                if (n > 1) topAdj[sub++] = static_cast<uint32_t>(row++);
            }
            e += deg[q];
        }
        longest_first(patLists.data() + a.pat0, static_cast<size_t>(at - a.pat0));
        longest_first(nodeLists.data() + a.node0, static_cast<size_t>(node - a.node0));
    });

    std::vector<PairList> fewLists;
    for (long long q = 0; q < Q; q++)
        if (few(q)) fewLists.push_back({0, static_cast<int>(P.low[P.seq[q]]), P.seq[q]});
    longest_first(fewLists.data(), fewLists.size());
    std::vector<longlong2> fewFrom(fewLists.size());
    long long fewEdges = 0;
    for (size_t i = 0; i < fewLists.size(); i++) {
        fewFrom[i] = {static_cast<long long>(d.up_off[fewLists[i].out]), static_cast<long long>(d.up_off[fewLists[i].out + 1])};
        fewLists[i].e0 = fewEdges;
        fewEdges += fewLists[i].len;
    }

    const uint2* dRowNodes = tmp.copy(rowNodes);
    unsigned *keys = tmp.get<unsigned>(2 * rows), *vals = tmp.get<unsigned>(2 * rows);
    unsigned *keys2 = tmp.get<unsigned>(2 * rows), *vals2 = tmp.get<unsigned>(2 * rows);
    node_pairs_kernel<<<blocks_for(rows, 256), 256>>>(dRowNodes, rows, static_cast<unsigned>(Q), keys, vals);
    GRGX_CUDA(cudaGetLastError());
    int bits = 1;
    while ((1LL << bits) <= Q) bits++;
    sort_pairs(tmp, keys, vals, keys2, vals2, 2 * rows, bits);
    uint32_t* adj = tmp.get<uint32_t>(ne);
    GRGX_CUDA(cudaMemcpyAsync(adj, vals, ne * sizeof(uint32_t), cudaMemcpyDeviceToDevice, cudaStreamLegacy));
    if (!fewLists.empty()) {
        P.few_lists = tmp.copy(fewLists);
        P.few_adj = tmp.get<uint32_t>(fewEdges);
        const longlong2* from = tmp.copy(fewFrom);
        few_ids_kernel<<<blocks_for(static_cast<long long>(fewLists.size()), 256), 256>>>(
            P.few_lists, from, static_cast<long long>(fewLists.size()), static_cast<unsigned>(h0), d.up.adj, P.few_adj);
        GRGX_CUDA(cudaGetLastError());
    }
    P.nfew = static_cast<long long>(fewLists.size());
    P.pat_lists = tmp.copy(patLists);
    P.node_lists = tmp.copy(nodeLists);
    P.top_lists = tmp.copy(topLists);
    P.top_adj = tmp.copy(topAdj);
    P.pat_adj = patAdj;
    P.node_adj = adj;
    GRGX_CUDA(cudaStreamSynchronize(cudaStreamLegacy));
    tmp.keep(d, patAdj, patEdges * sizeof(uint32_t));
    tmp.keep(d, adj, ne * sizeof(uint32_t));
    tmp.keep(d, P.top_adj, topAdj.size() * sizeof(uint32_t));
    tmp.keep(d, P.pat_lists, patLists.size() * sizeof(PairList));
    tmp.keep(d, P.node_lists, nodeLists.size() * sizeof(PairList));
    tmp.keep(d, P.top_lists, topLists.size() * sizeof(PairList));
    if (P.nfew > 0) {
        tmp.keep(d, P.few_lists, fewLists.size() * sizeof(PairList));
        tmp.keep(d, P.few_adj, fewEdges * sizeof(uint32_t));
    }
    P.segments = std::move(segments);
    return true;
}

// Everything about the form that needs one pass over the height-0 edges: the analysis on the first
// call, and the arrays of the direction asked for (none where only that direction is too large for them).
// False: the form is not worth using, or impossible.
// What a build that fails leaves behind is at most the finished analysis, for the next one.
bool build_pair_plan(DevicePlan& d, bool down) {
    PairPlan& P = d.pair;
    const bool forced = g_pair_mode.load() == 1 || P.usable;
    if (d.num_levels < 2 || d.up_off.size() < 2) return false;
    const long long h0 = static_cast<long long>(d.level_begin[1]);
    const long long n = static_cast<long long>(d.level_begin[d.num_levels]);
    const long long R = n - h0;
    // 16-bit matrix entries and 32-bit positions; small graphs stay as they are
    if (d.up_off.back() < (forced ? 1 : kPairMinEdges) || h0 > 0x3fffffff) return false;
    const unsigned H = static_cast<unsigned>(h0);
    Temps tmp;
    const long long* dOff = reinterpret_cast<long long*>(tmp.copy(d.up_off));
    if (P.seq.empty()) {
        std::vector<unsigned> low = count_low_children(d);
        std::vector<uint32_t> old2new(n);
        GRGX_CUDA(cudaMemcpy(old2new.data(), d.old2new, n * sizeof(uint32_t), cudaMemcpyDeviceToHost));
        // the nodes with height-0 children, in original id order
        std::vector<int> seq;
        for (long long v = 0; v < n; v++) {
            const long long r = static_cast<long long>(old2new[v]) - h0;
            if (r >= 0 && low[r]) seq.push_back(static_cast<int>(r));
        }
        P.low = std::move(low);
        P.seq = std::move(seq);
    }
    const long long Q = static_cast<long long>(P.seq.size());
    std::vector<long long> cum(1, 0);
    for (int r : P.seq) cum.push_back(cum.back() + P.low[r]);
    const long long E0 = cum.back();
    if (Q == 0 || E0 < (forced ? 1 : kPairMinEdges) || 2 * E0 < d.up_off.back()) return false;
    const int* dRow = tmp.copy(P.seq);

    if (P.blocks.empty()) {
        // ---- runs: stretches of at least 6 average haplotype sets, one thread block each -----------
        const long long S =
            std::max<long long>(1, std::min<long long>({2LL * sm_count(), E0 / h0 / 6, (1LL << 30) / h0 + 1, Q}));
        std::vector<long long> seg, warm;
        for (long long b = 0; b <= S; b++)
            seg.push_back(b == S ? Q : std::lower_bound(cum.begin(), cum.end(), E0 * b / S) - cum.begin());
        for (long long b = 0; b < S; b++)
            warm.push_back(std::lower_bound(cum.begin(), cum.end(), std::max<long long>(0, cum[seg[b]] - h0)) - cum.begin());
        std::vector<int> pv(Q);
        {
            Temps t2;
            const long long* dSeg = t2.copy(seg);
            const long long* dWarm = t2.copy(warm);
            int* last = t2.get<int>(S * h0);
            int* dPv = t2.get<int>(Q);
            GRGX_CUDA(cudaMemsetAsync(last, 0xff, S * h0 * sizeof(int), cudaStreamLegacy));
            prev_kernel<<<static_cast<unsigned>(S), kThreads>>>(d.up.adj, dOff, dRow, dSeg, dWarm, H, last, dPv);
            GRGX_CUDA(cudaGetLastError());
            GRGX_CUDA(cudaMemcpy(pv.data(), dPv, Q * sizeof(int), cudaMemcpyDeviceToHost));
        }
        std::vector<int> run = cut_runs(pv);
        // ---- blocks --------------------------------------------------------------------------------
        const int nruns = static_cast<int>(run.size()) - 1;
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
        P.run = std::move(run);
        P.blocks = std::move(blocks);
    }
    const std::vector<int>& run = P.run;
    const std::vector<PairBlock>& blocks = P.blocks;
    const int nruns = static_cast<int>(run.size()) - 1;
    const long long nblk = static_cast<long long>(blocks.size());
    const double edges = static_cast<double>(E0);
    if (!forced && static_cast<double>(nblk) * h0 > kPairMaxCost * edges) return false;

    // ---- patterns, a batch of blocks at a time -------------------------------------------------------
    std::vector<int> runOf(Q), seqNode(Q);
    for (int r = 0; r < nruns; r++) std::fill(runOf.begin() + run[r], runOf.begin() + run[r + 1], r);
    for (long long q = 0; q < Q; q++) seqNode[q] = static_cast<int>(P.seq[q] + h0);
    const int* dRunOf = tmp.copy(runOf);
    const int* dRun = tmp.copy(run);
    const int* dNode = tmp.copy(seqNode);
    const PairBlock* dBlocks = tmp.copy(blocks);
    const long long groups = (nblk + 3) / 4;
    const long long tiles = (h0 / kPairTile + 2) * (kPairTile / 32);  // padded: see kPairTile
    const long long batch = std::max<long long>(1, std::min(nblk, (1LL << 27) / h0));
    const size_t idBytes = static_cast<size_t>(tiles) * groups * 32 * 4 * sizeof(unsigned short);
    PairOut out{};
    out.seqNode = dNode;
    out.groups = groups;
    uint32_t* upAdj = nullptr;
    unsigned *keys = nullptr, *vals = nullptr, *keys2 = nullptr, *vals2 = nullptr;
    long long upEdges = 0;
    if (down) {
        out.ids = tmp.get<unsigned short>(idBytes / sizeof(unsigned short));
        GRGX_CUDA(cudaMemsetAsync(out.ids, 0, idBytes, cudaStreamLegacy));
    } else {
        upAdj = tmp.get<uint32_t>(nblk * h0);
        keys = tmp.get<unsigned>(batch * h0);
        vals = tmp.get<unsigned>(batch * h0);
        keys2 = tmp.get<unsigned>(batch * h0);
        vals2 = tmp.get<unsigned>(batch * h0);
    }
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
    std::vector<unsigned> counts;  // UP: each pattern's height-0 nodes
    for (long long b0 = 0; b0 < nblk; b0 += batch) {
        const long long b1 = std::min(nblk, b0 + batch), nb = b1 - b0;
        const PairBlock& last = blocks[b1 - 1];
        const int run0 = blocks[b0].run, run1 = last.run + (last.n1 ? 2 : 1);
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
        long long total = 0;
        for (long long b = 0; b < nb; b++) {
            rel[b] = static_cast<unsigned>(total);
            total += npat[b];
            patBase.push_back(patBase.back() + npat[b]);
        }
        // worth it so far?  (and pattern rows are numbered in 31 bits)
        if (patBase.back() >= 0x7fffffffLL ||
            (!forced && b0 == 0 && nb * h0 + kPairPatternCost * static_cast<double>(total) >
                                       kPairMaxCost * static_cast<double>(cum[run[run1]] - cum[run[run0]])))
            return false;
        GRGX_CUDA(cudaMemcpy(dBase, rel.data(), nb * sizeof(unsigned), cudaMemcpyHostToDevice));
        out.patBase = dBase;
        parts.push_back({tmp.get<uint2>(total), total});
        out.nodes = parts.back().nodes;
        if (!down) {
            out.keys = keys;
            out.vals = vals;
            out.count = tmp.get<unsigned>(total);
            GRGX_CUDA(cudaMemsetAsync(out.count, 0, total * sizeof(unsigned), cudaStreamLegacy));
        }
        emit_kernel<<<static_cast<unsigned>(nb), kThreads, most>>>(dBlocks + b0, run0, b0, H, par, out);
        GRGX_CUDA(cudaGetLastError());
        if (!down) {
            const size_t at = counts.size();
            counts.resize(at + total);
            GRGX_CUDA(cudaMemcpy(counts.data() + at, out.count, total * sizeof(unsigned), cudaMemcpyDeviceToHost));
            long long have = 0;
            for (size_t p = at; p < counts.size(); p++) have += counts[p];
            unsigned *k = keys, *v = vals;
            int bits = 1;
            while ((1LL << bits) <= total) bits++;
            // (the empty pair's key has every bit set: it sorts last within any number of bits)
            sort_pairs(tmp, k, v, keys2, vals2, nb * h0, bits);
            GRGX_CUDA(cudaMemcpyAsync(upAdj + upEdges, v, have * sizeof(uint32_t), cudaMemcpyDeviceToDevice, cudaStreamLegacy));
            upEdges += have;
            tmp.release(out.count);
        }
    }
    unsigned long long set = 0;
    GRGX_CUDA(cudaMemcpy(&set, dSet, sizeof(set), cudaMemcpyDeviceToHost));
    // every edge has its entry: no height-0 node has two parents in one run, or the same one twice
    if (static_cast<long long>(set) != E0) return false;
    const long long npat = patBase.back();
    if (!forced && nblk * h0 + kPairPatternCost * static_cast<double>(npat) > kPairMaxCost * edges) return false;

    uint2* nodes = tmp.get<uint2>(npat);
    long long at = 0;
    for (const Part& p : parts) {
        GRGX_CUDA(cudaMemcpyAsync(nodes + at, p.nodes, p.count * sizeof(uint2), cudaMemcpyDeviceToDevice, cudaStreamLegacy));
        at += p.count;
    }
    if (down) {
        std::vector<unsigned> base(groups * 4);
        for (long long b = 0; b < groups * 4; b++)  // padding blocks point at an empty pair
            base[b] = static_cast<unsigned>(patBase[std::min(b, nblk - 1)]);
        unsigned* dB = tmp.copy(base);
        GRGX_CUDA(cudaStreamSynchronize(cudaStreamLegacy));
        tmp.keep(d, out.ids, idBytes);
        tmp.keep(d, nodes, npat * sizeof(uint2));
        tmp.keep(d, dB, base.size() * sizeof(unsigned));
        P.base = dB;
        P.pat_nodes = nodes;
        P.ids = out.ids;
        P.down_built = true;
    } else {
        build_up_internal(d, P.low);
        if (!build_up_lists(d, tmp, patBase, counts, upAdj, upEdges, nodes)) return true;
        P.up_built = true;
    }
    // (the second direction's build finds the same numbers: calls of the first one are reading them)
    if (P.usable) return true;
    P.h0 = h0;
    P.nblk = nblk;
    P.npat = npat;
    P.pat_base = std::move(patBase);
    P.usable = true;
    return true;
}

}  // namespace

std::vector<unsigned> count_low_children(DevicePlan& d) {
    Temps tmp;
    const long long R = static_cast<long long>(d.up_off.size()) - 1;
    std::vector<unsigned> low(R);
    const long long* dOff = reinterpret_cast<long long*>(tmp.copy(d.up_off));
    unsigned* dLow = tmp.get<unsigned>(R);
    low_count_kernel<<<blocks_for(R, 8), 256>>>(d.up.adj, dOff, R, static_cast<unsigned>(d.level_begin[1]), dLow);
    GRGX_CUDA(cudaGetLastError());
    GRGX_CUDA(cudaMemcpy(low.data(), dLow, R * sizeof(unsigned), cudaMemcpyDeviceToHost));
    return low;
}

void pair_counts(grgx_graph* g, bool down, uint64_t out[4]) {
    const DevicePlan* dp = ensure_device_plan(g);
    std::lock_guard<std::mutex> lk(g->mu);
    const PairPlan& P = dp->pair;
    const bool built = P.usable && (down ? P.down_built : P.up_built);
    uint64_t low = 0;
    for (unsigned c : P.low) low += c;
    out[0] = built ? P.h0 : 0;
    out[1] = built ? P.nblk : 0;
    out[2] = built ? P.npat : 0;
    out[3] = built ? low : 0;
}

const void* pair_analysis(grgx_graph* g) {
    const DevicePlan* dp = ensure_device_plan(g);
    std::lock_guard<std::mutex> lk(g->mu);
    return dp->pair.usable ? dp->pair.pat_base.data() : nullptr;
}

void set_pair_rows(long long most) { g_most_rows.store(most); }

void set_pair_mode(int mode) { g_pair_mode.store(mode); }

void set_pair_choice(grgx_graph* g, DevicePlan* dp, const Layout& L, bool down, bool pair) {
    std::lock_guard<std::mutex> lk(g->mu);
    (down ? dp->down_pair_choice : dp->up_pair_choice)[{static_cast<int>(L.kind), L.stride}] = pair;
}

void clear_pair_choice(grgx_graph* g, DevicePlan* dp, const Layout& L, bool down) {
    std::lock_guard<std::mutex> lk(g->mu);
    (down ? dp->down_pair_choice : dp->up_pair_choice).erase({static_cast<int>(L.kind), L.stride});
}

namespace {
// While alive, this thread's allocations and synchronous copies neither fail for nor end another thread's
// stream capture.
class RelaxedCapture {
  public:
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode_); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode_); }
    RelaxedCapture(const RelaxedCapture&) = delete;
    RelaxedCapture& operator=(const RelaxedCapture&) = delete;

  private:
    cudaStreamCaptureMode mode_ = cudaStreamCaptureModeRelaxed;
};
}  // namespace

bool use_pair_form(grgx_graph* g, DevicePlan* dp, const Layout& L, bool down, cudaStream_t s) {
    const int mode = g_pair_mode.load();
    if (mode == 2) return false;
    // (a split form asked for by its test hooks)
    if (mode == 0 && (down ? down_split_forced() : split_threshold_bytes() != kDefaultSplitThreshold)) return false;
    // UP, a single 4-byte column: gathers from the height-0 values run at about one per SM clock
    // however narrow, and the staged lists at five edges per clock (int32 0.38 ms against 1.0,
    // N=200,000, M=250,000); compensated sums would lose the pattern rows' roundings.
    if (!down && L.stride == 1 && (L.kind == Kind::F32C || (staged_layout(L) && up_split_possible(dp)))) return false;
    std::lock_guard<std::mutex> lk(g->mu);
    const auto& choice = down ? dp->down_pair_choice : dp->up_pair_choice;
    const auto chosen = choice.find({static_cast<int>(L.kind), L.stride});
    if (mode == 0 && chosen != choice.end() && !chosen->second) return false;
    PairPlan& P = dp->pair;
    bool& tried = down ? P.down_tried : P.up_tried;
    if (tried || P.refused) return down ? P.down_built : P.up_built;
    // A call that an application captures into a CUDA graph takes another form, as a build's allocations and
    // copies cannot be captured; a capture on another thread is none of this build's business.
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    const cudaError_t asked = cudaStreamIsCapturing(s, &capturing);
    if (asked != cudaSuccess) cudaGetLastError();  // (the legacy stream, beside a blocking stream's capture)
    if (asked != cudaSuccess || capturing != cudaStreamCaptureStatusNone) return false;
    const RelaxedCapture relaxed;
    for (int attempt = 0; attempt < 2 && !tried; attempt++) {
        try {
            tried = true;
            P.refused = !build_pair_plan(*dp, down);
        } catch (const std::bad_alloc&) {
            // host memory: the other forms need little of it
        } catch (const Error& e) {
            if (e.code != GRGX_ERR_OUT_OF_MEMORY) throw;
            cudaGetLastError();
            // Once more with the memory the pool keeps between calls.  Then the direction stays with the
            // other forms, which need none of this: every further call would wait for the same failure.
            tried = attempt > 0;
            if (!tried) trim_pool();
        }
    }
    return down ? P.down_built : P.up_built;
}

}  // namespace grgx
