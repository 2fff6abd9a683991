// Single-column products of 4-byte values in split form: a block's source values (at most 32,768 of
// them, 128 KB) fit in shared memory, and its edges are 16-bit ids relative to the block
// (up_split.cu).  A row's edges in one block are a list; lists longer than kStagedPiece are cut, all
// lists of a block are sorted by length, and every list has a slot for its sum, a row's slots one
// after the other:
//   staged_kernel      one block of threads per SM copies its block's values and sums its share of
//                      the block's lists, eight lanes to a list
//   staged_sum_kernel  adds up each row's slots, in order
// All blocks are one launch: the SMs are shared out among them by their edges.
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "device_plan.h"

namespace grgx {

namespace {

constexpr int kStagedThreads = 1024;
constexpr long long kStagedPiece = 1024;
// What a list costs besides its edges, in edges (its descriptor, a step of 64 ids that it need not
// fill, the lanes' merge): half the lists have under 50 edges (float32 K=1 UP, N=200,000, M=250,000:
// 0.53 ms at 50, 0.46 at 100 and at 200, 0.70 by edges alone).
constexpr long long kStagedListCost = 100;


// Sums of the lists of one block by `parts` blocks of threads: this one takes every parts-th group
// of 128 lists.  Ids are loaded eight at a time from the 16-byte boundary at or below a list's start;
// what lies outside the list adds zero.
//
// Each id costs a random 4-byte read of shared memory: 32 of them hit the most loaded of 32 banks
// about 3.4 times, so about 9 edges per SM and clock is the most; the packed compensated additions
// and the id arithmetic take about as long (74% of the shared-memory pipe, 53% of the issue slots).
// UP K=1 on N=200,000, M=250,000 before (one launch per block, rows found from head bits in chunks,
// each row merged into its state per block) and now: float32 0.87 -> 0.42 ms, int32 0.63 -> 0.38.
template <class Op>
__global__ void __launch_bounds__(kStagedThreads, 1) staged_kernel(const StagedPart* __restrict__ parts,
                                                                   const PairList* __restrict__ lists,
                                                                   const unsigned short* __restrict__ adj,
                                                                   const typename Op::S* __restrict__ src,
                                                                   typename Op::A* __restrict__ sums) {
    using S = typename Op::S;
    extern __shared__ __align__(16) unsigned char raw[];
    S* values = reinterpret_cast<S*>(raw);
    const StagedPart P = parts[blockIdx.x];
    {
        const S* from = src + P.src;
        // 16-byte copies past the source's unaligned head, single values before and after them
        const int head = min(P.rows, static_cast<int>((16 - (reinterpret_cast<uintptr_t>(from) & 15)) / 4 % 4));
        const int vecs = (P.rows - head) / 4;
        for (int i = threadIdx.x; i < vecs; i += kStagedThreads) {
            const uint4 t = __ldg(reinterpret_cast<const uint4*>(from + head) + i);
            unsigned* to = reinterpret_cast<unsigned*>(values) + head + 4 * i;
            to[0] = t.x;
            to[1] = t.y;
            to[2] = t.z;
            to[3] = t.w;
        }
        for (int i = threadIdx.x; i < P.rows; i += kStagedThreads)
            if (i < head || i >= head + 4 * vecs) values[i] = __ldg(from + i);
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, gl = lane & 7;
    const int warp = threadIdx.x >> 5;
    // two lists ahead of the one being summed: its descriptor, and one ahead: its first ids
    const int stride = P.parts * (kStagedThreads / 32) * 4;
    auto list_at = [&](int l) { return l < P.list1 ? lists[l] : PairList{0, 0, 0}; };
    auto first_ids = [&](const PairList& t) {
        const int off = static_cast<int>(t.e0 & 7);
        uint4 w = make_uint4(0u, 0u, 0u, 0u);
        if (gl * 8 < off + t.len) w = __ldg(reinterpret_cast<const uint4*>(adj + (t.e0 - off)) + gl);
        return w;
    };
    int l = P.list0 + (P.part * (kStagedThreads / 32) + warp) * 4 + (lane >> 3);
    PairList after = list_at(l), afterNext = list_at(l + stride);
    uint4 afterIds = first_ids(after);
    for (; l - (lane >> 3) < P.list1; l += stride) {
        const PairList list = after;
        uint4 next = afterIds;
        after = afterNext;
        afterIds = first_ids(after);
        afterNext = list_at(l + 2 * stride);
        const int off = static_cast<int>(list.e0 & 7), end = off + list.len;
        const uint4* ids = reinterpret_cast<const uint4*>(adj + (list.e0 - off)) + gl;
        int most = end;
        most = max(most, __shfl_xor_sync(FULL_MASK, most, 8));
        most = max(most, __shfl_xor_sync(FULL_MASK, most, 16));
        VecAcc<Op, 1> acc;
        acc.zero();
        for (int k = 0; k < most; k += 64) {
            const uint4 w = next;
            const int at = k + 64 + gl * 8;
            if (at < end) next = __ldg(ids + (k + 64) / 8);
            const unsigned word[4] = {w.x, w.y, w.z, w.w};
            S v[8][1];
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const unsigned id = (u & 1) ? (word[u >> 1] >> 16) & 0x7fffu : word[u >> 1] & 0x7fffu;
                v[u][0] = values[id];
            }
            // (a step inside every list of the warp needs no masks; ids past a list's end are stale or
            // another list's, and read a staged value all the same)
            const int first = k + gl * 8;
            if (first < off || first + 8 > end) {
#pragma unroll
                for (int u = 0; u < 8; u++)
                    if (first + u < off || first + u >= end) v[u][0] = S{};
            }
            acc.template add_block<8>(v);
        }
        if constexpr (kGrouped<Op>) acc.seal();
#pragma unroll
        for (int m = 1; m < 8; m <<= 1) {
            const auto t = acc.shfl_xor(m);
            acc.merge(t);
        }
        if (gl == 0 && l < P.list1) sums[list.out] = acc.get(0);
    }
}

// Row i's slots are slot0[i] .. slot0[i+1]-1: their sum becomes the node's accumulator (state set) or
// its value (added onto it when rmw).
template <class Op>
__global__ void staged_sum_kernel(const typename Op::A* __restrict__ sums, const unsigned* __restrict__ slot0,
                                  const int* __restrict__ nodes, long long rows, typename Op::A* __restrict__ state,
                                  long long stateBase, typename Op::S* __restrict__ vals, int rmw) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < rows; i += (long long)gridDim.x * blockDim.x) {
        typename Op::A a = Op::zero();
        for (unsigned s = slot0[i], e = slot0[i + 1]; s < e; s++) Op::merge(a, sums[s]);
        const int node = nodes[i];
        if (state != nullptr) state[node - stateBase] = a;
        else vals[node] = rmw ? Op::finish_onto(vals[node], a) : Op::finish(a);
    }
}

template <class Op>
int run_staged(const StagedLists& T, void* vals, void* sums, void* state, long long stateBase, int rmw, cudaStream_t s) {
    using S = typename Op::S;
    using A = typename Op::A;
    // (always the whole 15-bit range: an id read past a list's end may be any)
    const int bytes = static_cast<int>(kStagedRows * sizeof(S));
    GRGX_CUDA(cudaFuncSetAttribute(staged_kernel<Op>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    staged_kernel<Op><<<T.nparts, kStagedThreads, bytes, s>>>(T.parts, T.lists, T.adj, static_cast<const S*>(vals),
                                                              static_cast<A*>(sums));
    const unsigned grid = static_cast<unsigned>(std::min<long long>((T.rows + 255) / 256, 64LL * sm_count()));
    staged_sum_kernel<Op><<<grid, 256, 0, s>>>(static_cast<const A*>(sums), T.slot0, T.nodes, T.rows, static_cast<A*>(state),
                                               stateBase, static_cast<S*>(vals), rmw);
    return 2;
}

template <typename T> T* to_device(DevicePlan& d, const std::vector<T>& v) {
    void* p = nullptr;
    GRGX_CUDA(cudaMalloc(&p, std::max<size_t>(1, v.size()) * sizeof(T)));
    d.allocs.push_back(p);
    d.bytes += v.size() * sizeof(T);
    if (!v.empty()) GRGX_CUDA(cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice));
    return static_cast<T*>(p);
}

}  // namespace

int launch_staged(Kind kind, const StagedLists& T, void* vals, void* sums, void* state, long long stateBase, int rmw,
                  cudaStream_t s) {
    switch (kind) {
    case Kind::U32: return run_staged<AddU32>(T, vals, sums, state, stateBase, rmw, s);
    case Kind::XOR: return run_staged<XorU32>(T, vals, sums, state, stateBase, rmw, s);
    case Kind::F32C: return run_staged<AddF32C>(T, vals, sums, state, stateBase, rmw, s);
    case Kind::F32: return run_staged<AddF32G>(T, vals, sums, state, stateBase, rmw, s);
    default: return 0;
    }
}

void build_staged(DevicePlan& d, StagedLists& T, const std::vector<uint32_t>& seg, const std::vector<long long>& start,
                  long long R, int nb, const std::vector<long long>& base, const std::vector<long long>& srcRows,
                  const std::vector<int>& nodeOf, const unsigned short* adj) {
    auto len = [&](long long i, int b) {
        return static_cast<long long>(seg[static_cast<size_t>(i) * (nb + 1) + b + 1]) - seg[static_cast<size_t>(i) * (nb + 1) + b];
    };
    std::vector<std::vector<PairList>> lists(nb);
    std::vector<long long> edges(nb, 0);
    std::vector<unsigned> slot0(1, 0);
    std::vector<int> nodes;
    long long slots = 0, total = 0;
    for (long long i = 0; i < R; i++) {
        const long long before = slots;
        for (int b = 0; b < nb; b++) {
            const long long n = len(i, b), pieces = (n + kStagedPiece - 1) / kStagedPiece;
            const long long e = start[static_cast<size_t>(i) * nb + b];
            for (long long p = 0; p < pieces; p++)
                lists[b].push_back({e + n * p / pieces, static_cast<int>(n * (p + 1) / pieces - n * p / pieces),
                                    static_cast<int>(slots++)});
            edges[b] += n;
            total += n;
        }
        if (slots == before) continue;
        nodes.push_back(nodeOf[static_cast<size_t>(i)]);
        slot0.push_back(static_cast<unsigned>(slots));
    }
    if (slots == 0 || slots >= 0x7fffffffLL) return;
    // SMs per block by its work, at least one; what is left over goes where a share is largest
    std::vector<int> share(nb, 1);
    int used = nb;
    auto cost = [&](int b) { return edges[b] + kStagedListCost * static_cast<long long>(lists[b].size()); };
    while (used < sm_count()) {
        int at = 0;
        for (int b = 1; b < nb; b++)
            if (cost(b) * share[at] > cost(at) * share[b]) at = b;
        share[at]++;
        used++;
    }
    std::vector<StagedPart> parts;
    std::vector<PairList> all;
    for (int b = 0; b < nb; b++) {
        const int l0 = static_cast<int>(all.size());
        std::stable_sort(lists[b].begin(), lists[b].end(), [](const PairList& x, const PairList& y) { return x.len > y.len; });
        all.insert(all.end(), lists[b].begin(), lists[b].end());
        for (int k = 0; k < share[b]; k++)
            parts.push_back({base[b], static_cast<int>(srcRows[b]), l0, static_cast<int>(all.size()), k, share[b]});
    }
    T.parts = to_device(d, parts);
    T.nparts = static_cast<unsigned>(parts.size());
    T.lists = to_device(d, all);
    T.slot0 = to_device(d, slot0);
    T.nodes = to_device(d, nodes);
    T.adj = adj;
    T.rows = static_cast<long long>(nodes.size());
    T.slots = slots;
}

}  // namespace grgx
