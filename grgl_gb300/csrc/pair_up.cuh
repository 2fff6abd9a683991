// UP in pair form: pattern rows from the height-0 rows, and the nodes' sums from the pattern rows
// (pair_plan.h).  Both are sums over lists of rows whose lengths differ widely (a block's patterns
// have 1 to thousands of height-0 nodes), so the plan cuts long pattern lists into pieces, sorts the
// lists by length and one kernel gives each list a group of lanes of its own.
#pragma once
#include <algorithm>
#include <stdexcept>
#include <type_traits>

#include "launch.h"

namespace grgx {

// Lanes per list: those for the columns, or at least eight.
constexpr int pair_list_lanes(int g) { return (g & (g - 1)) == 0 && g < 8 ? 8 : g; }

// One warp takes 32 / L lists of about equal length, L = G lanes for the columns, at least eight:
// with narrower rows the lanes left over share out the list (sub), and their sums are merged at the
// end.  The lanes of a list load its ids together and pass them round.
//
// Bound by the L2 -> SM reads of its gathers and the packed additions when rows are wide (float32
// K=64: 68% of L2 throughput, 65% of the FP32 pipe that takes packed instructions; its sources miss
// L1 throughout), by L1's rate of about one random row per clock when they are narrow.  The sweep
// over the same lists walks every row boundary (a quarter of the patterns hold a single height-0
// node) through its reductions: on N=200,000, M=250,000 float32 K=64 took 7.4 ms that way, 8.1
// without the pair form and 4.4 here, float64 K=32 11.9, 9.4 and 5.1, int32 K=48 3.7, 6.5 and 3.8.
// Four blocks of threads per SM against three: float32 K=64 4.43 against 4.83 ms; batches of four
// gathers instead of eight: within 3% either way.
template <class Op, int VW, int G> __device__ __forceinline__ void pair_up(const PairUpParams<typename Op::S>& p) {
    using S = typename Op::S;
    using Acc = VecAcc<Op, VW>;
    constexpr int L = pair_list_lanes(G);
    constexpr bool kOdd = (G & (G - 1)) != 0;
    constexpr int STEPS = kOdd ? 4 : (G < 8 ? 8 / G : 1);  // ids a lane loads at a time
    constexpr int SLOTS = G * STEPS;                       // rows a lane gathers from them
    static_assert(SLOTS % 8 == 0, "batches of eight");
    constexpr int FLUSH_EVERY = SLOTS > 16 ? 1 : 32 / SLOTS;
    constexpr bool kChains = ChainTraits<Op>::kChains;
    const int lane = threadIdx.x & 31;
    const int gl = lane % L, sub = gl / G;
    const int col = blockIdx.y * (G * VW) + (lane % G) * VW;
    const bool colok = col < p.stride;
    const bool inside = !kOdd || lane < 32 / L * L;  // (lanes past the last whole list have none)
    const long long r = ((long long)blockIdx.x * 8 + (threadIdx.x >> 5)) * (32 / L) + lane / L;
    PairList list{0, 0, 0};
    if (r < p.count && inside) list = p.lists[r];
    int most = list.len;
    if constexpr (kOdd) {
        most = __reduce_max_sync(FULL_MASK, most);
    } else {
#pragma unroll
        for (int m = L; m < 32; m <<= 1) most = max(most, __shfl_xor_sync(FULL_MASK, most, m));
    }
    const uint32_t* ids = p.adj + list.e0;
    // (lanes past the last column read with the tile's first lane: another tile's columns would take up L2)
    const char* src = reinterpret_cast<const char*>(p.src + blockIdx.y * p.tile_step + (colok ? (lane % G) * VW : 0));
    const unsigned rowBytes = static_cast<unsigned>(p.src_stride * sizeof(S));
    Acc acc;
    acc.zero();
    uint32_t next[STEPS];
#pragma unroll
    for (int s = 0; s < STEPS; s++) next[s] = (s * L + gl < list.len) ? __ldg(ids + s * L + gl) : 0x80000000u;
    int rounds = 0;
    for (int k = 0; k < most; k += L * STEPS) {
        uint32_t raw[STEPS];
#pragma unroll
        for (int s = 0; s < STEPS; s++) {
            raw[s] = next[s];
            const int at = k + (STEPS + s) * L + gl;
            next[s] = (at < list.len) ? __ldg(ids + at) : 0x80000000u;
        }
#pragma unroll
        for (int t0 = 0; t0 < SLOTS; t0 += 8) {
            if (t0 > 0 && k + t0 >= most) break;  // (only where a step has more than eight slots, sub = 0)
            S v[8][VW];
#pragma unroll
            for (int t = 0; t < 8; t++) {
                const int s = (t0 + t) / G, u = (t0 + t) % G;
                const uint32_t id = __shfl_sync(FULL_MASK, raw[s], (lane / L * L + sub * G + u) & 31);
                if (static_cast<int>(id) >= 0) {
                    Vec<S, VW>::ld(reinterpret_cast<const S*>(src + (unsigned long long)id * rowBytes), v[t]);
                } else {
#pragma unroll
                    for (int i = 0; i < VW; i++) v[t][i] = S{};
                }
            }
            acc.template add_block<8>(v);
            if (kChains && SLOTS > 32 && t0 % 32 == 24) acc.flush();  // a run is 32 additions at most
        }
        if (kChains && ++rounds == FLUSH_EVERY) {
            rounds = 0;
            acc.flush();
        }
    }
    if constexpr (kGrouped<Op>) acc.seal();
#pragma unroll
    for (int m = G; m < L; m <<= 1) {  // (none where L = G)
        const auto t = acc.shfl_xor(m);
        acc.merge(t);
    }
    if (r >= p.count || !inside || sub != 0 || !colok) return;
    if (list.out >= 0 && p.state != nullptr) {
        typename Op::A* d = static_cast<typename Op::A*>(p.state) + (long long)list.out * p.stride + col;
#pragma unroll
        for (int i = 0; i < VW; i++) d[i] = acc.get(i);
        return;
    }
    const bool onto = list.out >= 0 && p.rmw;
    S* d = (list.out >= 0 ? p.dst + (long long)list.out * p.stride : p.table + (long long)~list.out * p.stride) + col;
    S out[VW];
    if (onto) ld_plain<S, VW>(d, out);
#pragma unroll
    for (int i = 0; i < VW; i++) {
        if constexpr (std::is_base_of<AddF64SD, Op>::value) out[i] = onto ? df_add(out[i], acc.pair(i)) : acc.pair(i);
        else out[i] = onto ? Op::finish_onto(out[i], acc.get(i)) : Op::finish(acc.get(i));
    }
    Vec<S, VW>::st(d, out);
}

template <class Op, int VW, int G>
__global__ void __launch_bounds__(256, (G & (G - 1)) ? 3 : 4) pair_up_kernel(const PairUpParams<typename Op::S> p) {
    if constexpr (std::is_base_of<AddF64S, Op>::value) {
        if (p.gate != nullptr && *p.gate != 0) {
            pair_up<AddF64T, VW, G>(as_f64(p));
            return;
        }
    }
    pair_up<Op, VW, G>(p);
}

template <class Op, int VW, int G> void pair_up_as(const PairUpParams<typename Op::S>& p, cudaStream_t s) {
    constexpr int perBlock = 8 * (32 / pair_list_lanes(G));
    const dim3 grid(static_cast<unsigned>((p.count + perBlock - 1) / perBlock),
                    static_cast<unsigned>((p.stride / VW + G - 1) / G));
    pair_up_kernel<Op, VW, G><<<grid, 256, 0, s>>>(p);
}

#define GRGX_PAIR_UP_CASE(OP, VWV, GV) \
    if (vw == VWV && g == GV) {        \
        pair_up_as<OP, VWV, GV>(p, s); \
        return;                        \
    }
#define GRGX_PAIR_UP4(OP)        \
    GRGX_PAIR_UP_CASE(OP, 4, 4)  \
    GRGX_PAIR_UP4_BUT4(OP)
#define GRGX_PAIR_UP4_BUT4(OP)   \
    GRGX_PAIR_UP_CASE(OP, 1, 1)  \
    GRGX_PAIR_UP_CASE(OP, 2, 1)  \
    GRGX_PAIR_UP_CASE(OP, 4, 1)  \
    GRGX_PAIR_UP_CASE(OP, 4, 2)  \
    GRGX_PAIR_UP_CASE(OP, 4, 8)  \
    GRGX_PAIR_UP_CASE(OP, 4, 16) \
    GRGX_PAIR_UP_CASE(OP, 4, 32) \
    GRGX_PAIR_UP_CASE(OP, 4, 6)  \
    GRGX_PAIR_UP_CASE(OP, 4, 10)
#define GRGX_PAIR_UP8(OP)        \
    GRGX_PAIR_UP_CASE(OP, 1, 1)  \
    GRGX_PAIR_UP_CASE(OP, 2, 1)  \
    GRGX_PAIR_UP_CASE(OP, 2, 2)  \
    GRGX_PAIR_UP_CASE(OP, 2, 4)  \
    GRGX_PAIR_UP_CASE(OP, 2, 8)  \
    GRGX_PAIR_UP_CASE(OP, 2, 16) \
    GRGX_PAIR_UP_CASE(OP, 2, 32) \
    GRGX_PAIR_UP_CASE(OP, 2, 6)  \
    GRGX_PAIR_UP_CASE(OP, 2, 10)

}  // namespace grgx
