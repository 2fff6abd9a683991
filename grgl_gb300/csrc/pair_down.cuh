// DOWN in pair form: the height-0 rows' sums over patterns (pair_plan.h).
//
//   pair_table_kernel    pattern row = sum of its parents' rows, for the blocks of one table
//   pair_down_kernel     height-0 row += one pattern row per block
//   pair_finish_kernel   rows whose blocks were shared out over several items: the items' sums added
//                        up in order, onto the row's seed value
#pragma once
#include <algorithm>
#include <stdexcept>
#include <type_traits>

#include "launch.h"

namespace grgx {

// Accumulated sum of one item as it is kept between kernels: compensated sums stay pairs, float pairs' sums
// become pairs again.
template <class Op> struct PairPart {
    using T = typename Op::A;
    using Sum = typename Op::A;
    static __device__ __forceinline__ Sum zero() { return Op::zero(); }
    static __device__ __forceinline__ T of(const Sum& a) { return a; }
    static __device__ __forceinline__ void merge(Sum& a, const T& x) { Op::merge(a, x); }
    static __device__ __forceinline__ typename Op::S finish_onto(typename Op::S base, const Sum& a) { return Op::finish_onto(base, a); }
};
template <> struct PairPart<AddF64ST> {
    using T = DF;
    using Sum = DFSum;
    static __device__ __forceinline__ Sum zero() { return {0.0f, 0.0f, 0.0f}; }
    static __device__ __forceinline__ T of(const Sum& a) { return a.pair(); }
    static __device__ __forceinline__ void merge(Sum& a, const T& x) { a.fold(x); }
    static __device__ __forceinline__ DF finish_onto(DF base, Sum a) {
        a.fold(base);
        return a.pair();
    }
};

// Pattern row elements.  A pair of rows is summed in storage precision: compensated float32 rounds
// it once, which takes the place of the sweep's plain pre-sums (vecacc.cuh); float pairs keep 48
// bits.  A single compensated column, and the columns of short rows (AddF32CX), have no pre-sums in the
// sweep and keep the pair's error here.
template <class Op, int VW> struct PairTable {
    using T = typename Op::S;
    static __device__ __forceinline__ T sum(typename Op::S a, typename Op::S b) {
        if constexpr (std::is_base_of<AddF64S, Op>::value) return df_add(a, b);
        else if constexpr (std::is_base_of<AddF32C, Op>::value) return __fadd_rn(a, b);
        else {
            typename Op::A t = Op::zero();
            Op::add(t, a);
            Op::add(t, b);
            return Op::finish(t);
        }
    }
};
struct PairTableExact {
    using T = F32Pair;
    static __device__ __forceinline__ T sum(float a, float b) {
        T t;
        AddF32C::two_sum(a, b, t.hi, t.lo);
        return t;
    }
};
template <> struct PairTable<AddF32C, 1> : PairTableExact {};
template <> struct PairTable<AddF32CX, 2> : PairTableExact {};
template <typename T, int VW> struct TableVec : Vec<T, VW> {};
template <> struct TableVec<F32Pair, 2> {
    static __device__ __forceinline__ void ld(const F32Pair* p, F32Pair* v) {
        const float4 t = __ldg(reinterpret_cast<const float4*>(p));
        v[0] = {t.x, t.y};
        v[1] = {t.z, t.w};
    }
    static __device__ __forceinline__ void st(F32Pair* p, const F32Pair* v) {
        *reinterpret_cast<float4*>(p) = make_float4(v[0].hi, v[0].lo, v[1].hi, v[1].lo);
    }
};
template <> struct TableVec<F32Pair, 1> {
    static __device__ __forceinline__ void ld(const F32Pair* p, F32Pair* v) {
        const float2 t = __ldg(reinterpret_cast<const float2*>(p));
        v[0] = {t.x, t.y};
    }
    static __device__ __forceinline__ void st(F32Pair* p, const F32Pair* v) {
        *reinterpret_cast<float2*>(p) = make_float2(v[0].hi, v[0].lo);
    }
};

// The operator a float-pair kernel stands in for when its call takes the FP64 path.
template <class Op> constexpr bool kHasF64 = std::is_base_of<AddF64S, Op>::value;

template <class Op, int VW>
__device__ __forceinline__ void pair_table(const uint2* __restrict__ nodes, long long count,
                                           const typename Op::S* __restrict__ vals, long long stride,
                                           typename PairTable<Op, VW>::T* __restrict__ table) {
    using S = typename Op::S;
    using T = typename PairTable<Op, VW>::T;
    const unsigned vecs = static_cast<unsigned>(stride / VW);
    const unsigned long long total = (unsigned long long)count * vecs;
    for (unsigned long long x = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; x < total;
         x += (unsigned long long)gridDim.x * blockDim.x) {
        const unsigned long long pat = x / vecs;
        const int col = static_cast<int>(x - pat * vecs) * VW;
        const uint2 nd = __ldg(nodes + pat);
        S a[VW], b[VW];
#pragma unroll
        for (int i = 0; i < VW; i++) a[i] = b[i] = S{};
        if (nd.x != 0x7fffffffu) Vec<S, VW>::ld(vals + (long long)nd.x * stride + col, a);
        if (nd.y != 0x7fffffffu) Vec<S, VW>::ld(vals + (long long)nd.y * stride + col, b);
        T t[VW];
#pragma unroll
        for (int i = 0; i < VW; i++) t[i] = PairTable<Op, VW>::sum(a[i], b[i]);
        TableVec<T, VW>::st(table + (long long)pat * stride + col, t);
    }
}

template <class Op, int VW>
__global__ void pair_table_kernel(const uint2* nodes, long long count, const typename Op::S* vals, long long stride,
                                  typename PairTable<Op, VW>::T* table, const int* gate) {
    if constexpr (kHasF64<Op>) {
        if (gate != nullptr && *gate != 0) {
            pair_table<AddF64T, VW>(nodes, count, reinterpret_cast<const double*>(vals), stride, reinterpret_cast<double*>(table));
            return;
        }
    }
    pair_table<Op, VW>(nodes, count, vals, stride, table);
}

// Rows per group of lanes: a warp covers (32 / G) * kPairRows rows, four blocks of each at a time,
// so eight gathers are in flight per lane.  Four rows (sixteen gathers, two blocks of threads per
// SM instead of three), with the kernel's first version, ran within 3% either way for int32 and wide float64
// and slower for the rest (float32 K=64 4.29 against 4.11 ms, float64 K=8 1.92 against 1.66 ms; N=200,000, M=250,000).
constexpr int kPairRows = 2;

// Bound by the L2 -> SM reads of its gathers when rows are wide (float32 K=64: 16-17 TB/s of pattern
// rows, the read probe's rate), by the packed float32 additions for float pairs, and by the rate
// of gather instructions for the narrowest rows, whose tables mostly sit in L1.  It takes half the
// gathers of a sweep over edges, has no row boundaries to look for (each row has exactly one
// pattern per block), and reads one byte of ids per edge.  DOWN products on N=200,000, M=250,000
// before and now: int32 K=1 0.65 -> 0.28 ms (staged split passes before), float32 K=9 2.38 ->
// 1.18, float32 K=64 7.87 -> 3.63, float64 K=64 16.6 -> 8.06 ms.
//
// One warp per item (a share of the blocks x a tile of rows).  A row's columns are spread over G
// lanes as in the sweep; each lane loads its rows' ids of four blocks (8 bytes) and gathers the
// four pattern rows of each of its kRows rows before adding them.
template <class Op, int VW, int G> __device__ __forceinline__ void pair_down(const PairDownParams<typename Op::S>& p) {
    using S = typename Op::S;
    using T = typename PairTable<Op, VW>::T;
    using Acc = VecAcc<Op, VW>;
    using Part = PairPart<Op>;
    constexpr int NG = 32 / G, ROWS = kPairRows;
    static_assert(NG * ROWS <= kPairTile, "a warp's rows end within the padded ids");
    constexpr bool kRuns = std::is_same<Op, AddF64ST>::value;
    const int lane = threadIdx.x & 31;
    // (lanes without a column or past the last whole row follow along on the warp's first row)
    const int col = blockIdx.y * (G * VW) + (lane % G) * VW;
    const bool active = (NG * G == 32 || lane < NG * G) && col < p.stride;
    const int lg = (NG * G == 32 || lane < NG * G) ? lane / G : 0;
    const unsigned rowBytes = static_cast<unsigned>(p.stride * sizeof(T));
    const char* table = reinterpret_cast<const char*>(static_cast<const T*>(p.table) + (active ? col : 0));
    unsigned* counter = p.work + blockIdx.y;
    for (;;) {
        unsigned c = 0;
        if (lane == 0) c = atomicAdd(counter, 1u);
        c = __shfl_sync(FULL_MASK, c, 0);
        if (c >= p.tiles * p.items) return;
        const unsigned item = c / p.tiles;
        const long long row0 = (long long)(c - item * p.tiles) * (NG * ROWS) + lg;
        const int q0 = p.group_begin + static_cast<int>(item) * p.groups_per_item;
        const int q1 = min(p.group_end, q0 + p.groups_per_item);
        const uint2* idp[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; r++) {
            const long long row = row0 + r * NG;
            idp[r] = p.ids + ((row >> 5) * p.groups + q0) * 32 + (row & 31);
        }
        Acc acc[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; r++) acc[r].zero();
        uint2 next[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; r++) next[r] = __ldg(idp[r]);
        for (int q = q0; q < q1; q++) {
            const uint4 b = __ldg(p.base + q);
            uint2 id[ROWS];
#pragma unroll
            for (int r = 0; r < ROWS; r++) {
                id[r] = next[r];
                idp[r] += 32;
                if (q + 1 < q1) next[r] = __ldg(idp[r]);
            }
            T v[ROWS][4][VW];
#pragma unroll
            for (int r = 0; r < ROWS; r++) {
                const unsigned k[4] = {b.x - p.base0 + (id[r].x & 0xffffu), b.y - p.base0 + (id[r].x >> 16),
                                       b.z - p.base0 + (id[r].y & 0xffffu), b.w - p.base0 + (id[r].y >> 16)};
#pragma unroll
                for (int u = 0; u < 4; u++)
                    TableVec<T, VW>::ld(reinterpret_cast<const T*>(table + (unsigned long long)k[u] * rowBytes), v[r][u]);
            }
            if constexpr (kRuns) {
                if ((q - q0) & 1 & p.long_runs) {
#pragma unroll
                    for (int r = 0; r < ROWS; r++) acc[r].add_rows(v[r]);
                } else {
#pragma unroll
                    for (int r = 0; r < ROWS; r++) acc[r].start_rows(v[r]);
                }
                if ((q - q0) & 1 | !p.long_runs) {
#pragma unroll
                    for (int r = 0; r < ROWS; r++) acc[r].fold();
                }
            } else if constexpr (kGrouped<Op>) {
                if ((q - q0) & 1) {
#pragma unroll
                    for (int r = 0; r < ROWS; r++) acc[r].add_rows(v[r]);
                    if (((q - q0) & 7) == 7) {
#pragma unroll
                        for (int r = 0; r < ROWS; r++) acc[r].flush();
                    }
                } else {
#pragma unroll
                    for (int r = 0; r < ROWS; r++) acc[r].hold_rows(v[r]);
                }
            } else {
#pragma unroll
                for (int r = 0; r < ROWS; r++) acc[r].add_pairs(v[r]);
            }
        }
        if constexpr (kRuns) {
            if ((q1 - q0) & 1 & p.long_runs) {
#pragma unroll
                for (int r = 0; r < ROWS; r++) acc[r].fold();
            }
        }
        if constexpr (kGrouped<Op>) {
#pragma unroll
            for (int r = 0; r < ROWS; r++) {
                if ((q1 - q0) & 1) acc[r].add_held();
                acc[r].seal();
            }
        }
        if (!active) continue;
#pragma unroll
        for (int r = 0; r < ROWS; r++) {
            const long long row = row0 + r * NG;
            if (row >= p.rows) continue;
            if (p.parts == nullptr) {
                S base[VW], out[VW];
                S* d = p.vals + row * p.stride + col;
                ld_plain<S, VW>(d, base);
#pragma unroll
                for (int i = 0; i < VW; i++) out[i] = Part::finish_onto(base[i], acc[r].get(i));
                Vec<S, VW>::st(d, out);
            } else {
                typename Part::T* d = static_cast<typename Part::T*>(p.parts) +
                                      ((long long)(p.part_begin + item) * p.rows + row) * p.stride + col;
#pragma unroll
                for (int i = 0; i < VW; i++) d[i] = Part::of(acc[r].get(i));
            }
        }
    }
}

template <class Op, int VW, int G>
__global__ void __launch_bounds__(256, 3) pair_down_kernel(const PairDownParams<typename Op::S> p) {
    if constexpr (kHasF64<Op>) {
        if (p.gate != nullptr && *p.gate != 0) {
            pair_down<AddF64T, VW, G>(as_f64(p));
            return;
        }
    }
    pair_down<Op, VW, G>(p);
}

// Adds up `count` sums per row, in order: into the first one (vals null), or onto the node values.
template <class Op>
__device__ __forceinline__ void pair_finish(typename PairPart<Op>::T* __restrict__ parts, int count, long long rows,
                                            long long stride, typename Op::S* __restrict__ vals) {
    const long long total = rows * stride;
    for (long long x = (long long)blockIdx.x * blockDim.x + threadIdx.x; x < total; x += (long long)gridDim.x * blockDim.x) {
        typename PairPart<Op>::Sum a = PairPart<Op>::zero();
        for (int j = 0; j < count; j++) PairPart<Op>::merge(a, parts[j * total + x]);
        if (vals == nullptr) {
            parts[x] = PairPart<Op>::of(a);
            continue;
        }
        if constexpr (std::is_same<typename Op::S, DF>::value)
            df_put(vals, x, stride, PairPart<Op>::finish_onto(df_get(vals, x, stride), a));
        else
            vals[x] = PairPart<Op>::finish_onto(vals[x], a);
    }
}

template <class Op>
__global__ void pair_finish_kernel(typename PairPart<Op>::T* parts, int count, long long rows, long long stride,
                                   typename Op::S* vals, const int* gate) {
    if constexpr (kHasF64<Op>) {
        if (gate != nullptr && *gate != 0) {
            pair_finish<AddF64T>(reinterpret_cast<double*>(parts), count, rows, stride, reinterpret_cast<double*>(vals));
            return;
        }
    }
    pair_finish<Op>(parts, count, rows, stride, vals);
}

template <class Op, int VW, int G>
int pair_blocks_per_sm() {
    static int n = 0;
    if (n == 0) {
        int v = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, pair_down_kernel<Op, VW, G>, 256, 0);
        n = v > 0 ? v : 1;
    }
    return n;
}

template <class Op, int VW, int G> void pair_down_as(PairDownParams<typename Op::S> p, PairDownCall& c, int sms, cudaStream_t s) {
    if (c.step == PairDownCall::kShape) {
        c.rows_per_warp = (32 / G) * kPairRows;
        c.resident_warps = pair_blocks_per_sm<Op, VW, G>() * 8 * sms;
        c.part_bytes = sizeof(typename PairPart<Op>::T);
        c.table_bytes = sizeof(typename PairTable<Op, VW>::T);
        return;
    }
    if (c.step == PairDownCall::kTable) {
        const unsigned long long total = (unsigned long long)c.count * (p.stride / VW);
        const unsigned grid = static_cast<unsigned>(std::min<unsigned long long>((total + 255) / 256, sms * 64ull));
        pair_table_kernel<Op, VW><<<grid, 256, 0, s>>>(c.nodes, c.count, p.vals, p.stride,
                                                       static_cast<typename PairTable<Op, VW>::T*>(p.table), p.gate);
        return;
    }
    if (c.step == PairDownCall::kFinish) {
        const unsigned long long total = (unsigned long long)p.rows * p.stride;
        const unsigned grid = static_cast<unsigned>(std::min<unsigned long long>((total + 255) / 256, sms * 64ull));
        pair_finish_kernel<Op><<<grid, 256, 0, s>>>(static_cast<typename PairPart<Op>::T*>(p.parts), c.parts, p.rows, p.stride,
                                                    c.onto ? p.vals : nullptr, p.gate);
        return;
    }
    const unsigned warps = p.tiles * p.items;
    const unsigned most = static_cast<unsigned>(pair_blocks_per_sm<Op, VW, G>() * sms);
    const unsigned tilesY = static_cast<unsigned>((p.stride / VW + G - 1) / G);
    pair_down_kernel<Op, VW, G><<<dim3(std::min((warps + 7) / 8, most), tilesY), 256, 0, s>>>(p);
}

#define GRGX_PAIR_CASE(OP, VWV, GV)               \
    if (vw == VWV && g == GV) {                   \
        pair_down_as<OP, VWV, GV>(p, c, sms, s);  \
        return;                                   \
    }
// (lane counts that are no power of two fit more rows into a warp: see pair_lanes)
#define GRGX_PAIR_ODD(OP, VWV)                                                                      \
    GRGX_PAIR_CASE(OP, VWV, 5)                                                                      \
    GRGX_PAIR_CASE(OP, VWV, 6)                                                                      \
    GRGX_PAIR_CASE(OP, VWV, 10)
#define GRGX_PAIR4(OP)                                                                              \
    GRGX_PAIR_CASE(OP, 1, 1)                                                                        \
    GRGX_PAIR_WIDE4(OP)
#define GRGX_PAIR_WIDE4(OP)                                                                         \
    GRGX_PAIR_CASE(OP, 2, 1)                                                                        \
    GRGX_PAIR_CASE(OP, 4, 1)                                                                        \
    GRGX_PAIR_CASE(OP, 4, 2)                                                                        \
    GRGX_PAIR_CASE(OP, 4, 4)                                                                        \
    GRGX_PAIR_CASE(OP, 4, 8)                                                                        \
    GRGX_PAIR_CASE(OP, 4, 16)                                                                       \
    GRGX_PAIR_CASE(OP, 4, 32)                                                                       \
    GRGX_PAIR_ODD(OP, 4)
#define GRGX_PAIR8(OP)                                                                              \
    GRGX_PAIR_CASE(OP, 1, 1)                                                                        \
    GRGX_PAIR_CASE(OP, 2, 1)                                                                        \
    GRGX_PAIR_CASE(OP, 2, 2)                                                                        \
    GRGX_PAIR_CASE(OP, 2, 4)                                                                        \
    GRGX_PAIR_CASE(OP, 2, 8)                                                                        \
    GRGX_PAIR_CASE(OP, 2, 16)                                                                       \
    GRGX_PAIR_CASE(OP, 2, 32)                                                                       \
    GRGX_PAIR_ODD(OP, 2)

}  // namespace grgx
