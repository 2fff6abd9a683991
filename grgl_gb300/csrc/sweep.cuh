// Level-sweep kernel: one level of the pull-form traversal.
//
// For every row r of the level, dst[rows[r]] (+)= sum over its edges e of src[adj[e]]: the
// per-node edge sums of matmulSumChildrenUp / matmulSumChildrenDown (grg.h:1312-1334), one
// level of independent nodes at a time.
//
// Work split: one warp per chunk (a run of whole rows, or one piece of a heavy row).  The
// warp reads its edge ids 32 at a time (one coalesced 128-byte load) and finds row starts
// from the HEAD_BIT of each id with a single ballot.  A row's value vector (the K columns,
// `stride` elements padded for vector loads) is read by a group of G lanes, VW elements per
// lane with one vector load each, so 32/G edges are gathered per sub-step.  Partial sums stay
// in registers; at a row boundary they are combined across groups with shuffles (butterfly
// for the finishing row, segmented scan for rows that start and end inside the sub-step) and
// written once.  Pieces of a heavy row write partials; the last piece to finish (atomic
// ticket) adds them up in piece order, so results do not depend on scheduling.
#pragma once
#include <cstdint>
#include <cstring>
#include <type_traits>

#include "ops.cuh"
#include "vecacc.cuh"

namespace grgx {

struct ChunkDev {
    long long e0;
    int r0;
    int heavy;
};
struct HeavyDev {
    int first_chunk;
    int n_pieces;
    long long slot_base;
};

template <typename S> struct SweepParams {
    const uint32_t* adj;
    const int* rows;
    const ChunkDev* chunks;
    const HeavyDev* heavy;
    long long c_begin, c_end;  // chunk range of this level
    const S* src;              // gather source rows
    S* dst;                    // destination rows (node values)
    long long stride;          // elements per row (src and dst)
    int rmw;                   // add onto the existing dst value
    void* partials;            // Op::A per (slot, column)
    unsigned* tickets;         // per (heavy row, column tile)
    unsigned* work;            // per column tile: next chunk to take (zeroed before the launch)
    int ntiles;
    const int* gate;           // float64 as float pairs: when set and *gate != 0, the buffers hold doubles
    void* state;               // per-node Op::A carried between launches (UP split passes), or null
    long long state_base;      // node id of the first state row
    int state_mode;            // 1: merge each row sum into its state; 2: write state + row sum
    // Edge-id format.  id16 = 0: 32-bit source ids, HEAD_BIT on each row's first edge.  id16 = 1:
    // 16-bit ids relative to id_base (the split copies cut the sources into blocks of at most
    // 32,768 ids), bit 15 marking each row's first edge.
    int id16;
    long long id_base;
    // Levels of short rows (short_rows_kernel): the first edge of each row of the level, relative to
    // `adj` (short_rows + 1 entries), and the level's first row.
    const unsigned* short_off;
    long long short_row0, short_rows;
    int short_split;           // groups of lanes that share a row's edges (a power of two)
    // First column of the launch's tile 0 (a launch of the last, narrow tile starts past the
    // full tiles of another launch).
    int col_base;
};

// The parameters of a float64 call for its FP64 path: the same buffers, of doubles.  Every kernel of
// the float-pair pipeline carries this path and takes it when the call's gate says so (io_df.cu):
// a pipeline of its own behind it was a launch per step that did nothing, a third of the time of a
// small product (one float64 score on N=1,000, M=10,000: 28 launches before, 16 now).
template <template <typename> class Params> __device__ __forceinline__ Params<double> as_f64(const Params<DF>& p) {
    static_assert(sizeof(Params<double>) == sizeof(Params<DF>), "same layout");
    Params<double> q;
    memcpy(&q, &p, sizeof(q));
    return q;
}

// Edge id e of a chunk as stored (32-bit, or 16-bit zero-extended).  The load is issued a step
// ahead of its use; decode_id turns it into the 32-bit form the sweep works with (source id |
// HEAD_BIT) only when the step that needs it starts, so the warp does not wait for the load early.
// The id width is a template parameter (ID16 = p.id16), so the 32-bit kernels carry no 16-bit code.
template <bool ID16, typename S> __device__ __forceinline__ uint32_t load_id(const SweepParams<S>& p, long long e) {
    if constexpr (ID16) return static_cast<uint32_t>(__ldg(reinterpret_cast<const unsigned short*>(p.adj) + e));
    else return __ldg(p.adj + e);
}
template <bool ID16, typename S> __device__ __forceinline__ uint32_t decode_id(const SweepParams<S>& p, uint32_t r) {
    if constexpr (ID16) return ((r & 0x8000u) << 16) | (static_cast<uint32_t>(p.id_base) + (r & 0x7fffu));
    else return r;
}

template <typename S, int VW> struct Vec;
template <> struct Vec<uint32_t, 1> { static __device__ __forceinline__ void ld(const uint32_t* p, uint32_t* v) { v[0] = __ldg(p); } static __device__ __forceinline__ void st(uint32_t* p, const uint32_t* v) { p[0] = v[0]; } };
template <> struct Vec<uint32_t, 2> { static __device__ __forceinline__ void ld(const uint32_t* p, uint32_t* v) { uint2 t = __ldg(reinterpret_cast<const uint2*>(p)); v[0] = t.x; v[1] = t.y; } static __device__ __forceinline__ void st(uint32_t* p, const uint32_t* v) { *reinterpret_cast<uint2*>(p) = make_uint2(v[0], v[1]); } };
template <> struct Vec<uint32_t, 4> { static __device__ __forceinline__ void ld(const uint32_t* p, uint32_t* v) { uint4 t = __ldg(reinterpret_cast<const uint4*>(p)); v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w; } static __device__ __forceinline__ void st(uint32_t* p, const uint32_t* v) { *reinterpret_cast<uint4*>(p) = make_uint4(v[0], v[1], v[2], v[3]); } };
template <> struct Vec<float, 1> { static __device__ __forceinline__ void ld(const float* p, float* v) { v[0] = __ldg(p); } static __device__ __forceinline__ void st(float* p, const float* v) { p[0] = v[0]; } };
template <> struct Vec<float, 2> { static __device__ __forceinline__ void ld(const float* p, float* v) { float2 t = __ldg(reinterpret_cast<const float2*>(p)); v[0] = t.x; v[1] = t.y; } static __device__ __forceinline__ void st(float* p, const float* v) { *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]); } };
template <> struct Vec<float, 4> { static __device__ __forceinline__ void ld(const float* p, float* v) { float4 t = __ldg(reinterpret_cast<const float4*>(p)); v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w; } static __device__ __forceinline__ void st(float* p, const float* v) { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); } };
template <> struct Vec<double, 1> { static __device__ __forceinline__ void ld(const double* p, double* v) { v[0] = __ldg(p); } static __device__ __forceinline__ void st(double* p, const double* v) { p[0] = v[0]; } };
template <> struct Vec<double, 2> { static __device__ __forceinline__ void ld(const double* p, double* v) { double2 t = __ldg(reinterpret_cast<const double2*>(p)); v[0] = t.x; v[1] = t.y; } static __device__ __forceinline__ void st(double* p, const double* v) { *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]); } };
template <> struct Vec<DF, 1> { static __device__ __forceinline__ void ld(const DF* p, DF* v) { float2 t = __ldg(reinterpret_cast<const float2*>(p)); v[0] = {t.x, t.y}; } static __device__ __forceinline__ void st(DF* p, const DF* v) { *reinterpret_cast<float2*>(p) = make_float2(v[0].hi, v[0].lo); } };
// two columns of float pairs, stored (hi, hi, lo, lo): see df_get
template <> struct Vec<DF, 2> { static __device__ __forceinline__ void ld(const DF* p, DF* v) { float4 t = __ldg(reinterpret_cast<const float4*>(p)); v[0] = {t.x, t.z}; v[1] = {t.y, t.w}; } static __device__ __forceinline__ void st(DF* p, const DF* v) { *reinterpret_cast<float4*>(p) = make_float4(v[0].hi, v[1].hi, v[0].lo, v[1].lo); } };
template <> struct Vec<unsigned long long, 1> { static __device__ __forceinline__ void ld(const unsigned long long* p, unsigned long long* v) { v[0] = __ldg(p); } static __device__ __forceinline__ void st(unsigned long long* p, const unsigned long long* v) { p[0] = v[0]; } };
template <> struct Vec<unsigned long long, 2> { static __device__ __forceinline__ void ld(const unsigned long long* p, unsigned long long* v) { ulonglong2 t = __ldg(reinterpret_cast<const ulonglong2*>(p)); v[0] = t.x; v[1] = t.y; } static __device__ __forceinline__ void st(unsigned long long* p, const unsigned long long* v) { *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(v[0], v[1]); } };

// Plain (coherent) load of the current destination value, for read-modify-write.
template <typename S, int VW> __device__ __forceinline__ void ld_plain(const S* p, S* v) {
    if constexpr (std::is_same<S, DF>::value && VW == 2) {
        const float4 t = *reinterpret_cast<const float4*>(p);
        v[0] = {t.x, t.z};
        v[1] = {t.y, t.w};
    } else {
#pragma unroll
        for (int i = 0; i < VW; i++) v[i] = p[i];
    }
}

// The same from L2, past an L1 line that may be older than another SM's store.
template <typename S, int VW> __device__ __forceinline__ void ld_l2(const S* p, S* v) {
    if constexpr (VW * sizeof(S) == 16) {
        const uint4 t = __ldcg(reinterpret_cast<const uint4*>(p));
        if constexpr (std::is_same<S, DF>::value) {
            v[0] = {__uint_as_float(t.x), __uint_as_float(t.z)};
            v[1] = {__uint_as_float(t.y), __uint_as_float(t.w)};
        } else {
            memcpy(v, &t, 16);
        }
    } else if constexpr (VW * sizeof(S) == 8) {
        const uint2 t = __ldcg(reinterpret_cast<const uint2*>(p));
        memcpy(v, &t, 8);
    } else {
        const unsigned t = __ldcg(reinterpret_cast<const unsigned*>(p));
        memcpy(v, &t, 4);
    }
}

// Sum of a lane's accumulator over the 32/G groups of the warp (every group gets the result).
template <class Op, int VW, int G, class Acc> __device__ __forceinline__ void group_allreduce(Acc& x) {
#pragma unroll
    for (int m = G; m < 32; m <<= 1) {
        const auto t = x.shfl_xor(m);
        x.merge(t);
    }
}

// L2-coherent loads for the heavy-row partials written by other warps of the same launch.
__device__ __forceinline__ uint32_t ld_cg(const uint32_t* p) { return __ldcg(p); }
__device__ __forceinline__ unsigned long long ld_cg(const unsigned long long* p) { return __ldcg(p); }
__device__ __forceinline__ double ld_cg(const double* p) { return __ldcg(p); }
__device__ __forceinline__ float ld_cg(const float* p) { return __ldcg(p); }
__device__ __forceinline__ F64Run ld_cg(const F64Run* p) {
    // 16-byte records, 8-byte aligned: two 8-byte loads
    const double a = __ldcg(reinterpret_cast<const double*>(p));
    const float2 t = __ldcg(reinterpret_cast<const float2*>(reinterpret_cast<const char*>(p) + 8));
    return {a, t.x, t.y};
}
__device__ __forceinline__ F32Pair ld_cg(const F32Pair* p) {
    const float2 t = __ldcg(reinterpret_cast<const float2*>(p));
    return {t.x, t.y};
}

// CG: the row's value may have been written by another SM earlier in the same launch.
template <class Op, int VW, bool CG = false, class Acc>
__device__ __forceinline__ void write_row(const SweepParams<typename Op::S>& p, long long row, int col,
                                          const Acc& tot) {
    using S = typename Op::S;
    using A = typename Op::A;
    const long long node = p.rows[row];
    A sum[VW];
#pragma unroll
    for (int i = 0; i < VW; i++) sum[i] = tot.get(i);
    if (p.state != nullptr) {
        // the node's sum so far (earlier passes) stays in accumulator form: merge into it, and
        // either keep it (mode 1) or write the node value from it (mode 2)
        A* st = static_cast<A*>(p.state) + (node - p.state_base) * p.stride + col;
#pragma unroll
        for (int i = 0; i < VW; i++) {
            A cur = ld_cg(st + i);
            Op::merge(cur, sum[i]);
            sum[i] = cur;
        }
        if (p.state_mode == 1) {
#pragma unroll
            for (int i = 0; i < VW; i++) st[i] = sum[i];
            return;
        }
    }
    S* d = p.dst + node * p.stride + col;
    S out[VW];
    if (p.rmw) {
        S base[VW];
        if constexpr (CG) ld_l2<S, VW>(d, base);
        else ld_plain<S, VW>(d, base);
#pragma unroll
        for (int i = 0; i < VW; i++) out[i] = Op::finish_onto(base[i], sum[i]);
    } else {
#pragma unroll
        for (int i = 0; i < VW; i++) out[i] = Op::finish(sum[i]);
    }
    Vec<S, VW>::st(d, out);
}

// Accumulators may bound their running chains: AddF64S renormalises its float pair every 4
// additions (settle) and folds it into a double every 32 (flush).
template <class Op> struct ChainTraits {
    static constexpr bool kChains = false;
};
template <> struct ChainTraits<AddF64S> {
    static constexpr bool kChains = true;
};
template <> struct ChainTraits<AddF64SD> : ChainTraits<AddF64S> {};
template <> struct ChainTraits<AddF32G> : ChainTraits<AddF64S> {};
template <> struct ChainTraits<AddF64G> : ChainTraits<AddF64S> {};

// Chunk tail: the warp's last row sum is written, or -- a piece of a heavy row -- published as a
// partial; the last piece to finish (atomic ticket) adds all of them up in piece order.
template <class Op, int VW, int G, class Acc>
__device__ __forceinline__ void finish_chunk(const SweepParams<typename Op::S>& p, long long c, const ChunkDev& ch,
                                             long long cur, Acc& acc, int lane, int lg, int col, bool colok) {
    using A = typename Op::A;
    constexpr int NG = 32 / G;
    group_allreduce<Op, VW, G>(acc);
    if (ch.heavy < 0) {
        if (lg == 0 && colok) write_row<Op, VW>(p, cur, col, acc);
        return;
    }
    const HeavyDev hr = p.heavy[ch.heavy];
    const long long piece = c - hr.first_chunk;
    A* part = reinterpret_cast<A*>(p.partials);
    if (lg == 0 && colok) {
#pragma unroll
        for (int i = 0; i < VW; i++) part[(hr.slot_base + piece) * p.stride + col + i] = acc.get(i);
    }
    __threadfence();
    __syncwarp();
    unsigned ticket = 0;
    if (lane == 0) ticket = atomicAdd(p.tickets + (long long)ch.heavy * p.ntiles + blockIdx.y, 1u);
    ticket = __shfl_sync(FULL_MASK, ticket, 0);
    if (ticket != (unsigned)hr.n_pieces - 1u) return;
    __threadfence();
    Acc sum;
    sum.zero();
    if (colok) {
        for (int pc = lg; pc < hr.n_pieces; pc += NG) {
            const A* src = part + (hr.slot_base + pc) * p.stride + col;
#pragma unroll
            for (int i = 0; i < VW; i++) sum.add_partial(i, ld_cg(src + i));
        }
    }
    group_allreduce<Op, VW, G>(sum);
    if (lg == 0 && colok) write_row<Op, VW>(p, cur, col, sum);
}

template <class Op, int VW, int G, int D, bool ID16>
__device__ __forceinline__ void sweep_chunk(const SweepParams<typename Op::S>& p, long long c, int lane) {
    using S = typename Op::S;
    using A = typename Op::A;
    using Acc = VecAcc<Op, VW>;
    constexpr int NG = 32 / G;  // groups per warp = edges per sub-step
    // gathers in flight per lane: 4 for 16-byte vectors, 8 for narrower ones, times the depth D
    constexpr int BATCH = ((VW * sizeof(S) >= 16) ? 4 : 8) * D;
    constexpr int UNR = (G >= BATCH) ? 1 : BATCH / G;  // 32-edge blocks per step
    constexpr int STEPS = UNR * G;                     // sub-steps per step (a multiple of BATCH)
    constexpr unsigned NGMASK = (NG == 32) ? 0xffffffffu : ((1u << NG) - 1u);
    constexpr int FLUSH_EVERY = (STEPS >= 32) ? 1 : 32 / STEPS;
    constexpr bool kChains = ChainTraits<Op>::kChains;

    const int lg = lane / G;  // group
    const int li = lane % G;  // lane inside the group
    const int col = p.col_base + blockIdx.y * (G * VW) + li * VW;
    const bool colok = col < p.stride;
    const unsigned upto = (2u << lg) - 1u;  // groups 0..lg

    const ChunkDev ch = p.chunks[c];
    const long long eEnd = p.chunks[c + 1].e0;

    Acc acc;
    acc.zero();
    long long cur = ch.r0;
    bool first = true;
    int nsteps = 0;

    uint32_t nraw[UNR];
#pragma unroll
    for (int b = 0; b < UNR; b++) {
        const long long e = ch.e0 + 32 * b + lane;
        nraw[b] = (e < eEnd) ? load_id<ID16>(p, e) : 0u;
    }
    for (long long base = ch.e0; base < eEnd; base += 32 * UNR) {
        uint32_t raw[UNR];
        unsigned heads[UNR];
        unsigned anyHead = 0;
#pragma unroll
        for (int b = 0; b < UNR; b++) {
            raw[b] = decode_id<ID16>(p, nraw[b]);
            heads[b] = __ballot_sync(FULL_MASK, raw[b] & 0x80000000u);
            anyHead |= heads[b];
        }
        // prefetch the next step's edge ids while this step's gathers are in flight
        const long long nbase = base + 32 * UNR;
        if (nbase < eEnd) {
#pragma unroll
            for (int b = 0; b < UNR; b++) {
                const long long e = nbase + 32 * b + lane;
                nraw[b] = (e < eEnd) ? load_id<ID16>(p, e) : 0u;
            }
        }
        if (first) {
            cur = ch.r0 - (long long)(heads[0] & 1u);
            first = false;
        }
        const long long left = eEnd - base;  // valid edges from `base`
#pragma unroll
        for (int t0 = 0; t0 < STEPS; t0 += BATCH) {
            S v[BATCH][VW];
#pragma unroll
            for (int u = 0; u < BATCH; u++) {
                const int t = t0 + u;
                const int b = t / G, s = t % G;
                const int j = s * NG + lg;
                // with one lane per row (G == 1) each lane gathers the edge id it loaded itself
                const uint32_t idx = ((G == 1) ? raw[b] : __shfl_sync(FULL_MASK, raw[b], j)) & 0x7fffffffu;
                if (32 * b + j < left && colok) {
                    Vec<S, VW>::ld(p.src + (long long)idx * p.stride + col, v[u]);
                } else {
#pragma unroll
                    for (int i = 0; i < VW; i++) v[u][i] = S{};
                }
            }
            // No row starts in this batch of sub-steps: every edge continues the current row.  The
            // step's heads are tested first (one test when the step has none); a boundary elsewhere
            // in the step leaves this batch on the block path too, which adds its edges with fewer
            // compensated additions and runs the short, shared code -- per-sub-step boundary code
            // for every sub-step of a boundary step made UP split passes wait on instruction fetch.
            auto batch_heads = [&]() {
                unsigned bh = 0u;
#pragma unroll
                for (int u = 0; u < BATCH; u++) {
                    const int t = t0 + u;
                    const int b = t / G, s = t % G;
                    bh |= (NG == 32) ? heads[b] : ((heads[b] >> (s * NG)) & NGMASK);
                }
                return bh;
            };
            if (anyHead == 0u || batch_heads() == 0u) {
                acc.template add_block<BATCH>(v);
                continue;
            }
#pragma unroll
            for (int u = 0; u < BATCH; u++) {
                const int t = t0 + u;
                const int b = t / G, s = t % G;
                const unsigned hs = (NG == 32) ? heads[b] : ((heads[b] >> (s * NG)) & NGMASK);
                if (hs == 0u) {
                    acc.add(v[u]);
                    if (kChains && (u & 3) == 3) acc.settle();
                    continue;
                }
                const int q = __popc(hs & upto);  // rows started at or before my edge
                const int Q = __popc(hs);
                // 1) the current row ends in this sub-step
                Acc x = acc;
                if (q == 0) x.add(v[u]);
                group_allreduce<Op, VW, G>(x);
                if (cur >= ch.r0 && lg == 0 && colok) write_row<Op, VW>(p, cur, col, x);
                // 2) rows that start and end inside this sub-step: segmented scan over groups
                if (Q > 1) {
                    Acc y;
                    y.zero();
                    if (q >= 1) y.add(v[u]);
#pragma unroll
                    for (int d = 1; d < NG; d <<= 1) {
                        const int qu = __shfl_up_sync(FULL_MASK, q, d * G);
                        const auto tv = y.shfl_up(d * G);
                        if (lg >= d && qu == q) y.merge(tv);
                    }
                    const int qn = __shfl_down_sync(FULL_MASK, q, G);
                    const bool tail = (lg == NG - 1) || (qn != q);
                    if (tail && q >= 1 && q < Q && colok) write_row<Op, VW>(p, cur + q, col, y);
                }
                // 3) the last row continues into the next sub-step
                acc.zero();
                if (q == Q) acc.add(v[u]);
                cur += Q;
            }
        }
        if (kChains) {
            if (++nsteps == FLUSH_EVERY) {
                nsteps = 0;
                acc.settle();
                acc.flush();
            }
        }
    }

    finish_chunk<Op, VW, G>(p, c, ch, cur, acc, lane, lg, col, colok);
}

// Persistent warps: each warp takes chunks of the level from a shared counter until none are
// left, so long and short chunks balance across the SMs.
// Blocks per SM the register budget is sized for (65536 / (256 * blocks) registers per thread).
// The deep variant (D = 2) keeps twice the gathers in flight per lane and gives up one block
// per SM for the registers they take; which of the two a level runs is the autotuner's choice.
template <class Op, int VW, int G, int D> struct SweepOccupancy {
    // compensated float shapes with several 32-edge blocks per step hold more state per lane
    static constexpr bool kWide = (std::is_same<Op, AddF32C>::value || std::is_same<Op, AddF64S>::value) && G <= 2 && VW >= 2;
    static constexpr int kBlocks = (kWide ? 3 : 4) - (D > 1 ? 1 : 0);
};

template <class Op, int VW, int G, int D, bool ID16>
__device__ __forceinline__ void sweep_level(const SweepParams<typename Op::S>& p) {
    const int lane = threadIdx.x & 31;
    unsigned* counter = p.work + blockIdx.y;
    for (;;) {
        long long c = 0;
        if (lane == 0) c = (long long)atomicAdd(counter, 1u);
        c = __shfl_sync(FULL_MASK, c, 0) + p.c_begin;
        if (c >= p.c_end) return;
        sweep_chunk<Op, VW, G, D, ID16>(p, c, lane);
    }
}

template <class Op, int VW, int G, int D, bool ID16>
__global__ void __launch_bounds__(256, SweepOccupancy<Op, VW, G, D>::kBlocks) sweep_kernel(const SweepParams<typename Op::S> p) {
    if constexpr (std::is_same<Op, AddF64S>::value) {
        if (p.gate != nullptr && *p.gate != 0) {
            sweep_level<AddF64, VW, G, D, ID16>(as_f64(p));
            return;
        }
    }
    sweep_level<Op, VW, G, D, ID16>(p);
}

// A level of short rows (most with one edge: a node's only parent, a node's only mutation): G lanes
// per row walk the row's edges from its offset, many rows at a time.  sweep_kernel would walk such
// rows one boundary after the other within a chunk, a chain of dependent steps that sets the
// launch's time however few edges the level has: float64 K=20 on N=20,000, M=50,000, 130-150 us for
// a DOWN level of a few thousand one-edge rows.  Bound by the latency of three dependent loads.
// A level with longer rows among them has `short_split` groups of lanes to a row, which take its
// edges in turns of four and merge their sums at the end.
constexpr int kShortBatch = 4;

// Row `row` of such a level, from its edges e, e + split batches on, ..: `id` holds the first batch's
// ids (past `end`: any).  The warp's lanes call it together; `live` lanes have a row and a column.
template <class Op, int VW, int G, bool CG>
__device__ __forceinline__ void short_row(const SweepParams<typename Op::S>& p, const uint32_t* __restrict__ adj, long long row,
                                          int col, int split, int sub, bool live, unsigned e, unsigned end,
                                          uint32_t (&id)[kShortBatch]) {
    using S = typename Op::S;
    constexpr bool kPairs = std::is_same<Op, AddF64S>::value;
    ScalarAcc<Op, VW> acc;
    acc.zero();
    while (e < end) {
        S v[kShortBatch][VW];
#pragma unroll
        for (int u = 0; u < kShortBatch; u++) {
            if (e + u < end) {
                const S* from = p.src + (long long)(id[u] & 0x7fffffffu) * p.stride + col;
                if constexpr (CG) ld_l2<S, VW>(from, v[u]);
                else Vec<S, VW>::ld(from, v[u]);
            } else {
#pragma unroll
                for (int i = 0; i < VW; i++) v[u][i] = S{};
            }
        }
        const unsigned at = e;
        e += kShortBatch * split;
#pragma unroll
        for (int u = 0; u < kShortBatch; u++)
            if (e + u < end) id[u] = __ldg(adj + e + u);
        if constexpr (kPairs) {
            // normalised float pairs throughout: no run to fold, and no FP64 pipe
#pragma unroll
            for (int i = 0; i < VW; i++) {
                const DF t = df_add(df_add(v[0][i], v[1][i]), df_add(v[2][i], v[3][i]));
                const DF r = df_add(DF{acc.a[i].hi, acc.a[i].lo}, t);
                acc.a[i].hi = r.hi;
                acc.a[i].lo = r.lo;
            }
        } else if constexpr (std::is_same<Op, AddF32>::value || std::is_same<Op, AddF64>::value) {
            // plain sums: the batch as a tree (what lies past the row's end is zero)
#pragma unroll
            for (int i = 0; i < VW; i++) acc.a[i] += (v[0][i] + v[1][i]) + (v[2][i] + v[3][i]);
        } else {
#pragma unroll
            for (int u = 0; u < kShortBatch; u++)
                if (at + u < end) acc.add(v[u]);
        }
    }
    for (int m = G; m < G * split; m <<= 1) {
        const ScalarAcc<Op, VW> t = acc.shfl_xor(m);
        if constexpr (kPairs) {
#pragma unroll
            for (int i = 0; i < VW; i++) {
                const DF r = df_add(DF{acc.a[i].hi, acc.a[i].lo}, DF{t.a[i].hi, t.a[i].lo});
                acc.a[i].hi = r.hi;
                acc.a[i].lo = r.lo;
            }
        } else {
            acc.merge(t);
        }
    }
    if (!live || sub != 0) return;
    if constexpr (kPairs) {
        if (p.state == nullptr) {
            DF* d = p.dst + (long long)p.rows[row] * p.stride + col;
            DF out[VW];
            if (p.rmw) {
                if constexpr (CG) ld_l2<DF, VW>(d, out);
                else ld_plain<DF, VW>(d, out);
            }
#pragma unroll
            for (int i = 0; i < VW; i++) {
                const DF r{acc.a[i].hi, acc.a[i].lo};
                out[i] = p.rmw ? df_add(out[i], r) : r;
            }
            Vec<DF, VW>::st(d, out);
            return;
        }
    }
    write_row<Op, VW, CG>(p, row, col, acc);
}

template <class Op, int VW, int G>
__device__ __forceinline__ void short_rows(const SweepParams<typename Op::S>& p) {
    const int split = p.short_split;
    const long long thread = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long row = thread / (G * split);
    const int sub = static_cast<int>(thread / G) & (split - 1);
    const int col = blockIdx.y * (G * VW) + (threadIdx.x % G) * VW;
    const bool live = row < p.short_rows && col < p.stride;
    unsigned e = 0, end = 0;
    if (live) {
        e = __ldg(p.short_off + row) + kShortBatch * sub;
        end = __ldg(p.short_off + row + 1);
    }
    uint32_t id[kShortBatch];
#pragma unroll
    for (int u = 0; u < kShortBatch; u++) id[u] = (e + u < end) ? __ldg(p.adj + e + u) : 0u;
    short_row<Op, VW, G, false>(p, p.adj, p.short_row0 + row, col, split, sub, live, e, end, id);
}

template <class Op, int VW, int G>
__global__ void __launch_bounds__(256) short_rows_kernel(const SweepParams<typename Op::S> p) {
    if constexpr (std::is_same<Op, AddF64S>::value) {
        if (p.gate != nullptr && *p.gate != 0) {
            short_rows<AddF64, VW, G>(as_f64(p));
            return;
        }
    }
    short_rows<Op, VW, G>(p);
}

}  // namespace grgx
